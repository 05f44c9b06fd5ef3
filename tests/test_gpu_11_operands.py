"""The product build's reciprocals and square roots (ib_fast.cuh) at the ends of their operands' range.

Each case is one sweep against the oracle, whose divisions and roots are IEEE's: cells without pressure
(square roots of exactly zero), densities and speeds far from one, and slopes so small that the limiters'
products underflow.  The tolerance is the sweeps' own (FMA contraction, a few units in the last place
per operation); underflowing slopes are compared with the field's scale, because the oracle's own
quotient of subnormal numbers carries no digits there."""
import numpy as np
import pytest

from gpuimogen_b200 import problems
from helpers import host, product_close, to_fluid

pytestmark = pytest.mark.gpu

SHAPE = (24, 20, 16)
N = SHAPE[0] * SHAPE[1] * SHAPE[2]


def _run(ib, po, q, method, direction, slope, dt, gamma=1.4):
    geo = ib.Geometry(SHAPE, (0.05, 0.05, 0.05))
    ref = q.copy()
    kw = {"fluxlim": slope} if method == 3 else {"slope": slope}
    po.fluid_sweep(ref, SHAPE, po.step_params(dt, geo.h, gamma, rho_min=1e-300, method=method, **kw), direction)
    fl = to_fluid(q.copy(), SHAPE, gamma=gamma)
    ib.cudaFluidStep(fl, geo, [dt, 1, gamma, 1e-300, method, direction], ib.numerics(**kw))
    return host(fl), ref


@pytest.mark.parametrize("direction", [1, 2, 3])
@pytest.mark.parametrize("slope", ["mc", "ospre"])
def test_hllc_cold_cells(cuda, ib, po, direction, slope):
    """Every other cell without internal energy: sound speeds of exactly zero at each face (every value is
    a power of two or zero, so that no rounding makes a pressure negative)."""
    i = np.arange(SHAPE[direction - 1])
    view = [1, 1, 1]
    view[3 - direction] = len(i)
    along = lambda a: np.broadcast_to(np.asarray(a, dtype=float).reshape(view), SHAPE[::-1])  # noqa: E731
    v, e = along(np.where(i % 4 < 2, 1.0, -0.5)), along(i % 2)
    z = np.zeros_like(v)
    p = [z, z, z]
    p[direction - 1] = v
    q = problems.pack(SHAPE, np.ones_like(v), 0.5 * v * v + e, *p)
    out, ref = _run(ib, po, q, 2, direction, slope, 4e-3)
    assert np.isfinite(ref[:, :N]).all()
    ok, info = product_close(out, ref, N)
    assert ok, info


@pytest.mark.parametrize("direction", [1, 2, 3])
@pytest.mark.parametrize("method,slope", [(2, "mc"), (2, "ospre"), (1, "vanleer"), (3, "ospre")])
@pytest.mark.parametrize("rho,vel", [(1e-140, 1.0), (1e20, 1e12), (1e-24, 1e7)])
def test_units_far_from_one(cuda, ib, po, direction, method, slope, rho, vel):
    q = problems.random_smooth(SHAPE, gamma=1.4, seed=3, amp=0.3)
    q[0] *= rho
    q[1] *= rho * vel * vel
    q[2:] *= rho * vel
    out, ref = _run(ib, po, q, method, direction, slope, 4e-3 / vel)
    assert np.isfinite(ref[:, :N]).all()
    ok, info = product_close(out, ref, N)
    assert ok, info


@pytest.mark.parametrize("direction", [1, 2, 3])
@pytest.mark.parametrize("method,slope", [(2, "mc"), (2, "ospre"), (2, "vanleer"), (1, "ospre"), (3, "ospre"), (3, "vanleer")])
@pytest.mark.parametrize("tiny", [1e-140, 1e-158, 1e-300])
def test_underflowing_slopes(cuda, ib, po, direction, method, slope, tiny):
    """A transverse momentum of the order of `tiny`: products of two of its slopes are subnormal or zero."""
    q = problems.random_smooth(SHAPE, gamma=1.4, seed=4, amp=0.3)
    t = 2 + direction % 3
    rng = np.random.Generator(np.random.Philox(9))
    q[1, :N] -= 0.5 * q[t, :N] ** 2 / q[0, :N]
    q[t, :N] = tiny * rng.uniform(-1, 1, N)
    out, ref = _run(ib, po, q, method, direction, slope, 4e-3)
    assert np.isfinite(out[:, :N]).all() and np.isfinite(ref[:, :N]).all()
    assert np.max(np.abs(out[t, :N])) <= 4 * tiny
    out[t], ref[t] = 0.0, 0.0
    ok, info = product_close(out, ref, N)
    assert ok, info
