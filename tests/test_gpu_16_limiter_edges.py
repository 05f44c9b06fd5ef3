"""The MC slope limiter where its two differences are not ordinary numbers of one sign: beside a NaN (the slope is the
left difference, as in the reference's form with the quotient, so that a cell's left face stays finite beside a NaN
right neighbour) and where their product underflows (the slope is zero).  Product build against the oracle."""
import numpy as np
import pytest

from gpuimogen_b200 import problems
from helpers import host, rel_l1, to_fluid

pytestmark = pytest.mark.gpu


def _sweep(ib, po, q, shape, method, direction):
    geo = ib.Geometry(shape, (0.05, 0.05, 0.05))
    ref = q.copy()
    po.fluid_sweep(ref, shape, po.step_params(2e-3, geo.h, 1.4, rho_min=1e-5, method=method, slope="mc"), direction)
    fl = to_fluid(q.copy(), shape)
    ib.cudaFluidStep(fl, geo, [2e-3, 1, 1.4, 1e-5, method, direction], ib.numerics(slope="mc"))
    return host(fl), ref


@pytest.mark.parametrize("direction", [1, 2, 3])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("shape", [(24, 20, 18), (66, 68, 70)])
def test_beside_a_nan(cuda, ib, po, shape, method, direction):
    n = shape[0] * shape[1] * shape[2]
    q = problems.random_smooth(shape, gamma=1.4, seed=6, amp=0.3)
    q[:, n // 2 + shape[0] // 2] = np.nan
    out, ref = _sweep(ib, po, q, shape, method, direction)
    fin = np.isfinite(ref[:, :n])
    assert not fin.all() and np.array_equal(np.isfinite(out[:, :n]), fin)
    out[:, :n][~fin] = ref[:, :n][~fin] = 0.0
    assert np.all(rel_l1(out, ref, n) <= 1e-13)


@pytest.mark.parametrize("direction", [1, 2, 3])
@pytest.mark.parametrize("method", [1, 2])
def test_underflowing_product(cuda, ib, po, method, direction):
    shape = (24, 20, 18)
    n = shape[0] * shape[1] * shape[2]
    q = problems.random_smooth(shape, gamma=1.4, seed=4, amp=0.3)
    t = 2 + direction % 3
    q[1, :n] -= 0.5 * q[t, :n] ** 2 / q[0, :n]
    q[t, :n] = 1e-170 * np.random.Generator(np.random.Philox(9)).uniform(-1, 1, n)
    out, ref = _sweep(ib, po, q, shape, method, direction)
    assert np.all(rel_l1(out, ref, n) <= 1e-13), rel_l1(out, ref, n)
