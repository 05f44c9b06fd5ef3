"""The fill of the rows' ends that x sweeps take along inside a fluid step, and the fill with one thread per
pencil, side and slab, against the oracle's sweep followed by its fill: every mode on either side, rows just
long enough for the two sides to be filled apart and one cell shorter (a launch of its own), rows that share a
CTA, odd rows, Xin-Jin's kernels, and the longest rows.  Strict build, bit for bit."""
import numpy as np
import pytest

from gpuimogen_b200 import problems
from helpers import bits_equal, first_diff, host, to_fluid

pytestmark = pytest.mark.gpu

MODES = [("const", "const"), ("mirror", "const"), ("outflow", "outflow"), ("linear", "mirror"), ("outflow", "linear"),
         ("circular", "const"), ("const", "stationary")]


def _step(ib, po, shape, method, bc):
    q = problems.random_smooth(shape, gamma=1.4, seed=8, amp=0.3)
    n = shape[0] * shape[1] * shape[2]
    geo = ib.Geometry(shape, (0.05, 0.04, 0.03))
    codes = [ib.BC[b] for b in bc] + [ib.BC["circular"]] * 4
    ref = q.copy()
    po.fluid_step_3d(ref, shape, po.step_params(2e-3, geo.h, 1.4, rho_min=1e-5, method=method, slope="ospre"), codes, 1, 0)
    ib.use_variant("strict")
    try:
        fl = to_fluid(q.copy(), shape, bc=list(bc) + ["circular"] * 4)
        ib.fluidstep([fl], geo, [2e-3, 1, 1, 0, method])
        out = host(fl)
    finally:
        ib.use_variant("product")
    assert bits_equal(out, ref, n), first_diff(out, ref, n)


@pytest.mark.parametrize("bc", MODES)
@pytest.mark.parametrize("method", [1, 2, 3])
@pytest.mark.parametrize("shape", [(64, 6, 5), (33, 7, 4)])
def test_fill_with_the_sweep(cuda, ib, po, shape, method, bc):
    _step(ib, po, shape, method, bc)


@pytest.mark.parametrize("method", [2, 3])
@pytest.mark.parametrize("nx", [15, 16, 17, 256, 300, 513, 1024, 1025])
def test_fill_by_length(cuda, ib, po, nx, method):
    _step(ib, po, (nx, 5, 4), method, ("mirror", "outflow"))
    _step(ib, po, (nx, 1, 1), method, ("outflow", "const"))


@pytest.mark.parametrize("direction", [1, 2, 3])
@pytest.mark.parametrize("bc", MODES)
@pytest.mark.parametrize("n", [9, 15, 16, 40])
def test_boundary_alone(cuda, ib, po, n, direction, bc):
    shape = [5, 5, 5]
    shape[direction - 1] = n
    shape = tuple(shape)
    q = problems.random_smooth(shape, gamma=1.4, seed=9, amp=0.3)
    codes = [ib.BC["circular"]] * 6
    codes[2 * direction - 2:2 * direction] = [ib.BC[b] for b in bc]
    ref = q.copy()
    po.fluid_boundary(ref, shape, codes, direction)
    ib.use_variant("strict")
    try:
        fl = to_fluid(q.copy(), shape, bc=codes)
        ib.setFluidBoundary(fl, direction)
    finally:
        ib.use_variant("product")
    N = shape[0] * shape[1] * shape[2]
    assert bits_equal(host(fl), ref, N), first_diff(host(fl), ref, N)
