"""The fill's forms by size and modes (one thread per pencil; per side; per side and slab) against the oracle: one or both
ends outflow, and as many pencils as send a fill along y or z to the first form.  Strict build, bit for bit."""
import pytest

from gpuimogen_b200 import problems
from helpers import bits_equal, first_diff, host, to_fluid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc", [("outflow", "circular"), ("stationary", "outflow"), ("outflow", "outflow"), ("outflow", "const")])
@pytest.mark.parametrize("shape,direction", [((20, 6, 5), 1), ((6, 20, 5), 2), ((7, 5, 33), 3), ((1023, 16, 129), 2), ((363, 364, 16), 3)])
def test_fill(cuda, ib, po, shape, direction, bc):
    n = shape[0] * shape[1] * shape[2]
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
    assert bits_equal(host(fl), ref, n), first_diff(host(fl), ref, n)
