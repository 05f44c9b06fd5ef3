"""The kernels with two neighbouring cells a thread (ib_duo.cuh) against the oracle, at the sizes where their
index rules can go wrong: the shortest pencils, odd lengths (the last thread owns one cell), rows that share a
CTA, each thread count's first and last length, pencils that do not fill the last CTA, and arrays that are not
16-byte aligned.  Strict build bit for bit, product build within the sweeps' tolerance (FMA contraction)."""
import numpy as np
import pytest
import torch

from gpuimogen_b200 import problems
from helpers import bits_equal, first_diff, host, product_close, to_fluid

pytestmark = pytest.mark.gpu

# x rows: CTAs of 128 (up to 128 cells, 161-256), 160 (129-160, 257-320), 192, 256 and 512 threads
ROWS = [3, 4, 5, 31, 64, 65, 127, 128, 129, 160, 161, 255, 256, 257, 320, 321, 384, 385, 511, 512, 513, 1023, 1024]
# y, z pencils by plain loads: 8 of up to 32 cells (128 threads), 8 of 64, 4 of 128, 2 of 256, 1 of 512
PENCILS = [3, 4, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512]


def _sweep(ib, po, shape, method, direction, variant, slope="mc", precision="fp64", shift=0):
    n = shape[0] * shape[1] * shape[2]
    q = problems.random_jumpy(shape, gamma=1.4, seed=7 + direction)
    geo = ib.Geometry(shape, (0.05, 0.04, 0.03))
    ref = q.copy()
    po.fluid_sweep(ref, shape, po.step_params(3e-3, geo.h, 1.4, rho_min=1e-5, method=method, slope=slope), direction)
    ib.use_variant(variant)
    try:
        fl = to_fluid(q, shape)
        if shift:   # the same state at an address that is 8 bytes past a 16-byte boundary
            buf = torch.zeros(fl.q.numel() + 2, dtype=torch.float64, device="cuda")
            fl.q = buf[1:1 + fl.q.numel()].view(5, -1).copy_(fl.q)
            assert fl.q.data_ptr() % 16 == 8
        ib.cudaFluidStep(fl, geo, [3e-3, 1, 1.4, 1e-5, method, direction], ib.numerics(slope=slope, precision=precision))
        return host(fl), ref, n
    finally:
        ib.use_variant("product")


def _check(out, ref, n, variant):
    if variant == "strict":
        assert bits_equal(out, ref, n), first_diff(out, ref, n)
    else:
        ok, info = product_close(out, ref, n)
        assert ok, info


@pytest.mark.parametrize("variant", ["strict", "product"])
@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("nx", ROWS)
def test_rows(cuda, ib, po, nx, method, variant):
    _check(*_sweep(ib, po, (nx, 7, 3), method, 1, variant), variant)


@pytest.mark.parametrize("variant", ["strict", "product"])
@pytest.mark.parametrize("direction", [2, 3])
@pytest.mark.parametrize("n", PENCILS)
def test_pencils_of_odd_planes(cuda, ib, po, n, direction, variant):
    shape = (5, n, 3) if direction == 2 else (5, 3, n)
    _check(*_sweep(ib, po, shape, 1 + n % 2, direction, variant), variant)


@pytest.mark.parametrize("direction,shape", [(2, (6, 16, 3)), (2, (6, 63, 2)), (3, (4, 5, 40)), (3, (364, 364, 64))])
def test_short_pencils_of_even_planes(cuda, ib, po, direction, shape):
    _check(*_sweep(ib, po, shape, 2, direction, "product"), "product")


@pytest.mark.parametrize("direction,shape", [(1, (64, 6, 5)), (2, (6, 100, 5)), (3, (6, 5, 300))])
def test_arrays_off_the_16_byte_boundary(cuda, ib, po, direction, shape):
    _check(*_sweep(ib, po, shape, 2, direction, "strict", shift=1), "strict")


@pytest.mark.parametrize("direction,shape", [(1, (75, 6, 5)), (1, (256, 6, 5)), (1, (700, 3, 4)), (2, (7, 90, 3)), (3, (7, 3, 201)),
                                             (2, (7, 257, 3)), (2, (8, 403, 2)), (3, (5, 3, 512))])
def test_fp32_flux(cuda, ib, po, direction, shape):
    out, ref, n = _sweep(ib, po, shape, 2, direction, "product", precision="fp32flux")
    ok, info = product_close(out, ref, n, l1=1e-5, scale=1e-4)  # the form's stated bound
    assert ok, info


@pytest.mark.parametrize("nx", [64, 65, 150, 256, 300, 600])
def test_two_sweeps_equal_one_twice(cuda, ib, po, nx):
    """The middle same-axis pair of an iteration: one launch for even rows, the same bits as two sweeps."""
    shape = (nx, 5, 4)
    q = problems.random_smooth(shape, gamma=1.4, seed=3, amp=0.3)
    geo, num = ib.Geometry(shape), ib.numerics(slope="mc")
    a, b = to_fluid(q.copy(), shape), to_fluid(q.copy(), shape)
    it = 2   # forward order of iteration 2 ends, and the backward one begins, along x
    ib.completeTimestep([a], geo, [1e-3, 1, it, 2], num)
    ib.fluidstep([b], geo, [1e-3, 1, 1, it, 2], num)
    ib.fluidstep([b], geo, [1e-3, 1, -1, it, 2], num)
    n = shape[0] * shape[1] * shape[2]
    assert bits_equal(host(a), host(b), n)
