"""The pencil boxes of 4 (32-byte swizzled; the SSPRK sum in the box): z pencils of 65-256 cells in x-y planes above
1 MB, and the FP32 flux's 512-cell y and z pencils, against the oracle: strict build bit for bit, run-time lengths
(odd ones too) and the compile-time 256; two sweeps in one launch; a wait that runs out.

A z pencil depends on itself alone, so the oracle takes two lines of pencils and the grid repeats them."""
import numpy as np
import pytest
import torch

from gpuimogen_b200 import problems
from helpers import bits_equal, first_diff, product_close, to_fluid

pytestmark = pytest.mark.gpu

NX, NY = 364, 364  # a plane of 1.06 MB


def _tiled(small, n):
    """The state of (NX, NY, n) that repeats the (NX, 2, n) state `small` along y."""
    t = torch.from_numpy(small[:, :NX * 2 * n].reshape(5, n, 2, NX)).cuda()
    q = torch.zeros((5, problems.slab_pitch(NX, NY, n)), dtype=torch.float64, device="cuda")
    q[:, :NX * NY * n].view(5, n, NY // 2, 2, NX).copy_(t[:, :, None])
    return q


def _first(q, n):
    """The first two lines, after a check that every repetition has the same bits."""
    v = q[:, :NX * NY * n].view(5, n, NY // 2, 2, NX)
    bits = v.view(torch.int64)
    assert bool((bits == bits[:, :, :1]).all())
    return v[:, :, 0].reshape(5, -1).cpu().numpy()


def _fluid(ib, q, n):
    return ib.Fluid((NX, NY, n), q=q, gamma=1.4)


@pytest.mark.parametrize("variant", ["strict", "product"])
@pytest.mark.parametrize("n", [65, 100, 255, 256])
@pytest.mark.parametrize("method,slope", [(2, "mc"), (1, "ospre")])
def test_z_of_large_planes(cuda, ib, po, method, slope, n, variant):
    small = problems.random_jumpy((NX, 2, n), gamma=1.4, seed=7)
    geo = ib.Geometry((NX, NY, n), (0.05, 0.04, 0.03))
    ref = small.copy()
    po.fluid_sweep(ref, (NX, 2, n), po.step_params(3e-3, geo.h, 1.4, rho_min=1e-5, method=method, slope=slope), 3)
    ib.use_variant(variant)
    try:
        fl = _fluid(ib, _tiled(small, n), n)
        ib.cudaFluidStep(fl, geo, [3e-3, 1, 1.4, 1e-5, method, 3], ib.numerics(slope=slope))
        out = _first(fl.q, n)
    finally:
        ib.use_variant("product")
    m = NX * 2 * n
    if variant == "strict":
        assert bits_equal(out, ref, m), first_diff(out, ref, m)
    else:
        ok, info = product_close(out, ref, m)
        assert ok, info


@pytest.mark.parametrize("shape,direction", [((8, 512, 3), 2), ((12, 512, 1), 2), ((8, 3, 512), 3)])
@pytest.mark.parametrize("variant", ["strict", "product"])
def test_fp32_512_cell_pencils(cuda, ib, po, shape, direction, variant):
    n = shape[0] * shape[1] * shape[2]
    q = problems.random_smooth(shape, gamma=1.4, seed=7, amp=0.3)
    geo = ib.Geometry(shape, (0.05, 0.04, 0.03))
    ref = q.copy()
    po.fluid_sweep(ref, shape, po.step_params(3e-3, geo.h, 1.4, rho_min=1e-5, method=2, slope="mc"), direction)
    ib.use_variant(variant)
    try:
        fl = to_fluid(q.copy(), shape)
        ib.cudaFluidStep(fl, geo, [3e-3, 1, 1.4, 1e-5, 2, direction], ib.numerics(slope="mc", precision="fp32flux"))
        torch.cuda.synchronize()
        out = fl.q.cpu().numpy()
    finally:
        ib.use_variant("product")
    assert not np.array_equal(out[:, :n], q[:, :n])
    ok, info = product_close(out, ref, n, l1=1e-5, scale=1e-4)  # the form's stated bound
    assert ok, info


@pytest.mark.parametrize("precision,n", [("fp64", 72), ("fp64", 256), ("fp32flux", 72)])
def test_two_sweeps_in_one_launch(cuda, ib, precision, n):
    """Iteration 4's middle pair runs along z: the same bits as two fluid steps."""
    small = problems.random_smooth((NX, 2, n), gamma=1.4, seed=11, amp=0.3)
    geo, num = ib.Geometry((NX, NY, n)), ib.numerics(slope="mc", precision=precision)
    a, b = _fluid(ib, _tiled(small, n), n), _fluid(ib, _tiled(small, n), n)
    ib.completeTimestep([a], geo, [2e-4, 1, 4, 2], num)
    ib.fluidstep([b], geo, [2e-4, 1, 1, 4, 2], num)
    ib.fluidstep([b], geo, [2e-4, 1, -1, 4, 2], num)
    m = NX * NY * n
    assert bool((a.q[:, :m].view(torch.int64) == b.q[:, :m].view(torch.int64)).all())


@pytest.mark.parametrize("precision,shape,direction", [("fp64", (NX, NY, 72), 3), ("fp32flux", (8, 512, 6), 2)])
def test_wait_runs_out(cuda, ib, po, precision, shape, direction):
    L = ib.load("product")
    n = shape[0] * shape[1] * shape[2]
    small = problems.random_smooth((NX, 2, 72), gamma=1.4, seed=5, amp=0.3)
    q = _tiled(small, 72) if direction == 3 else torch.from_numpy(problems.random_smooth(shape, gamma=1.4, seed=5, amp=0.3)).cuda()
    geo, num = ib.Geometry(shape), ib.numerics(slope="mc", precision=precision)
    params = [2e-4, 1, 1.4, 1e-5, 2, direction]
    ib.device_wait_status(clear=True)
    fl = ib.Fluid(shape, q=q.clone(), gamma=1.4)
    try:
        assert L.ib_setTileWaitLimit(0) == 0
        ib.cudaFluidStep(fl, geo, params, num)
        assert ib.device_wait_status() == 1
        assert torch.equal(fl.q[:, :n], q[:, :n])   # no box was computed or stored
    finally:
        L.ib_setTileWaitLimit(-1)
        ib.device_wait_status(clear=True)
    ib.cudaFluidStep(fl, geo, params, num)
    assert ib.device_wait_status() == 0
    again = ib.Fluid(shape, q=q.clone(), gamma=1.4)
    ib.cudaFluidStep(again, geo, params, num)
    assert torch.equal(fl.q[:, :n], again.q[:, :n]) and not torch.equal(fl.q[:, :n], q[:, :n])
