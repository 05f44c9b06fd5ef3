"""The product build outside the range of its short reciprocals and roots (ib_fast.cuh): subnormal and huge
densities, subnormal and infinite squared sound speeds, through every kernel that a sweep can take.

The functions are compared with CUDA's division and square root directly, over random exponents and at the ends
of their ranges.  The sweeps are compared with the oracle, whose operations are IEEE's.  Tolerance of the
sweeps: subnormal numbers here keep 50 to 51 of 53 bits, so 8 times the sweeps' 1e-13 (relative L1)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

import gpuimogen_b200.build as build
from gpuimogen_b200 import ensemble as en
from gpuimogen_b200 import problems
from helpers import host, oracle_cyl_loop, rel_l1, to_fluid

pytestmark = pytest.mark.gpu

SRC = r'''
#include "ib_fast.cuh"
__global__ void k(const double *a, const double *x, double *o, long n)
{
    const long i = threadIdx.x + (long)blockIdx.x * blockDim.x;
    if (i >= n) return;
    const double v = x[i];
    double r[12] = {ib::rcp_fast(v), ib::rcp_full(v), ib::rcp_fast_pos(v), 1.0 / v, ib::sqrt_fast(v), ib::sqrt_full(v),
                    sqrt(v), ib::quotient_fast(a[i], v, ib::rcp_fast(v)), a[i] / v, ib::rcp_outside(v) ? 1.0 : 0.0,
                    ib::rcp_any(v), ib::root_any(v)};
    for (int j = 0; j < 12; j++) o[j * n + i] = r[j];
}
extern "C" __attribute__((visibility("default"))) int run(const double *a, const double *x, double *o, long n)
{
    k<<<(unsigned)((n + 255) / 256), 256>>>(a, x, o, n);
    return (int)cudaDeviceSynchronize();
}
'''


@pytest.fixture(scope="module")
def functions(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("fast")
    src, lib = os.path.join(d, "fast.cu"), os.path.join(d, "fast.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build.NVCC, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + build.CSRC, "-shared",
                    "-Xcompiler", "-fPIC", "-o", lib, src], check=True)
    run = ctypes.CDLL(lib).run

    def call(a, x):
        a, x = torch.tensor(a, device="cuda"), torch.tensor(x, device="cuda")
        o = torch.empty((12, len(x)), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert run(*[ctypes.c_void_p(t.data_ptr()) for t in (a, x, o)], ctypes.c_long(len(x))) == 0
        names = ["rcp", "rcp_full", "rcp_pos", "ref_rcp", "root", "root_full", "ref_root", "quotient", "ref_quotient", "outside",
                 "rcp_any", "root_any"]
        return dict(zip(names, o.cpu().numpy()))

    return call


def _ulps(a, b):
    """|a - b| in units of the last place of b (finite, same sign)."""
    return np.abs(a.view(np.int64) - b.view(np.int64))


def _same(a, b):
    return np.where(np.isnan(b), np.isnan(a), a == b)


def _numbers(seed, n=400000):
    rng = np.random.Generator(np.random.Philox(seed))
    e = rng.integers(-1074, 1024, n)
    x = np.ldexp(1.0 + rng.random(n), e) * rng.choice([-1.0, 1.0], n)
    t = np.finfo(float)
    edge = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, t.tiny, -t.tiny, np.nextafter(t.tiny, 0), t.smallest_subnormal, t.max, -t.max,
                     2.0 ** 1022, np.nextafter(2.0 ** 1022, 0), 2.0 ** -1024, 2.0 ** -1023, 1.0, np.nextafter(1.0, 2), 3.0])
    return np.concatenate([x, edge])


def test_reciprocals(functions):
    x = _numbers(1)
    o = functions(np.ones_like(x), x)
    inside = (np.abs(x) >= 2.0 ** -1022) & (np.abs(x) < 2.0 ** 1022)
    assert np.array_equal(o["outside"] == 0, inside)
    assert _ulps(o["rcp"][inside], o["ref_rcp"][inside]).max() <= 1
    assert _ulps(o["rcp_full"][inside], o["ref_rcp"][inside]).max() <= 1
    assert _same(o["rcp_full"][~inside], o["ref_rcp"][~inside]).all()
    special = ~np.isfinite(o["ref_rcp"]) | (o["ref_rcp"] == 0)
    assert _same(o["rcp_any"][special], o["ref_rcp"][special]).all()
    assert _ulps(o["rcp_any"][~special], o["ref_rcp"][~special]).max() <= 1
    # outside: NaN, or 0 for numbers above 2^1022
    low = ~(np.abs(x) >= 2.0 ** -1022) | np.isinf(x)
    assert np.isnan(o["rcp"][low]).all() and (o["rcp"][~inside & ~low & (np.abs(x) > 2.0 ** 1022)] == 0).all()
    pos = ~np.signbit(x) & (x < 2.0 ** 1022)
    assert _ulps(o["rcp_pos"][pos & inside], o["ref_rcp"][pos & inside]).max() <= 1
    assert (np.isfinite(o["rcp_pos"][pos]) & (o["rcp_pos"][pos] > 0)).all()


def test_roots(functions):
    x = _numbers(2)
    o = functions(np.ones_like(x), x)
    inside = (x >= 2.0 ** -1022) & np.isfinite(x)
    assert _ulps(o["root"][inside], o["ref_root"][inside]).max() <= 1
    assert _ulps(o["root_full"][inside], o["ref_root"][inside]).max() <= 1
    small = ~inside & (np.abs(x) < 2.0 ** -1022) & (x != 0)
    assert np.isnan(o["root"][~inside & ~small]).all() and np.isinf(o["root"][small]).all()
    assert _same(o["root_full"][~inside], o["ref_root"][~inside]).all()
    special = ~np.isfinite(o["ref_root"]) | (x == 0)
    assert _same(o["root_any"][special], o["ref_root"][special]).all()
    assert _ulps(o["root_any"][~special], o["ref_root"][~special]).max() <= 1
    assert np.array_equal(np.signbit(o["root_full"][x == 0]), np.signbit(x[x == 0]))


def test_quotients(functions):
    x, a = _numbers(3), np.random.Generator(np.random.Philox(4)).permutation(_numbers(5))
    o = functions(a, x)
    ok = (o["outside"] == 0) & (np.abs(a) >= 2.0 ** -960) & np.isfinite(a) & (np.abs(o["ref_quotient"]) >= 2.0 ** -960)
    fin = ok & np.isfinite(o["ref_quotient"])
    assert fin.sum() > 200000 and _ulps(o["quotient"][fin], o["ref_quotient"][fin]).max() <= 1
    assert (np.isinf(o["quotient"][ok & ~fin])).all()


# shape and direction per kernel: rows and pencils of the two-cell kernels (even, odd), the pencil boxes (2 and 4
# pencils, fixed and run-time lengths), the pipeline, the chunks, the tile kernel
KERNELS = [((24, 6, 4), 1), ((25, 6, 4), 1), ((600, 3, 2), 1), ((6, 24, 4), 2), ((5, 33, 2), 2), ((6, 4, 40), 3), ((6, 100, 3), 2),
           ((6, 3, 128), 3), ((8, 512, 2), 2), ((364, 364, 66), 3), ((6, 8, 5), 2), ((6, 300, 3), 2), ((1030, 4, 2), 1),
           ((8, 520, 2), 2), ((1031, 3, 2), 1), ((5, 521, 2), 2)]


def _state(kind, shape, seed=5):
    """(q, dt): smooth states whose densities, sound speeds or both lie outside the short forms' range."""
    q = problems.random_smooth(shape, gamma=1.4, seed=seed, amp=0.3)
    dt = 2e-3
    if kind == "subnormal density":       # 1/rho finite, rho not normal
        q *= 1.2e-308
    elif kind == "huge density":          # 1/rho subnormal; gas at rest, so that momenta squared stay finite
        P = 0.4 * (q[1] - 0.5 * (q[2] ** 2 + q[3] ** 2 + q[4] ** 2) / np.where(q[0] > 0, q[0], 1))
        q[0] *= 7e307
        q[1] = P / 0.4 * 1e140
        q[2:] = 0.0
        dt *= 1e10
    elif kind == "subnormal sound speed":  # c^2 = 1e-309
        v, p = 2e-155, 1e-109
        q[0] *= 1e200
        q[1] *= p
        q[2:] *= p / v * 0.5
        dt /= v
    return q, dt


@pytest.mark.parametrize("shape,direction", KERNELS)
@pytest.mark.parametrize("method,slope,kind", [
    (2, "mc", "subnormal density"), (2, "mc", "huge density"), (2, "mc", "subnormal sound speed"),
    (1, "mc", "subnormal density"), (3, "vanleer", "subnormal density")])
def test_sweeps(cuda, ib, po, shape, direction, method, slope, kind):
    q, dt = _state(kind, shape)
    n = shape[0] * shape[1] * shape[2]
    geo = ib.Geometry(shape, (0.05, 0.05, 0.05))
    kw = {"fluxlim": slope} if method == 3 else {"slope": slope}
    ref = q.copy()
    po.fluid_sweep(ref, shape, po.step_params(dt, geo.h, 1.4, rho_min=5e-324, method=method, **kw), direction)
    assert np.isfinite(ref[:, :n]).all() and not np.array_equal(ref[:, :n], q[:, :n])
    fl = to_fluid(q.copy(), shape)
    ib.cudaFluidStep(fl, geo, [dt, 1, 1.4, 5e-324, method, direction], ib.numerics(**kw))
    err = rel_l1(host(fl), ref, n)
    assert np.all(err <= 8e-13), err


@pytest.mark.parametrize("shape,direction", [((1030, 4, 2), 1), ((8, 520, 2), 2), ((8, 3, 520), 3)])
@pytest.mark.parametrize("method", [1, 2])
def test_operands_beyond_a_chunk(cuda, ib, po, shape, direction, method):
    """A cell without internal energy (its sound speed is zero: the short root does not reach it)
    at each distance from a chunk's end, so that in turn it is only among the neighbouring chunk's halo cells."""
    n = shape[0] * shape[1] * shape[2]
    L = {1: 248, 2: 120, 3: 120}[direction]
    stride = {1: 1, 2: shape[0], 3: shape[0] * shape[1]}[direction]
    geo = ib.Geometry(shape, (0.05, 0.05, 0.05))
    for d in range(-5, 6):
        q = problems.random_smooth(shape, gamma=1.4, seed=7, amp=0.1)
        i = (L + d) * stride + (1 if direction > 1 else 0)
        rho = q[0, i]
        q[:, i] = [rho, 0.0, 0.0, 0.0, 0.0]          # at rest, without pressure: P is exactly zero
        ref = q.copy()
        po.fluid_sweep(ref, shape, po.step_params(1e-3, geo.h, 1.4, rho_min=1e-5, method=method, slope="mc"), direction)
        fl = to_fluid(q.copy(), shape)
        ib.cudaFluidStep(fl, geo, [1e-3, 1, 1.4, 1e-5, method, direction], ib.numerics(slope="mc"))
        out = host(fl)
        fin = np.isfinite(ref[:, :n])
        assert np.array_equal(np.isfinite(out[:, :n]), fin), d
        out[:, :n][~fin] = ref[:, :n][~fin] = 0.0
        assert np.all(rel_l1(out, ref, n) <= 1e-13), d


@pytest.mark.parametrize("direction", [1, 2])
@pytest.mark.parametrize("shape", [(32, 24, 6), (21, 9, 5), (12, 72, 3)])
@pytest.mark.parametrize("method", [1, 2])
def test_cylindrical_sweeps(cuda, ib, po, shape, direction, method):
    n = shape[0] * shape[1] * shape[2]
    h = [0.05, 0.04, 0.1]
    q = problems.rotating_annulus(shape, r_inner=1.0, dr=h[0], seed=13) * 0.62e-308
    geo = ib.Geometry(shape, h=h, cylindrical=True, r_inner=1.0)
    fl = to_fluid(q.copy(), shape)
    ib.cudaFluidStep(fl, geo, [0.004, 1, 1.4, 5e-324, method, direction, -1.0, 0], ib.numerics(slope="mc"))
    ref = q.copy()
    po.fluid_sweep(ref, shape, po.step_params(0.004, h, 1.4, rho_min=5e-324, method=method, slope="mc", cylindrical=True, r_inner=1.0),
                   direction)
    assert np.isfinite(ref[:, :n]).all()
    err = rel_l1(host(fl), ref, n)
    assert np.all(err <= 1e-11), err


@pytest.mark.parametrize("direction", [1, 2, 3])
@pytest.mark.parametrize("method", [1, 2, 3])
@pytest.mark.parametrize("shape", [(24, 20, 18), (66, 68, 70)])
def test_one_infinite_cell(cuda, ib, po, shape, method, direction):
    """Which cells stay finite, and their values, beside a cell of infinite energy (Xin-Jin: the freezing speed is
    the pencil's maximum, so an infinite sound speed leaves no cell of its pencil finite)."""
    n = shape[0] * shape[1] * shape[2]
    q = problems.random_smooth(shape, gamma=1.4, seed=6, amp=0.3)
    q[1, n // 2 + shape[0] // 2] = np.inf
    geo = ib.Geometry(shape, (0.05, 0.05, 0.05))
    ref = q.copy()
    po.fluid_sweep(ref, shape, po.step_params(2e-3, geo.h, 1.4, rho_min=1e-5, method=method), direction)
    fl = to_fluid(q.copy(), shape)
    ib.cudaFluidStep(fl, geo, [2e-3, 1, 1.4, 1e-5, method, direction], ib.numerics())
    out = host(fl)
    fin = np.isfinite(ref[:, :n])
    assert not fin.all() and np.array_equal(np.isfinite(out[:, :n]), fin)
    out[:, :n][~fin] = ref[:, :n][~fin] = 0.0
    assert np.all(rel_l1(out, ref, n) <= 1e-13)


@pytest.mark.parametrize("sizes", [[9, 40, 255, 256, 503, 600], [13, 120, 249, 300] * 500])
@pytest.mark.parametrize("method", [1, 2])
def test_ensemble(cuda, ib, po, sizes, method):
    """One row and two rows a thread: every problem scaled to subnormal densities, two iterations.  (Densities between
    1 and 1.5 and velocities of the order of 1, so that no reciprocal overflows.)"""
    rng = np.random.Generator(np.random.Philox(8))
    s = np.ones((len(sizes), 2, 3))
    s[:, :, 0] += 0.5 * rng.random((len(sizes), 2))
    s[:, :, 1] = 0.1 * rng.random((len(sizes), 2))
    q, off, h = en.pack_problems(np.array(sizes), s, 1.4)
    q = q * 1.1e-308
    ens = en.RiemannEnsemble(q, off, h, gamma=1.4, rho_min=5e-324, bc=("const", "const"))
    ens.run(t_end=10.0, method=method, slope="mc", itermax=2)
    torch.cuda.synchronize()
    for p in list(range(len(sizes)))[:8]:
        n = sizes[p]
        ref = np.ascontiguousarray(q[:, off[p]:off[p] + n])
        hh = [h[p], 1.0, 1.0]
        sp = po.step_params(0.0, hh, 1.4, rho_min=5e-324, method=method, slope="mc")
        bc = ["const"] * 2 + ["circular"] * 4
        for it in range(2):
            sp.dt = 0.4 * po.cfl_timestep(ref, (n, 1, 1), 1.4, hh, method)
            po.fluid_step_3d(ref, (n, 1, 1), sp, bc, 1, it)
            po.fluid_step_3d(ref, (n, 1, 1), sp, bc, -1, it)
        got = ens.host_problem(p)[:, :n]
        assert np.isfinite(ref).all()
        err = np.abs(got - ref).sum(axis=1) / np.maximum(np.abs(ref).sum(axis=1), 1e-320)
        assert np.all(err[:3] <= 1e-11), (p, err)


def test_cylindrical_timestep(cuda, ib, po):
    """A whole iteration with the cylinder source, whose quotients by the density leave the corrected form's range."""
    shape, h = (32, 12, 6), [0.05, 0.04, 0.1]
    n = shape[0] * shape[1] * shape[2]
    q = problems.rotating_annulus(shape, r_inner=1.0, dr=h[0], seed=13) * 0.62e-308
    bc = ["const", "const", "circular", "circular", "circular", "circular"]
    ref = q.copy()
    dts = oracle_cyl_loop(po, ref, shape, h, 1.0, 2, 1.4, -1.0, [ib.BC[b] for b in bc], 0.4, 1, slope="mc")
    assert np.isfinite(ref[:, :n]).all()
    fl = to_fluid(q.copy(), shape, bc=bc)
    geo = ib.Geometry(shape, h=h, cylindrical=True, r_inner=1.0)
    ib.completeTimestep([fl], geo, [dts[0], 1, 0, 2], ib.numerics(slope="mc"))
    err = rel_l1(host(fl), ref, n)
    assert np.all(err <= 1e-11), err
