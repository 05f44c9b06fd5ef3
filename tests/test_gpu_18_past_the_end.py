"""Iterations replayed past the end time change nothing: with the device timestep at 0 neither the sweeps nor the fills
after them (nor statics, nor the cylinder source and its fill) touch the state, in any direction, so a graph loop that
overshoots ends with the host loop's bits."""
import numpy as np
import pytest
import torch

import gpuimogen_b200 as ib
from gpuimogen_b200 import problems
from helpers import bits_equal, first_diff, host, to_fluid

pytestmark = pytest.mark.gpu

BC = {"mixed": ["mirror", "const", "const", "mirror", "const", "const"],
      "y": ["circular", "circular", "outflow", "mirror", "circular", "circular"],
      "x": ["const", "mirror", "circular", "circular", "circular", "circular"]}


def _compare(make, geo, method, num, tmax):
    n = geo.shape[0] * geo.shape[1] * geo.shape[2]
    a = make()
    tm = ib.TimeManager(cfl=0.4, tmax=tmax)
    while tm.running:
        ib.run_iteration([a], geo, tm, method, num)
    b = make()
    loop = ib.GraphLoop([b], geo, method, num, cfl=0.4, tmax=tmax).run(check_every=7)
    s = loop.state()
    assert s.iteration == tm.iteration >= 6 and s.time == tm.time
    assert bits_equal(host(a), host(b), n), first_diff(host(a), host(b), n)
    before = host(b).copy()
    loop.run(6)
    assert bits_equal(before, host(b), n), first_diff(before, host(b), n)


@pytest.mark.parametrize("bc", list(BC))
@pytest.mark.parametrize("method", [1, 2, 3])
@pytest.mark.parametrize("shape", [(40, 36, 20), (33, 70, 1), (66, 18, 17)])
def test_overshooting_replays(cuda, shape, method, bc):
    q = problems.random_smooth(shape, gamma=1.4, seed=3, amp=0.3)
    geo = ib.Geometry(shape)
    _compare(lambda: to_fluid(q.copy(), shape, bc=BC[bc], gamma=1.4), geo, method, ib.numerics(), 0.15)


@pytest.mark.parametrize("method", [2, 3])
def test_overshooting_replays_with_statics(cuda, method):
    shape = (36, 30, 1)
    n = 36 * 30
    q = problems.random_smooth(shape, gamma=1.4, seed=3, amp=0.2)
    idx = np.arange(0, n, 97)
    st = np.stack([idx.astype(float), q[0, idx], np.full(len(idx), 0.5)])
    statics = [torch.tensor(st, dtype=torch.float64, device="cuda")] + [None] * 4
    geo = ib.Geometry(shape)
    _compare(lambda: to_fluid(q.copy(), shape, bc=BC["y"], gamma=1.4, statics=statics), geo, method, ib.numerics(), 0.15)


@pytest.mark.parametrize("method", [2, 3])
def test_overshooting_replays_of_an_annulus(cuda, method):
    shape = (40, 24, 6)
    q = problems.rotating_annulus(shape, r_inner=1.0, dr=0.05, seed=13)
    geo = ib.Geometry(shape, h=[0.05, 0.04, 0.1], cylindrical=True, r_inner=1.0)
    _compare(lambda: to_fluid(q.copy(), shape, bc=["const", "mirror"] + ["circular"] * 4, gamma=1.4), geo, method,
             ib.numerics(slope="mc"), 0.12)
