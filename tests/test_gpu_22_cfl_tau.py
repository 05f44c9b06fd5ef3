"""cfl_tau of one fluid and of several, finite and not, against the library's own CFL call."""
import numpy as np
import pytest

import gpuimogen_b200 as ib
from gpuimogen_b200 import problems
from gpuimogen_b200.timestep import cfl_tau
from helpers import to_fluid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [1, 2, 3])
def test_one_and_several_fluids(cuda, method):
    shape = (24, 20, 16)
    geo = ib.Geometry(shape)
    fl = [to_fluid(problems.random_smooth(shape, gamma=1.4, seed=s, amp=0.3), shape) for s in (3, 4)]
    t = [ib.cflTimestepFused(f, f.gamma, geo, method) for f in fl]
    assert t[0] != t[1]
    assert [cfl_tau([f], geo, method) for f in fl] == t
    assert cfl_tau(fl, geo, method) == min(t)
    fl[1].q[:, :24 * 20 * 16] = np.nan      # no candidate at all
    if not np.isfinite(ib.cflTimestepFused(fl[1], fl[1].gamma, geo, method)):
        for fluids in ([fl[1]], fl):
            with pytest.raises(ib.ImogenError):
                cfl_tau(fluids, geo, method)
