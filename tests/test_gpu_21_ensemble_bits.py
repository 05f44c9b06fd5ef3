"""A problem's bits do not depend on how many problems share its launch: an ensemble large enough for two rows a thread
against the same problems in launches of one row a thread, product build (the strict build's comparison is in
test_gpu_15_ensemble_rows.py)."""
import numpy as np
import pytest
import torch

from gpuimogen_b200 import ensemble as en

pytestmark = pytest.mark.gpu

SIZES = [9, 13, 40, 120, 121, 247, 248, 249, 255, 256, 300, 503, 505]


@pytest.mark.parametrize("slope", ["mc", "ospre"])
@pytest.mark.parametrize("method,precision", [(2, "fp64"), (1, "fp64"), (2, "fp32flux")])
def test_bits_do_not_depend_on_the_count(cuda, ib, method, precision, slope):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    parts = 12                                           # each below the 9 problems per SM of the rule
    np_ = 12 * sms                                       # and together above it
    sizes = np.resize(SIZES, np_)
    _, states = en.riemann_states(np_, 21)

    def run(lo, hi):
        q, off, h = en.pack_problems(sizes[lo:hi], states[lo:hi], 1.4)
        ens = en.RiemannEnsemble(q, off, h, gamma=1.4, bc=("outflow", "mirror"))
        ens.run(t_end=0.05, method=method, slope=slope, itermax=6, precision=precision)
        return ens.q[:, :int(off[-1])], ens.iters, ens.t_out

    whole = run(0, np_)
    step = np_ // parts
    assert np_ >= 9 * sms > step
    some = [run(k, k + step) for k in range(0, np_, step)]
    assert torch.equal(whole[0], torch.cat([p[0] for p in some], dim=1))
    assert torch.equal(whole[1], torch.cat([p[1] for p in some])) and torch.equal(whole[2], torch.cat([p[2] for p in some]))
