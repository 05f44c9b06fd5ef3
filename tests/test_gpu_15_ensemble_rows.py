"""Ensembles large enough for two rows a thread against the same problems in small ensembles, which run one row a
thread: lengths of one chunk and of several, even and odd, the shortest included.  Strict build: the same bits.
Product build: within the 1e-12 of the ensembles' comparison with the oracle, and the same bits for every launch
shape (a cell's result does not depend on which of a thread's rows it is)."""
import numpy as np
import pytest
import torch

from gpuimogen_b200 import ensemble as en

pytestmark = pytest.mark.gpu

SIZES = np.array([9, 13, 40, 120, 121, 247, 248, 249, 255, 256, 300, 503, 505] * 150)


def _run(ib, variant, lo, hi, method, slope, precision, tuning=None):
    _, states = en.riemann_states(len(SIZES), 21)
    q, off, h = en.pack_problems(SIZES[lo:hi], states[lo:hi], 1.4)
    ens = en.RiemannEnsemble(q, off, h, gamma=1.4, bc=("outflow", "mirror"))
    ib.use_variant(variant)
    try:
        ens.run(t_end=0.05, method=method, slope=slope, itermax=4, precision=precision, tuning=tuning)
        torch.cuda.synchronize()
    finally:
        ib.use_variant("product")
    return ens.q[:, :int(off[-1])].clone(), ens.iters.clone(), ens.t_out.clone()


@pytest.mark.parametrize("slope", ["mc", "ospre"])
@pytest.mark.parametrize("method,precision", [(2, "fp64"), (1, "fp64"), (2, "fp32flux")])
def test_two_rows_equal_one(cuda, ib, method, slope, precision):
    for variant in ("strict", "product"):
        whole = _run(ib, variant, 0, len(SIZES), method, slope, precision)
        parts = [_run(ib, variant, k, k + 390, method, slope, precision) for k in range(0, len(SIZES), 390)]
        q = torch.cat([p[0] for p in parts], dim=1)
        t = torch.cat([p[2] for p in parts])
        assert torch.equal(whole[1], torch.cat([p[1] for p in parts]))
        if variant == "strict" and precision == "fp64":
            assert torch.equal(whole[0], q) and torch.equal(whole[2], t)
        else:  # FP32 fluxes are approximate to 2^-24 in either form: 4 iterations, 4 stages each
            tol = 1e-12 if precision == "fp64" else 4 * 4 * 2.0 ** -23
            err = (whole[0] - q).abs().sum(dim=1) / q.abs().sum(dim=1).clamp(min=1e-300)
            assert float(err[:3].max()) <= tol, err
    for tuning in en.CANDIDATES:
        out = _run(ib, "product", 0, len(SIZES), method, slope, precision, tuning)
        assert all(torch.equal(a, b) for a, b in zip(out, whole)), tuning
