"""The band scan of a whole matrix against the oracle: every width of its
maps, rows in the caller's order and reversed, sizes around a chunk and a CTA
and past one CTA per SM, several right-hand sides, the three precisions, and
b and x the same array."""
import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sub", [rbs.FORWARD, rbs.BACKWARD])
@pytest.mark.parametrize("bw", [1, 2, 3, 8])
@pytest.mark.parametrize("n", [1023, 1025, 60001, 200003])
def test_chains(n, bw, sub):
    rp, ci, va = rbs.gen_lower_csr(rbs.GEN_CHAIN, n=n, chain_bw=bw, seed=n + bw)
    fmt = rbs.FMT_CSR if sub == rbs.FORWARD else rbs.FMT_CSC
    plan = rbs.analyse(rp, ci, va, substitution=sub, lv=2, fmt=fmt)
    L = (rp, ci, va) if sub == rbs.FORWARD else oracle.transpose(rp, ci, va)
    B = rbs.gen_uniform(5, 3 * n).reshape(3, n)
    ref = np.stack([oracle.sptrsv_csr(*L, sub, b) for b in B])
    for k, prec, tol in ((1, rbs.PREC_FP64, 1e-12), (3, rbs.PREC_FP64, 1e-12), (3, rbs.PREC_MIXED, 1e-12),
                         (2, rbs.PREC_FP32, 1e-5), (1, rbs.PREC_FP64, 1e-12)):
        b = torch.tensor(B[:k], device="cuda")
        x = torch.full_like(b, float("nan"))
        plan.solve(b, x, k=k, prec=prec)
        assert rel_err(x.cpu().numpy(), ref[:k]) <= tol, (k, prec)
    b = torch.tensor(B[0], device="cuda")
    plan.solve(b, b)
    assert rel_err(b.cpu().numpy(), ref[0]) <= 1e-12
