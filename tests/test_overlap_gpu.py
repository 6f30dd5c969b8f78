"""b and x in one buffer, shifted against each other by rows or by columns: the
right-hand sides are those at the call, whatever the walk writes when."""
import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FACTORS = {
    "blocks": (0, dict(kind=rbs.GEN_ZIPF, n=20000, zipf_alpha=2.1, zipf_max=1000, seed=5)),
    "look-ahead": (1, dict(kind=rbs.GEN_BAND_POISSON, n=6000, lam=8, band=256, seed=3)),
    "strip": (2, dict(kind=rbs.GEN_LAPLACE2D, grid=90, seed=4)),
    "band": (3, dict(kind=rbs.GEN_CHAIN, n=60001, chain_bw=3, seed=5)),
}


@pytest.mark.parametrize("mixed", [1, 0])
@pytest.mark.parametrize("name", FACTORS)
def test_shifted(name, mixed):
    walk, spec = FACTORS[name]
    L = rbs.gen_lower_csr(**spec)
    n = len(L[0]) - 1
    for sub in (rbs.FORWARD, rbs.BACKWARD):
        plan = rbs.analyse(*L, substitution=sub, lv=1, fmt=rbs.FMT_CSR if sub == rbs.FORWARD else rbs.FMT_CSC,
                           opts=rbs.options(mixed=mixed))
        assert plan.export("walk")[0] == walk
        T = L if sub == rbs.FORWARD else oracle.transpose(*L)
        for k, ld, shift in ((1, n, 100), (1, n, -100), (3, n, n), (3, n, -n), (3, n, 1), (2, n + 7, n - 3), (2, 2 * n, n),
                             (2, n, 0), (1, n, n), (3, n + 1, -2 * (n + 1)), (2, n, 1 - n), (1, n, 1)):
            at = max(0, -shift)
            host = rbs.gen_uniform(9, at + max(0, shift) + (k - 1) * ld + n)
            buf = torch.tensor(host, device="cuda")
            torch.cuda.synchronize()
            plan.solve(buf[at:], buf[at + shift:], k=k, ld=ld)
            got = buf.cpu().numpy()
            for c in range(k):
                ref = oracle.sptrsv_csr(*T, sub, host[at + c * ld:at + c * ld + n])
                assert rel_err(got[at + shift + c * ld:][:n], ref) <= 1e-12, (sub, k, ld, shift, c)
