"""The look-ahead level kernel on the GPU against the oracle: every line count
(4, 8, 12), several right-hand sides, the three precisions, batches, wide
levels cut into chunks, entries that left the window, long rows, and a plan
saved and loaded."""
import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def solve(plan, b, k=1, prec=rbs.PREC_FP64):
    d = torch.tensor(b, device="cuda")
    x = torch.full_like(d, float("nan"))
    for _ in range(2):
        plan.solve(d, x, k=k, prec=prec)
    return x.cpu().numpy()


@pytest.mark.parametrize("sub", [rbs.FORWARD, rbs.BACKWARD])
@pytest.mark.parametrize("n,lam,band", [(700, 2, 40), (6000, 8, 256), (9001, 12, 3000), (30000, 6, 5000), (4000, 60, 900),
                                        (3000, 40, 60)])
def test_band_factors(n, lam, band, sub):
    rp, ci, va = rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=n, lam=lam, band=band, seed=n + lam)
    fmt = rbs.FMT_CSR if sub == rbs.FORWARD else rbs.FMT_CSC
    plan = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=fmt)
    assert len(plan.export("la_dim")) == 10
    L = (rp, ci, va) if sub == rbs.FORWARD else oracle.transpose(rp, ci, va)
    B = rbs.gen_uniform(5, 3 * n).reshape(3, n)
    ref = np.stack([oracle.sptrsv_csr(*L, sub, b) for b in B])
    assert rel_err(solve(plan, B[0]), ref[0]) <= 1e-12
    assert rel_err(solve(plan, B, k=3), ref) <= 1e-12
    assert rel_err(solve(plan, B, k=3, prec=rbs.PREC_MIXED), ref) <= 1e-12
    assert rel_err(solve(plan, B[1], prec=rbs.PREC_FP32), ref[1]) <= 1e-5
    assert rel_err(solve(plan, B[2]), ref[2]) <= 1e-12


def test_batch_and_saved_plan(tmp_path):
    systems = [rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=n, lam=8, band=64, seed=70 + n) for n in (40, 1500, 7, 900)]
    plan, offs = rbs.batch_analyse(systems, substitution=rbs.FORWARD, fmt=rbs.FMT_CSR)
    assert len(plan.export("la_dim")) == 10 and plan.export("walk")[0] == 1
    b = rbs.gen_uniform(9, int(offs[-1]))
    x = solve(plan, b)
    for (rp, ci, va), a, e in zip(systems, offs[:-1], offs[1:]):
        assert rel_err(x[a:e], oracle.sptrsv_csr(rp, ci, va, rbs.FORWARD, b[a:e])) <= 1e-12
    plan.save(tmp_path / "p")
    assert np.array_equal(solve(rbs.load_plan(tmp_path / "p"), b), x)
