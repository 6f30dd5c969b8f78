"""Edges of the whole-matrix walks, each asserted to be the walk taken: the
band scan at its smallest matrix, around a CTA's rows and past one CTA per SM
(where chunks double); systems of one or two rows in a batch of the look-ahead
kernel; wide and narrow strip solves in turn; and a band scan whose waits run
out of polls."""
import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle
from test_strip_layout import grid_rows

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def check(plan, L, sub, k, seed=5, prec=rbs.PREC_FP64):
    B = rbs.gen_uniform(seed, k * plan.n).reshape(k, plan.n)
    b = torch.tensor(B, device="cuda")
    x = torch.full_like(b, float("nan"))
    torch.cuda.synchronize()
    plan.solve(b, x, k=k, prec=prec)
    ref = np.stack([oracle.sptrsv_csr(*L, sub, r) for r in B])
    assert rel_err(x.cpu().numpy(), ref) <= 1e-12, (k, prec)


@pytest.mark.parametrize("sub", [rbs.FORWARD, rbs.BACKWARD])
@pytest.mark.parametrize("bw", [1, 2, 3, 8])
@pytest.mark.parametrize("n", [3500, 4095, 4096, 4097, 148 * 1024 - 1, 148 * 1024, 148 * 1024 + 1])
def test_band_sizes(n, bw, sub):
    rp, ci, va = rbs.gen_lower_csr(rbs.GEN_CHAIN, n=n, chain_bw=bw, seed=n + bw)
    plan = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=rbs.FMT_CSR if sub == rbs.FORWARD else rbs.FMT_CSC)
    assert plan.export("walk")[0] == 3
    L = (rp, ci, va) if sub == rbs.FORWARD else oracle.transpose(rp, ci, va)
    check(plan, L, sub, 1)
    check(plan, L, sub, 3)
    check(plan, L, sub, 2, prec=rbs.PREC_MIXED)


@pytest.mark.parametrize("sizes", [(1, 2, 1500, 1, 40), (1, 900), (1200, 1, 1, 1, 1)])
def test_batches_with_tiny_systems(sizes):
    systems = [rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=n, lam=8, band=64, seed=70 + i) for i, n in enumerate(sizes)]
    plan, offs = rbs.batch_analyse(systems, substitution=rbs.FORWARD, fmt=rbs.FMT_CSR)
    assert plan.export("walk")[0] == 1 and offs.tolist() == np.concatenate([[0], np.cumsum(sizes)]).tolist()
    for k, prec in ((1, rbs.PREC_FP64), (3, rbs.PREC_FP64), (2, rbs.PREC_MIXED)):
        B = rbs.gen_uniform(9, k * plan.n).reshape(k, plan.n)
        b = torch.tensor(B, device="cuda")
        x = torch.full_like(b, float("nan"))
        torch.cuda.synchronize()
        plan.solve(b, x, k=k, prec=prec)
        got = x.cpu().numpy()
        for L, a, e in zip(systems, offs[:-1], offs[1:]):
            for c in range(k):
                assert rel_err(got[c, a:e], oracle.sptrsv_csr(*L, rbs.FORWARD, B[c, a:e])) <= 1e-12, (k, a, c)


@pytest.mark.parametrize("mixed", [1, 0])
def test_wide_and_narrow_strip_solves(mixed):
    L = grid_rows(301, 257, [(-1, 0), (0, -1)], 9)
    plan = rbs.analyse(*L, substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR, opts=rbs.options(mixed=mixed))
    assert plan.export("walk")[0] == 2
    for k in (1, 5, 128, 1, 90, 3, 128, 2):  # work vectors grow twice; one and two columns per CTA
        check(plan, L, rbs.FORWARD, k, seed=k)
        if mixed and k in (3, 128):
            check(plan, L, rbs.FORWARD, k, seed=k, prec=rbs.PREC_MIXED)


def test_band_scan_out_of_polls():
    # CTAs on every SM start together and wait for the totals of all before them
    L = rbs.gen_lower_csr(rbs.GEN_CHAIN, n=1000000, chain_bw=3, seed=5)
    plan = rbs.analyse(*L, substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR, opts=rbs.options(spin_limit=1))
    assert plan.export("walk")[0] == 3
    b, x = torch.ones(plan.n, dtype=torch.float64, device="cuda"), torch.empty(plan.n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    codes = set()
    for _ in range(50):  # two polls may just suffice for one solve
        try:
            plan.solve(b, x)
        except rbs.RbsError as e:
            codes.add(e.code)
    assert codes == {rbs.ERR_TIMEOUT}
    plan = rbs.analyse(*L, substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR)
    check(plan, L, rbs.FORWARD, 1)
