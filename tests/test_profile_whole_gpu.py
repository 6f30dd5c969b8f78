"""Profiled solves of whole-matrix walks: the first block's time is the
launch's, not that of the other blocks' events (63 blocks here).  It is at
most the solve's own time without profiling, plus a quarter and 10 us for
timing noise, and the blocks' sum is within the profiled solve's."""
import pytest

import rbs

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("walk,spec", [
    (1, dict(kind=rbs.GEN_BAND_POISSON, n=60000, lam=8, band=256, seed=3)),
    (2, dict(kind=rbs.GEN_LAPLACE2D, grid=400, seed=4)),
    (3, dict(kind=rbs.GEN_CHAIN, n=1000000, chain_bw=3, seed=5))])
def test_first_block_is_the_launch(walk, spec):
    L = rbs.gen_lower_csr(**spec)
    plan = rbs.analyse(*L, substitution=rbs.FORWARD, lv=5, fmt=rbs.FMT_CSR)
    assert plan.export("walk")[0] == walk and plan.info().sum_block == 63
    b, x = (torch.ones(plan.n, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    for _ in range(3):
        plan.solve(b, x)
    plain = min(plan.solve(b, x).ms for _ in range(20))
    first, within = [], []
    for _ in range(20):  # the least of 20: the host may be late with a launch
        plan.profile(True)
        total = plan.solve(b, x).ms
        ms, _, solves = plan.block_times()
        assert solves == 1
        first.append(ms[0])
        within.append(ms.sum() <= total)
    assert 0 < min(first) <= 1.25 * plain + 0.010
    assert all(within)
