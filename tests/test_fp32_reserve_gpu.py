"""FP32 solves of plans that run whole-matrix walks in FP64: they have device
state of their own, which rbs_plan_reserve and the server's admission build,
so that later solves and batches allocate nothing, and which no other thread
that looks at the plan gets to see."""
import threading

import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FACTORS = {
    "look-ahead": (1, dict(kind=rbs.GEN_BAND_POISSON, n=6000, lam=8, band=256, seed=3)),
    "strip": (2, dict(kind=rbs.GEN_LAPLACE2D, grid=90, seed=4)),
    "band": (3, dict(kind=rbs.GEN_CHAIN, n=60001, chain_bw=3, seed=5)),
}


def factor(name):
    walk, spec = FACTORS[name]
    L = rbs.gen_lower_csr(**spec)
    plan = rbs.analyse(*L, substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR)
    assert plan.export("walk")[0] == walk
    return plan, L


@pytest.mark.parametrize("name", FACTORS)
def test_reserved_solves_allocate_nothing(name):
    plan, L = factor(name)
    n = plan.n
    plan.reserve(8)
    held = plan.info().device_bytes
    B = rbs.gen_uniform(7, 8 * n).reshape(8, n)
    ref = np.stack([oracle.sptrsv_csr(*L, rbs.FORWARD, b) for b in B])
    b, x = torch.tensor(B, device="cuda"), torch.empty(8, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for k in (3, 1, 8, 3, 3, 8):
        for prec, tol in ((rbs.PREC_FP32, 1e-5), (rbs.PREC_FP64, 1e-12), (rbs.PREC_MIXED, 1e-12)):
            plan.solve_async(b, x, k=k, prec=prec)
            plan.sync()
            assert rel_err(x[:k].cpu().numpy(), ref[:k]) <= tol, (k, prec)
            assert plan.info().device_bytes == held, (k, prec)


@pytest.mark.parametrize("name", FACTORS)
def test_server_charges_fp32_at_admission(name):
    plan, L = factor(name)
    n = plan.n
    srv = rbs.Server(hbm_budget_bytes=8 << 30, max_batch_rhs=4)
    fid = srv.add_factor(plan)
    used = srv.stats().hbm_used
    probe, _ = factor(name)
    probe.reserve(4)
    probe.solve(*(torch.zeros(4, n, dtype=torch.float64, device="cuda") for _ in range(2)), k=4, prec=rbs.PREC_FP32)
    assert used >= probe.info().device_bytes
    B = rbs.gen_uniform(8, 3 * n).reshape(3, n)
    b, x = torch.tensor(B, device="cuda"), torch.empty(3, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    srv.wait(srv.submit_device(fid, b, x, k=3, prec=rbs.PREC_FP32))
    ref = np.stack([oracle.sptrsv_csr(*L, rbs.FORWARD, r) for r in B])
    assert rel_err(x.cpu().numpy(), ref) <= 1e-5
    assert srv.stats().hbm_used == used
    srv.close()


def test_other_threads_see_the_plans_own_state():
    plan, L = factor("strip")
    plan.reserve(1)
    held, walk = plan.info().device_bytes, plan.export("walk").tolist()
    b, x = torch.ones(plan.n, dtype=torch.float64, device="cuda"), torch.empty(plan.n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    seen, done = set(), threading.Event()

    def look():
        while not done.is_set():
            seen.add((plan.info().device_bytes, tuple(plan.export("walk").tolist())))

    t = threading.Thread(target=look)
    t.start()
    for _ in range(2000):
        plan.solve_async(b, x, prec=rbs.PREC_FP32)
    plan.sync()
    done.set()
    t.join()
    assert seen == {(held, tuple(walk))}
