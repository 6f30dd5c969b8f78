"""Solves on a plan's own stream and the legacy default stream: walks that
write the caller's solutions early come after work queued there, every other
solve (block walks, host arrays, look-ahead) does not wait for it, and none
of them disturbs a capture of a blocking stream."""
import pytest

import rbs
from _util import rel_err
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SLEEP = 1 << 30  # cycles: half a second

FACTORS = {
    "blocks": (0, dict(kind=rbs.GEN_ZIPF, n=20000, zipf_alpha=2.1, zipf_max=1000, seed=5)),
    "look-ahead": (1, dict(kind=rbs.GEN_BAND_POISSON, n=6000, lam=8, band=256, seed=3)),
    "strip": (2, dict(kind=rbs.GEN_LAPLACE2D, grid=90, seed=4)),
    "band": (3, dict(kind=rbs.GEN_CHAIN, n=60001, chain_bw=3, seed=5)),
}


def setup(name):
    walk, spec = FACTORS[name]
    L = rbs.gen_lower_csr(**spec)
    plan = rbs.analyse(*L, substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR)
    assert plan.export("walk")[0] == walk
    b = rbs.gen_uniform(7, plan.n)
    db, dx = torch.tensor(b, device="cuda"), torch.empty(plan.n, dtype=torch.float64, device="cuda")
    torch.cuda._sleep(1)  # its kernel loaded
    torch.cuda.synchronize()
    for _ in range(3):  # kernels, descriptors and graphs
        plan.solve(db, dx)
        plan.solve_host(b)
    return plan, b, db, dx, oracle.sptrsv_csr(*L, rbs.FORWARD, b)


@pytest.mark.parametrize("name", FACTORS)
def test_host_arrays_do_not_wait(name):
    plan, b, _, _, ref = setup(name)
    torch.cuda._sleep(SLEEP)
    end = torch.cuda.Event()
    end.record()
    x, _ = plan.solve_host(b)
    early = not end.query()
    torch.cuda.synchronize()
    assert early and rel_err(x, ref) <= 1e-12


@pytest.mark.parametrize("name,waits", [("blocks", False), ("look-ahead", False), ("strip", True), ("band", True)])
def test_device_arrays(name, waits):
    plan, _, db, dx, ref = setup(name)
    torch.cuda._sleep(SLEEP)
    if waits:
        dx.fill_(float("nan"))  # queued before the solve
    end = torch.cuda.Event()
    end.record()
    plan.solve(db, dx)
    assert end.query() == waits
    torch.cuda.synchronize()
    assert rel_err(dx.cpu().numpy(), ref) <= 1e-12


@pytest.mark.parametrize("name", FACTORS)
def test_capture_of_a_blocking_stream_survives(name):
    runtime = pytest.importorskip("cuda.bindings.runtime")
    plan, _, db, dx, ref = setup(name)
    err, st = runtime.cudaStreamCreate()  # synchronises with the legacy stream
    assert err == 0
    err, = runtime.cudaStreamBeginCapture(st, runtime.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)
    assert err == 0
    plan.solve(db, dx)
    err, graph = runtime.cudaStreamEndCapture(st)
    assert err == 0
    runtime.cudaGraphDestroy(graph)
    runtime.cudaStreamDestroy(st)
    assert rel_err(dx.cpu().numpy(), ref) <= 1e-12
