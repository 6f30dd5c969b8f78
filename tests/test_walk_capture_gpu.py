"""Solves recorded into a CUDA graph and replayed with other right-hand sides,
between eager solves of other widths: the look-ahead, strip and band walks
keep no state of theirs on the host."""
import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle
from test_strip_layout import grid_rows

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FACTORS = {
    "look-ahead": (1, lambda: rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=6000, lam=8, band=256, seed=3)),
    "strip": (2, lambda: grid_rows(301, 257, [(-1, 0), (0, -1)], 9)),
    "band": (3, lambda: rbs.gen_lower_csr(rbs.GEN_CHAIN, n=60001, chain_bw=3, seed=5)),
}


@pytest.mark.parametrize("widths", [(1, 1, 1), (3, 1, 100), (100, 64, 2)])  # recorded, then eager ones between replays
@pytest.mark.parametrize("name", FACTORS)
def test_replayed_solves(name, widths):
    walk, make = FACTORS[name]
    rp, ci, va = make()
    n, most = len(rp) - 1, max(widths)
    plan = rbs.analyse(rp, ci, va, substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR)
    assert plan.export("walk")[0] == walk
    plan.reserve(most)
    st = torch.cuda.Stream()
    plan.set_stream(st.cuda_stream)
    B = rbs.gen_uniform(5, 4 * most * n).reshape(4, most, n)
    ref = np.stack([np.stack([oracle.sptrsv_csr(rp, ci, va, rbs.FORWARD, r) for r in m]) for m in B])
    k = widths[0]
    with torch.cuda.stream(st):
        b, x = torch.tensor(B[0, :k], device="cuda"), torch.empty(k, n, dtype=torch.float64, device="cuda")
        be, xe = torch.tensor(B[3], device="cuda"), torch.empty(most, n, dtype=torch.float64, device="cuda")
        st.synchronize()
        plan.solve_async(b, x, k=k)  # kernels loaded
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            plan.solve_async(b, x, k=k)
        for i in (1, 2, 0, 1):
            b.copy_(torch.tensor(B[i, :k]))
            x.fill_(float("nan"))
            g.replay()
            st.synchronize()
            assert rel_err(x.cpu().numpy(), ref[i, :k]) <= 1e-12, i
            for w in widths[1:]:
                plan.solve_async(be, xe, k=w)
                st.synchronize()
                assert rel_err(xe[:w].cpu().numpy(), ref[3, :w]) <= 1e-12, (i, w)
    plan.sync()
    del g


@pytest.mark.parametrize("k", [1, 3, 100])
@pytest.mark.parametrize("sub", [rbs.FORWARD, rbs.BACKWARD])
def test_strip_in_place(k, sub):
    rp, ci, va = grid_rows(301, 257, [(-1, 0), (0, -1)], 9)
    n = len(rp) - 1
    plan = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=rbs.FMT_CSR if sub == rbs.FORWARD else rbs.FMT_CSC)
    assert plan.export("walk")[0] == 2
    L = (rp, ci, va) if sub == rbs.FORWARD else oracle.transpose(rp, ci, va)
    B = rbs.gen_uniform(6, k * n).reshape(k, n)
    x = torch.tensor(B, device="cuda")
    plan.solve(x, x, k=k)
    assert rel_err(x.cpu().numpy(), np.stack([oracle.sptrsv_csr(*L, sub, b) for b in B])) <= 1e-12
