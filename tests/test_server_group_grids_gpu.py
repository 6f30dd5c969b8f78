"""Grids on the diagonal of one matrix, analysed as a single system (so their
factor runs on the strip kernel), then served as a group: requests of every
member, FP64, mixed and FP32, one and several columns, against the oracle."""
import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle
from test_strip_layout import grid_rows

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_block_diagonal_grids():
    parts = [grid_rows(g, h, [(-1, 0), (0, -1)], g + h) for g, h in ((60, 60), (41, 57))]
    sizes = [len(p[0]) - 1 for p in parts]
    offs = np.concatenate([[0], np.cumsum(sizes)])
    rp = np.concatenate([parts[0][0], parts[1][0][1:] + parts[0][0][-1]]).astype(np.int32)
    ci = np.concatenate([parts[0][1], parts[1][1] + offs[1]]).astype(np.int32)
    va = np.concatenate([p[2] for p in parts])
    plan = rbs.analyse(rp, ci, va, substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR)
    assert plan.export("walk")[0] == 2
    b = rbs.gen_uniform(4, int(offs[-1]))
    x = torch.zeros(int(offs[-1]), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    plan.solve(torch.tensor(b, device="cuda"), x)
    assert rel_err(x.cpu().numpy(), oracle.sptrsv_csr(rp, ci, va, rbs.FORWARD, b)) <= 1e-12
    srv = rbs.Server(hbm_budget_bytes=8 << 30, max_batch_rhs=8)
    fids = srv.add_group(plan, offs)
    for prec, tol in ((rbs.PREC_FP64, 1e-12), (rbs.PREC_MIXED, 1e-12), (rbs.PREC_FP32, 1e-5)):
        reqs = []
        for m, k in ((0, 1), (1, 3), (0, 2), (1, 1)):
            B = rbs.gen_uniform(10 * m + k, k * sizes[m]).reshape(k, sizes[m])
            dB = torch.tensor(B, device="cuda")
            dX = torch.full_like(dB, float("nan"))
            torch.cuda.synchronize()
            reqs.append((m, B, dX, srv.submit_device(fids[m], dB, dX, k=k, prec=prec)))
        for m, B, dX, t in reqs:
            srv.wait(t)
            ref = np.stack([oracle.sptrsv_csr(*parts[m], rbs.FORWARD, r) for r in B])
            assert rel_err(dX.cpu().numpy(), ref) <= tol, (prec, m)
    srv.close()
