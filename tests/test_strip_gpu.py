"""The strip kernel on the GPU against the oracle: both slot counts, several
right-hand sides (one and two columns per CTA), the three precisions, odd
grids, remote values from far rows, and a plan saved and loaded."""
import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle
from test_strip_layout import grid_rows

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def solve(plan, b, k=1, prec=rbs.PREC_FP64):
    d = torch.tensor(b, device="cuda")
    x = torch.full_like(d, float("nan"))
    for _ in range(2):
        plan.solve(d, x, k=k, prec=prec)
    return x.cpu().numpy()


@pytest.mark.parametrize("sub", [rbs.FORWARD, rbs.BACKWARD])
@pytest.mark.parametrize("g,h,offsets", [
    (40, 40, [(-1, 0), (0, -1)]), (301, 257, [(-1, 0), (0, -1)]), (70, 245, [(-1, -1), (-1, 0), (-1, 1), (0, -1)]),
    (400, 33, None)])
def test_grid_factors(g, h, offsets, sub, tmp_path):
    rp, ci, va = grid_rows(g, h, offsets or [(-1, 0), (0, -1)], g, far=0 if offsets else 50)
    n = len(rp) - 1
    fmt = rbs.FMT_CSR if sub == rbs.FORWARD else rbs.FMT_CSC
    plan = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=fmt)
    assert len(plan.export("strip_dim")) == 4
    L = (rp, ci, va) if sub == rbs.FORWARD else oracle.transpose(rp, ci, va)
    B = rbs.gen_uniform(5, 100 * n).reshape(100, n)
    ref = np.stack([oracle.sptrsv_csr(*L, sub, b) for b in B])
    assert rel_err(solve(plan, B[0]), ref[0]) <= 1e-12
    assert rel_err(solve(plan, B[:3], k=3), ref[:3]) <= 1e-12
    assert rel_err(solve(plan, B, k=100), ref) <= 1e-12
    assert rel_err(solve(plan, B[1]), ref[1]) <= 1e-12
    assert rel_err(solve(plan, B[2], prec=rbs.PREC_MIXED), ref[2]) <= 1e-12
    assert rel_err(solve(plan, B[:5], k=5, prec=rbs.PREC_MIXED), ref[:5]) <= 1e-12
    assert rel_err(solve(plan, B, k=100, prec=rbs.PREC_FP32), ref) <= 1e-5
    plan.save(tmp_path / "p")
    assert np.array_equal(solve(rbs.load_plan(tmp_path / "p"), B[3]), solve(plan, B[3]))
