"""Banded chains whose maps grow: products of their
maps over the whole chain overflow although the solutions are finite, so the
band scan must not form them.  The right-hand side is a unit vector 1,000 rows
before the end of the substitution (all earlier solutions are zero, the last
1,000 grow by a fixed ratio): NaN or infinity anywhere is an overflowed
product.  One sign throughout, so every solution carries at most 1,000 rows of
roundings and the tolerance is 1,000 * 8 * 2^-53 rounded up."""
import numpy as np
import pytest

import rbs
from _util import rel_err
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def chain(n, coefs):
    """Row i: -coefs[d - 1] in column i - d, then the unit diagonal."""
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.ones(n)]
    for d, c in enumerate(coefs, 1):
        rows.append(np.arange(d, n))
        cols.append(np.arange(n - d))
        vals.append(np.full(n - d, -c))
    row, col, val = map(np.concatenate, (rows, cols, vals))
    order = np.lexsort((col, row))
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(row, minlength=n))
    return rp, col[order].astype(np.int32), val[order]


@pytest.mark.parametrize("sub", [rbs.FORWARD, rbs.BACKWARD])
@pytest.mark.parametrize("select", [rbs.SELECT_AUTO, rbs.SELECT_REFERENCE])
@pytest.mark.parametrize("coefs", [(1.02,), (0.32, 0.4, 0.3)])
def test_growing_chain(coefs, select, sub):
    n = 600011
    rp, ci, va = chain(n, coefs)
    fmt = rbs.FMT_CSR if sub == rbs.FORWARD else rbs.FMT_CSC
    plan = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=fmt, opts=rbs.options(select=select, max_rhs=3))
    kernels = plan.export("kernel")
    assert kernels[0] == rbs.K_BANDSCAN and kernels[2] == rbs.K_BANDSCAN
    walk = plan.export("walk")[0]
    L = (rp, ci, va) if sub == rbs.FORWARD else oracle.transpose(rp, ci, va)
    B = np.zeros((3, n))
    for c, back in enumerate((1000, 900, 500)):
        B[c, n - back if sub == rbs.FORWARD else back - 1] = 1.0
    ref = np.stack([oracle.sptrsv_csr(*L, sub, b) for b in B])
    assert np.isfinite(ref).all()
    for k in (1, 3, 1):
        b = torch.tensor(B[:k], device="cuda")
        x = torch.full_like(b, float("nan"))
        plan.solve(b, x, k=k)
        assert rel_err(x.cpu().numpy(), ref[:k]) <= 1e-12, k
    assert walk == 0  # not one scan over the whole matrix


@pytest.mark.parametrize("bw", [1, 2, 3, 8])
@pytest.mark.parametrize("n", [5000, 60001, 1000000])
def test_transposed_dominant_chain_keeps_the_whole_scan(n, bw):
    # rows of the transpose are not dominant, their products decay all the same
    rp, ci, va = rbs.gen_lower_csr(rbs.GEN_CHAIN, n=n, chain_bw=bw, seed=n + bw)
    L = oracle.transpose(rp, ci, va)
    off = np.abs(L[2]).copy()
    first = L[0][:-1]
    assert bw == 1 or (np.add.reduceat(off, first) > 2 * off[first]).any()
    plan = rbs.analyse(rp, ci, va, substitution=rbs.BACKWARD, lv=1, fmt=rbs.FMT_CSC)
    assert n == 5000 or plan.export("walk")[0] == 3
    b = rbs.gen_uniform(3, n)
    x = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    plan.solve(torch.tensor(b, device="cuda"), x)
    assert rel_err(x.cpu().numpy(), oracle.sptrsv_csr(*L, rbs.BACKWARD, b)) <= 1e-12


@pytest.mark.parametrize("coefs,walk", [((1.0,), 3), ((0.5, 0.25, 0.25), 3), ((1.0 + 1e-9,), 0)])
def test_rows_at_the_limit_of_dominance(coefs, walk):
    n = 60001
    rp, ci, va = chain(n, coefs)
    plan = rbs.analyse(rp, ci, va, substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR)
    assert plan.export("walk")[0] == walk
    b = rbs.gen_uniform(3, n)
    x = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    plan.solve(torch.tensor(b, device="cuda"), x)
    assert rel_err(x.cpu().numpy(), oracle.sptrsv_csr(rp, ci, va, rbs.FORWARD, b)) <= 1e-9
