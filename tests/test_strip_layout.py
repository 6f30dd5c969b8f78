"""The strip layout on the CPU: strips are replayed one after another (each
may read only strips before it), chunk by chunk with the kernel's window and
remote buffers, and the solution is compared with the oracle's substitution."""
import numpy as np
import pytest

import rbs
from oracle import oracle


def replay(plan, b):
    """x in processing order from the plan's records, b in processing order."""
    W, rows, steps, win = plan.export("strip_dim").tolist()
    first, perm = plan.export("strip_first"), plan.export("strip_perm")
    per, head = 32 * steps, 136
    nw, nv = head + per * W, per * (W + 1)
    rec = plan.export("strip_rec").reshape(len(perm) // per, -1)
    assert rec.shape[1] * 4 == 2 * nw + 8 * nv and first[-1] * per == rows == len(perm)
    assert np.array_equal(np.sort(perm[perm >= 0]), np.arange(len(b)))
    # the original rows of every chunk, ascending, and where they sit in it
    orig = plan.export("perm")
    want = np.where(perm >= 0, orig[np.maximum(perm, 0)], -1).reshape(-1, per)
    srows, at = (plan.export(q).reshape(-1, 32, 8).transpose(0, 2, 1).reshape(-1, per) for q in ("strip_rows", "strip_rows_at"))
    assert np.array_equal(np.take_along_axis(want, at, 1), srows)
    assert all((np.diff(r[r >= 0]) > 0).all() and (r[(r >= 0).sum():] == -1).all() for r in srows)
    published = int(rec[-1][32] + rec[-1][33])
    ex = np.full(published, np.nan)
    owner = np.full(published, -1)  # chunk that publishes a number
    for c in range(len(rec)):
        owner[rec[c][32]:rec[c][32] + rec[c][33]] = c
    assert (owner >= 0).all()
    xs = np.full(rows, np.nan)
    zero = win * 32 + 64
    for s in range(len(first) - 1):
        vals = np.full(zero + 1, np.nan)
        vals[zero] = 0.0
        for c in range(first[s], first[s + 1]):
            k = c - first[s]
            m, v = rec[c][:nw // 2].view(np.uint16), rec[c][nw // 2:].view(np.float64)
            rem = rec[c][:32]
            n = int((rem >= 0).sum())
            assert (rem[n:] == -1).all() and len(set(rem[:n].tolist())) == n
            # published by earlier strips, or by this one before the chunk at whose start they are asked for
            assert ((owner[rem[:n]] < first[s]) | (owner[rem[:n]] < c - 1)).all()
            vals[win * 32 + (k & 1) * 32:win * 32 + (k & 1) * 32 + n] = ex[rem[:n]]
            assert not np.isnan(ex[rem[:n]]).any()
            slots = m[head:].reshape(32, steps, W)
            vv = v[:per * W].reshape(steps, W // 2, 32, 2).transpose(0, 2, 1, 3).reshape(steps, 32, W)
            inv = v[per * W:].reshape(steps, 32)
            for st in range(steps):
                p = perm[c * per + st * 32:c * per + st * 32 + 32]
                bb = np.where(p >= 0, b[np.maximum(p, 0)], 0.0)
                x = (bb - (vv[st] * vals[slots[:, st]]).sum(1)) * inv[st]
                assert not np.isnan(x).any()
                vals[(k * steps + st) % win * 32:(k * steps + st) % win * 32 + 32] = x
                xs[c * per + st * 32:c * per + st * 32 + 32] = x
            n0, np_ = int(rec[c][32]), int(rec[c][33])
            assert np_ <= 64
            ex[n0:n0 + np_] = vals[k % (win // steps) * per + m[72:72 + np_].astype(int)]
    x = np.empty(len(b))
    x[perm[perm >= 0]] = xs[perm >= 0]
    return x


def check(plan, rp, ci, va, sub):
    n = len(rp) - 1
    b = rbs.gen_uniform(4, n)
    perm = plan.export("perm")
    x = np.empty(n)
    x[perm] = replay(plan, b[perm])
    ref = oracle.sptrsv_csr(rp, ci, va, sub, b)
    assert np.linalg.norm(x - ref) <= 1e-14 * np.linalg.norm(ref)  # at most four products per row


def grid_rows(g, h, offsets, seed, far=0):
    """Lower factor of a g x h grid: row (r, c) reads (r + dr, c + dc) for every offset inside, one row in 101 also
    the row `far` above it."""
    rng = np.random.default_rng(seed)
    rp, ci, va = [0], [], []
    for r in range(g):
        for c in range(h):
            cols = sorted((r + dr) * h + c + dc for dr, dc in offsets if 0 <= r + dr and 0 <= c + dc < h)
            if far and r >= far and (r * h + c) % 101 == 0:
                cols = sorted(cols + [(r - far) * h + c])
            v = rng.uniform(-1, 1, len(cols))
            ci += cols + [r * h + c]
            va += v.tolist() + [1 + np.abs(v).sum()]
            rp.append(len(ci))
    return np.array(rp, np.int32), np.array(ci, np.int32), np.array(va)


@pytest.mark.parametrize("sub", [rbs.FORWARD, rbs.BACKWARD])
@pytest.mark.parametrize("g,h,offsets", [
    (40, 40, [(-1, 0), (0, -1)]), (97, 61, [(-1, 0), (0, -1)]), (33, 200, [(-1, 0), (0, -1)]),
    (70, 45, [(-1, -1), (-1, 0), (-1, 1), (0, -1)]),      # 9-point
    (64, 50, [(-1, 0), (0, -1), (-2, 0)]), (200, 33, None)])  # None: 5-point with far rows
def test_replay_matches_substitution(g, h, offsets, sub):
    rp, ci, va = grid_rows(g, h, offsets or [(-1, 0), (0, -1)], g, far=0 if offsets else 50)
    opts = rbs.options(host_only=1)
    if sub == rbs.FORWARD:
        plan, L = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=rbs.FMT_CSR, opts=opts), (rp, ci, va)
    else:
        plan, L = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=rbs.FMT_CSC, opts=opts), oracle.transpose(rp, ci, va)
    assert len(plan.export("strip_dim")) == 4
    check(plan, *L, sub)


def test_random_structures_are_refused():
    rp, ci, va = rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=6000, lam=2, band=300, seed=9)
    plan = rbs.analyse(rp, ci, va, substitution=rbs.FORWARD, lv=0, fmt=rbs.FMT_CSR, opts=rbs.options(host_only=1))
    assert len(plan.export("strip_dim")) == 0
