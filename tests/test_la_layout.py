"""The look-ahead level layout on the CPU: the records are replayed with the
kernel's schedule (old values gathered five chunks ahead, early sums one
chunk ahead, both before and after the rows of the chunk in between are
written) and the solution is compared with the oracle's substitution."""
import numpy as np
import pytest

import rbs
from oracle import oracle

def replay(plan, b):
    """x in processing order from the plan's records, b in processing order."""
    xw, nm, nh, q, nx, s64, s32, rb, aux, ahead = plan.export("la_dim").tolist()
    tab = plan.export("la_tab").reshape(-1, 4)
    segs = plan.export("la_segs").reshape(-1, 2)
    rec = plan.export("la_rec").reshape(-1, rb // 4)
    oldp = plan.export("la_old")
    assert s64 >= 5 and s32 >= 5 and nm % 32 == 0 and nh % 32 == 0 and nm <= nh and nm + nh <= 960 and q in (4, 8, 12)
    oh, ox, ov = 16 + 8 * nm, 16 + 8 * nm + 2 * q * nh, 16 + 8 * nm + 2 * q * nh + 2 * nx
    assert rb == ov + 8 * (4 * nm + q * nh + nx) and len(rec) == len(tab)
    x = np.full(len(b), np.nan)
    covered = np.zeros(len(b), int)
    for first, count in segs:
        vals = np.full(xw + aux + 2 * nh + 16, np.nan)  # window, old values, two buffers of sums, zero
        vals[xw + aux + 2 * nh] = 0.0
        recs = []
        for (lo, nr, oo, on), r in zip(tab[first:first + count].tolist(), rec[first:first + count]):
            m, v = r[:ov // 4].view(np.uint16), r[ov // 4:].view(np.float64)
            assert r[0] == lo and r[2] == nr and nr <= nm and on <= 64
            hs = m[oh // 2:ox // 2].reshape(nh // 32, q // 4, 32, 4).transpose(0, 2, 1, 3).reshape(nh, q)
            hv = v[4 * nm:4 * nm + q * nh].reshape(nh // 32, q // 2, 32, 2).transpose(0, 2, 1, 3).reshape(nh, q)
            mv = v[:4 * nm].reshape(nm // 32, 2, 32, 2).transpose(0, 2, 1, 3).reshape(nm, 4)
            assert hs.max() < len(vals) and m[8:oh // 2].reshape(nm, 4)[:, :3].max() < len(vals)
            recs.append((lo, nr, int(r[1]), m[8:oh // 2].reshape(nm, 4), hs, hv, m[ox // 2:], v, mv, oldp[oo:oo + on],
                         oo - tab[first][2]))
            covered[lo:lo + nr] += 1

        def gather(j):
            if j >= count:
                return
            old, a0 = recs[j][9], recs[j][10]
            assert not np.isnan(x[old]).any(), "an old value is not final when it is gathered"
            vals[xw + ((a0 + np.arange(len(old))) & (aux - 1))] = x[old]

        def early(j):
            s = (recs[j][5] * vals[recs[j][4]]).sum(1)
            assert not np.isnan(s).any(), "an early dependency was not in the window"
            return s

        def store(j, s):
            vals[xw + aux + (j & 1) * nh:xw + aux + (j & 1) * nh + nh] = s

        for j in range(ahead):
            gather(j)
        store(0, early(0))
        for c in range(count):
            lo, nr, vb, mw, _, _, xsl, v, mv, _, _ = recs[c]
            gather(c + ahead)
            before = early(c + 1) if c + 1 < count else None
            if before is not None:
                store(c + 1, before)  # the other buffer: this chunk's sums stay
            xs = np.full(nr, np.nan)
            for t in range(nr):
                w0, w1, w2, e = mw[t].tolist()
                s = vals[xw + aux + (c & 1) * nh + t] + (mv[t, :3] * vals[[w0, w1, w2]]).sum()
                for k in range(e >> 5, (e >> 5) + (e & 31)):
                    s += v[4 * nm + q * nh + k] * vals[xsl[k]]
                xs[t] = (b[lo + t] - s) * mv[t, 3]
            assert not np.isnan(xs).any()
            vals[(vb + np.arange(nr)) & (xw - 1)] = xs
            x[lo:lo + nr] = xs
            if before is not None:
                assert np.array_equal(early(c + 1), before), "rows of a chunk overwrite slots still in use"
    assert (covered == 1).all()
    return x


def check(plan, rp, ci, va, sub, seed=3):
    n = len(rp) - 1
    b = rbs.gen_uniform(seed, n)
    perm = plan.export("perm")
    x = np.empty(n)
    x[perm] = replay(plan, b[perm])
    ref = oracle.sptrsv_csr(rp, ci, va, sub, b)
    # a row's sum in another order: n*eps bound of a sum of at most a few hundred terms
    assert np.linalg.norm(x - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("sub", [rbs.FORWARD, rbs.BACKWARD])
@pytest.mark.parametrize("n,lam,band", [(5, 2, 3), (700, 6, 32), (6000, 8, 256), (9000, 12, 3000), (30000, 6, 5000),
                                        (4000, 60, 900), (3000, 40, 60)])
def test_replay_matches_substitution(n, lam, band, sub):
    rp, ci, va = rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=n, lam=lam, band=band, seed=n + lam)
    opts = rbs.options(host_only=1)
    if sub == rbs.FORWARD:
        plan = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=rbs.FMT_CSR, opts=opts)
        check(plan, rp, ci, va, sub)
    else:
        plan = rbs.analyse(rp, ci, va, substitution=sub, lv=1, fmt=rbs.FMT_CSC, opts=opts)
        check(plan, *oracle.transpose(rp, ci, va), sub)


def test_replay_wide_levels_and_old_entries():
    # 6,000 independent rows, then rows that read scattered ones of them (most
    # have left the window) and a neighbour
    rng = np.random.default_rng(5)
    n0, n1 = 6000, 3000
    rows = [[] for _ in range(n0)]
    for i in range(n1):
        r = [n0 + i - 1] if i else []
        far = rng.integers(max(0, n0 + i - 300), n0 + i - 1 if i > 1 else n0, 12).tolist()
        if i % 8 == 0:
            far.append(int(rng.integers(0, 500)))
        rows.append(sorted(set(r + far)))
    rp, ci, va = [0], [], []
    for i, r in enumerate(rows):
        v = rng.uniform(-1, 1, len(r))
        ci += r + [i]
        va += v.tolist() + [1 + np.abs(v).sum()]
        rp.append(len(ci))
    rp, ci, va = np.array(rp, np.int32), np.array(ci, np.int32), np.array(va)
    plan = rbs.analyse(rp, ci, va, substitution=rbs.FORWARD, lv=0, fmt=rbs.FMT_CSR, opts=rbs.options(host_only=1))
    assert len(plan.export("la_old")) > 50
    check(plan, rp, ci, va, rbs.FORWARD)


def test_replay_batch():
    systems = [rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=n, lam=8, band=64, seed=70 + n) for n in (40, 1500, 7, 900)]
    plan, offs = rbs.batch_analyse(systems, substitution=rbs.FORWARD, fmt=rbs.FMT_CSR, opts=rbs.options(host_only=1))
    assert len(plan.export("la_segs")) == 2 * len(systems)
    rp, ci, va = [np.zeros(1, np.int32)], [], []
    for (p, c, v), o in zip(systems, offs[:-1]):
        rp.append(p[1:] + rp[-1][-1])
        ci.append(c + o)
        va.append(v)
    check(plan, np.concatenate(rp).astype(np.int32), np.concatenate(ci).astype(np.int32), np.concatenate(va), rbs.FORWARD)


def test_scattered_dependencies_are_refused():
    rp, ci, va = rbs.gen_lower_csr(rbs.GEN_ZIPF, n=60000, zipf_alpha=2.1, zipf_max=1000, seed=9)
    plan = rbs.analyse(rp, ci, va, substitution=rbs.FORWARD, lv=0, fmt=rbs.FMT_CSR, opts=rbs.options(host_only=1))
    assert len(plan.export("la_dim")) == 0
