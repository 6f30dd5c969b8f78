"""Performance cases of the B200 recursive-block triangular solve.

Each case is one call (or one chain of calls) of a program that keeps an
analysed factor on the GPU and applies it again and again: a sparse
preconditioner apply, a direct solver's substitution phase, a batch of small
systems, or the incomplete factorisation that makes such a factor.  The
program runs its work on a stream of its own, which the plan is told to use
(Plan.set_stream), and enqueues solves without waiting (Plan.solve_async).

Structures (the ones of the benchmark and the tests, generated here on the
GPU from the seed):
  laplace   strictly lower part of the 2D 5-point Laplacian, grid x grid
  band      Poisson(lam) entries per row, uniform in the last `band` columns
  zipf      power-law row lengths (exponent 2.1, at most 1000), columns uniform
  chain     the last `bw` columns of every row
  batch     `count` independent band systems, rows log-uniform in [nmin, nmax]
  ilu0      the full 5-point pattern, factored in place of its own pattern

Off-diagonal values are uniform in (-1, 1), on a grid of 2^-30 so that sums
of their magnitudes do not depend on the order of a parallel reduction; the
diagonal is 1 + the sum of the row's magnitudes.  Forward cases pass L as
CSR; backward cases solve with its transpose, whose CSC arrays are L's CSR
arrays.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "recblock-sptrsv_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

_PREC = {"fp64": 0, "mixed": 1, "fp32": 2}
_ZIPF_ALPHA, _ZIPF_MAX = 2.1, 1000
_stream = None


def listed():
    return [
        # a small factor, one right-hand side: launch and latency bound
        dict(name="band_small", kind="band", n=16384, lam=6.0, band=512, backward=False, k=1, prec="fp64"),
        # the benchmark's headline: 2D Laplacian factor, 2,047 narrow levels
        dict(name="laplace_fwd", kind="laplace", grid=1024, backward=False, k=1, prec="fp64"),
        # the transposed factor (second half of a preconditioner apply), an odd grid
        dict(name="laplace_bwd_odd", kind="laplace", grid=777, backward=True, k=1, prec="fp64"),
        # power-law factor (graph problems): few wide levels, heavy-tailed rows
        dict(name="zipf_fwd", kind="zipf", n=2000000, backward=False, k=1, prec="fp64"),
        # its transpose at an odd, smaller size: heavy-tailed columns
        dict(name="zipf_bwd_odd", kind="zipf", n=499979, backward=True, k=1, prec="fp64"),
        # banded chain (1D problems, splines): one row per level
        dict(name="chain_fwd", kind="chain", n=1000000, bw=3, backward=False, k=1, prec="fp64"),
        # the largest factor: 4M rows, about 44M entries, 23k levels of random dependencies
        dict(name="band_large", kind="band", n=4000000, lam=10.0, band=4096, backward=False, k=1, prec="fp64"),
        # block Krylov / several loads: 32 right-hand sides on the headline factor
        dict(name="laplace_k32", kind="laplace", grid=1024, backward=False, k=32, prec="fp64"),
        # an odd number of right-hand sides on a band factor, backward
        dict(name="band_bwd_k5", kind="band", n=200003, lam=8.0, band=1024, backward=True, k=5, prec="fp64"),
        # FP32 sweeps with FP64 refinement, 8 right-hand sides
        dict(name="zipf_mixed_k8", kind="zipf", n=1000000, backward=False, k=8, prec="mixed"),
        # many small independent systems in one plan
        dict(name="batch_256", kind="batch", count=256, nmin=1000, nmax=50000, lam=8.0, band=256, backward=False, k=1,
             prec="fp64"),
        # ILU(0) of the 5-point matrix: the producer of such factors
        dict(name="ilu0_1024", kind="ilu0", grid=1024),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["laplace", "laplace", "band", "band", "zipf", "zipf", "chain", "batch", "ilu0"])
    if kind == "ilu0":
        return dict(kind=kind, grid=int(_log(rng, 65, 1025)))
    backward = rng.random() < 0.5
    if kind == "batch":
        return dict(kind=kind, count=int(_log(rng, 16, 256)), nmin=1000, nmax=int(_log(rng, 4000, 50000)), lam=8.0,
                    band=256, backward=backward, k=1, prec=rng.choice(["fp64", "fp64", "mixed"]))
    k = 1 if rng.random() < 0.55 else int(round(_log(rng, 2, 64)))
    prec = rng.choice(["fp64", "fp64", "fp64", "mixed", "fp32"])
    rows = 2000000 if k == 1 else min(1048576, 24000000 // k)
    c = dict(kind=kind, backward=backward, k=k, prec=prec)
    if kind == "laplace":
        c["grid"] = int(_log(rng, 63, min(1025, math.isqrt(rows))))
    elif kind == "zipf":
        c["n"] = int(_log(rng, 4000, rows))
    elif kind == "chain":
        c["n"] = int(_log(rng, 4000, min(rows, 1000000)))
        c["bw"] = rng.choice([1, 2, 3, 5])
    else:
        c["n"] = int(_log(rng, 4000, min(rows, 1200000)))
        c["band"] = int(max(_log(rng, 128, 4096), c["n"] / 900))
        c["lam"] = round(rng.uniform(4.0, 12.0), 2)
    return c


# ---------------------------------------------------------------------------
# inputs (plain torch, on the GPU)
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 1)
    return g


def _rand(g, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _values(g, n):
    return torch.round((2.0 * _rand(g, n) - 1.0) * (1 << 30)) / (1 << 30)


def _batch_rows(case):
    """Rows of every system: the program's systems keep their sizes from one set of values to the next."""
    r = np.random.default_rng(int(case["count"]) * 100003 + int(case["nmax"]))
    u = r.uniform(math.log(case["nmin"]), math.log(case["nmax"]), int(case["count"]))
    return np.exp(u).astype(np.int64)


def _strict_entries(case, g):
    """Rows and columns (row-major, ascending, distinct) of the strictly lower part, and n."""
    kind = case["kind"]
    dev = "cuda"
    if kind == "laplace":
        s = int(case["grid"])
        n = s * s
        i = torch.arange(n, device=dev)
        pair = torch.stack([torch.where(i >= s, i - s, -1), torch.where(i % s > 0, i - 1, -1)], 1)
        keep = pair >= 0
        return i.repeat_interleave(keep.sum(1)), pair[keep], n
    if kind == "chain":
        n, bw = int(case["n"]), int(case["bw"])
        i = torch.arange(n, device=dev)
        pair = i[:, None] - torch.arange(bw, 0, -1, device=dev)[None, :]
        keep = pair >= 0
        return i.repeat_interleave(keep.sum(1)), pair[keep], n
    if kind == "zipf":
        n = int(case["n"])
        i = torch.arange(n, device=dev)
        p = torch.arange(1, _ZIPF_MAX + 1, dtype=torch.float64).pow(-_ZIPF_ALPHA)
        cdf = (torch.cumsum(p, 0) / p.sum()).to(dev)
        cnt = torch.minimum(torch.searchsorted(cdf, _rand(g, n)).clamp_(max=_ZIPF_MAX - 1) + 1, i)
        first = torch.zeros(n, dtype=torch.int64, device=dev)
    else:
        if kind == "batch":
            ns = torch.from_numpy(_batch_rows(case)).to(dev)
            n = int(ns.sum())
            base = (torch.cumsum(ns, 0) - ns).repeat_interleave(ns)
        else:
            n = int(case["n"])
            base = torch.zeros(n, dtype=torch.int64, device=dev)
        i = torch.arange(n, device=dev)
        first = torch.maximum(base, i - int(case["band"]))
        lam = torch.full((n,), float(case["lam"]), dtype=torch.float64, device=dev)
        cnt = torch.minimum(torch.poisson(lam, generator=g).to(torch.int64), i - first)
    row = i.repeat_interleave(cnt)
    col = first[row] + (_rand(g, row.numel()) * (i - first)[row]).to(torch.int64)
    key = torch.unique(row * n + torch.minimum(col, row - 1))
    return key // n, key % n, n


def _system(case, seed):
    """L as CSR with the diagonal last in every row: (ptr, idx, val), its parts, and n."""
    g = _gen(seed)
    row, col, n = _strict_entries(case, g)
    val = _values(g, row.numel())
    diag = torch.ones(n, dtype=torch.float64, device="cuda").index_add_(0, row, val.abs())
    cnt = torch.bincount(row, minlength=n)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(cnt + 1, 0, out=ptr[1:])
    place = torch.arange(row.numel(), device="cuda") + row  # one diagonal before it for every earlier row
    nnz = row.numel() + n
    idx = torch.empty(nnz, dtype=torch.int32, device="cuda")
    va = torch.empty(nnz, dtype=torch.float64, device="cuda")
    idx[place] = col.to(torch.int32)
    va[place] = val
    last = ptr[1:] - 1
    idx[last] = torch.arange(n, dtype=torch.int32, device="cuda")
    va[last] = diag
    k = int(case["k"])
    b = (2.0 * _rand(g, n * k) - 1.0).reshape(k, n)  # one right-hand side per row: column-major n x k
    return ptr.to(torch.int32), idx, va, (row, col, val, diag), b, n


def _ilu_matrix(case, seed):
    """The 5-point matrix of a grid with random couplings, columns ascending: (ptr, idx, val)."""
    s = int(case["grid"])
    n = s * s
    g = _gen(seed)
    i = torch.arange(n, device="cuda")
    cols = torch.stack([torch.where(i >= s, i - s, -1), torch.where(i % s > 0, i - 1, -1), i,
                        torch.where(i % s < s - 1, i + 1, -1), torch.where(i < n - s, i + s, -1)], 1)
    keep = cols >= 0
    v = -0.5 - 0.5 * _values(g, n * 5).abs().reshape(n, 5)
    v[:, 2] = 0.0
    v = torch.where(keep, v, torch.zeros_like(v))
    v[:, 2] = 1.0 + v.abs().sum(1)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(keep.sum(1), 0, out=ptr[1:])
    return ptr.to(torch.int32), cols[keep].to(torch.int32), v[keep], v.reshape(s, s, 5), keep


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def prepare(case, seed):
    import rbs

    global _stream
    if case["kind"] == "ilu0":
        ptr, idx, val, _, _ = _ilu_matrix(case, seed)
        return dict(ptr=ptr, idx=idx, val=val, lu=torch.empty_like(val))
    ptr, idx, val, _, b, n = _system(case, seed)
    opts = rbs.options(max_rhs=int(case["k"]))
    sub = rbs.BACKWARD if case["backward"] else rbs.FORWARD
    fmt = rbs.FMT_CSC if case["backward"] else rbs.FMT_CSR
    torch.cuda.synchronize()
    if case["kind"] == "batch":
        hp, hi, hv = ptr.cpu().numpy(), idx.cpu().numpy(), val.cpu().numpy()
        systems, r0 = [], 0
        for m in _batch_rows(case):
            r1 = r0 + int(m)
            a, e = int(hp[r0]), int(hp[r1])
            systems.append((hp[r0:r1 + 1] - hp[r0], hi[a:e] - r0, hv[a:e]))
            r0 = r1
        plan, _ = rbs.batch_analyse(systems, substitution=sub, fmt=fmt, opts=opts)
    else:
        plan = rbs.analyse_device(ptr, idx, val, n, idx.numel(), substitution=sub, lv=-1, fmt=fmt, opts=opts)
    if _stream is None:
        _stream = torch.cuda.Stream()
    plan.set_stream(_stream.cuda_stream)  # the program's stream: its solves follow one another
    return dict(plan=plan, b=b, x=torch.empty_like(b), k=int(case["k"]), prec=_PREC[case["prec"]])


def run(state):
    if "lu" in state:
        import rbs

        rbs.ilu0_device(state["ptr"], state["idx"], state["val"], state["lu"])
        return state["lu"]
    state["plan"].solve_async(state["b"], state["x"], k=state["k"], prec=state["prec"])
    return state["x"]


def _mean_zipf():
    p = np.arange(1, _ZIPF_MAX + 1, dtype=np.float64) ** -_ZIPF_ALPHA
    return float((p * np.arange(1, _ZIPF_MAX + 1)).sum() / p.sum())


def work(case):
    kind = case["kind"]
    if kind in ("laplace", "ilu0"):
        s = int(case["grid"])
        n, strict = s * s, 2 * s * (s - 1)
    elif kind == "chain":
        n = int(case["n"])
        strict = n * int(case["bw"])
    elif kind == "zipf":
        n = int(case["n"])
        strict = n * _mean_zipf()
    elif kind == "batch":
        ratio = case["nmax"] / case["nmin"]
        n = case["count"] * (case["nmax"] - case["nmin"]) / math.log(ratio)  # the mean of the log-uniform rows
        strict = n * float(case["lam"])
    else:
        n = int(case["n"])
        strict = n * float(case["lam"])
    if kind == "ilu0":  # pattern and values in, factor out; two updates of a multiply and a subtraction, two divisions per row
        nnz = n + 2 * strict
        return {"bytes": nnz * (4 + 8 + 8) + 4 * (n + 1), "flops": 3.0 * strict}
    nnz, k = strict + n, int(case["k"])
    # the factor (64-bit values, 32-bit indices) once, right-hand sides in and solutions out in 64 bits
    return {"bytes": 12.0 * nnz + 4.0 * (n + 1) + 16.0 * n * k, "flops": 2.0 * nnz * k}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _exact_ilu0(case, seed):
    ptr, idx, val, v, keep = _ilu_matrix(case, seed)
    s = int(case["grid"])
    v = v.cpu().numpy().copy()
    # entry order north, west, diagonal, east, south; a row's only updates are of its diagonal
    for t in range(2 * s - 1):  # anti-diagonals: rows that depend on earlier ones alone
        r = np.arange(max(0, t - s + 1), min(s, t + 1))
        c = t - r
        up, left = r > 0, c > 0
        v[r[up], c[up], 0] /= v[r[up] - 1, c[up], 2]
        v[r[up], c[up], 2] -= v[r[up], c[up], 0] * v[r[up] - 1, c[up], 4]
        v[r[left], c[left], 1] /= v[r[left], c[left] - 1, 2]
        v[r[left], c[left], 2] -= v[r[left], c[left], 1] * v[r[left], c[left] - 1, 3]
    return torch.from_numpy(v.reshape(-1, 5)).to(keep.device)[keep]


def exact(case, seed):
    if case["kind"] == "ilu0":
        return _exact_ilu0(case, seed)
    _, _, _, (row, col, val, diag), b, n = _system(case, seed)
    if case["backward"]:
        order = torch.argsort(col * n + row)
        row, col, val = col[order], row[order], val[order]
    # x = D^-1 (b - N x) repeated until it stands still: N is nilpotent, so the
    # sweep reaches the substitution's solution to rounding
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(row, minlength=n), 0, out=ptr[1:])
    N = torch.sparse_csr_tensor(ptr, col, val, size=(n, n))
    bt, d = b.T.contiguous(), diag[:, None]
    x = bt / d
    for _ in range(4000):
        y = (bt - N @ x) / d
        far = float((y - x).abs().max())
        x = y
        if far <= 1e-17 * float(x.abs().max()):
            break
    return x.T.contiguous()
