"""The look-ahead layout's size: bounded by a multiple of the matrix's CSR,
whatever the levels look like (records are as large for one row as for many)."""
import numpy as np
import pytest

import rbs


def layout_bytes(systems, **kw):
    if len(systems) == 1:
        plan = rbs.analyse(*systems[0], substitution=rbs.FORWARD, lv=-1, fmt=rbs.FMT_CSR, opts=rbs.options(host_only=1))
    else:
        plan, _ = rbs.batch_analyse(systems, substitution=rbs.FORWARD, fmt=rbs.FMT_CSR, opts=rbs.options(host_only=1))
    dim = plan.export("la_dim")
    if len(dim) == 0:
        return None
    assert len(plan.export("la_rec")) * 4 == len(plan.export("la_tab")) // 4 * int(dim[7])
    return len(plan.export("la_tab")) // 4 * int(dim[7])


def csr_bytes(systems):
    return sum(12 * len(ci) + 4 * len(rp) for rp, ci, _ in systems)


def diagonals(n, bw):
    """Every row reads its last bw rows: one row a level."""
    row = np.arange(n)
    cols = row[:, None] - np.arange(bw, -1, -1)[None, :]
    keep = cols >= 0
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    ci = cols[keep].astype(np.int32)
    return rp, ci, np.where(ci == np.repeat(row, keep.sum(1)), 2.0 * bw, -1.0)


@pytest.mark.parametrize("make", [
    lambda: [diagonals(20000, 16)], lambda: [diagonals(20000, 9)],
    lambda: [rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=60000, lam=10, band=24, seed=3)]])
def test_layouts_many_times_the_matrix_are_refused(make):
    assert layout_bytes(make()) is None


@pytest.mark.parametrize("n,lam,band", [(16384, 6, 512), (60000, 12, 128), (60000, 4, 128), (200003, 8, 1024)])
def test_ordinary_bands_keep_theirs(n, lam, band):
    L = [rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=n, lam=lam, band=band, seed=n)]
    assert layout_bytes(L) <= max(8 * csr_bytes(L), 16e6)


def test_a_batch_keeps_its():
    L = [rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=n, lam=8, band=256, seed=n) for n in (1000, 1700, 4000, 11000, 26000)]
    assert layout_bytes(L) <= max(8 * csr_bytes(L), 16e6)


def test_small_matrices_keep_theirs():
    L = [diagonals(3000, 9)]
    assert 8 * csr_bytes(L) < layout_bytes(L) <= 16e6
