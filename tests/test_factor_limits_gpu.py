"""ILU(0) and IC(0) when a wait of the level search runs out of polls: the call
returns RBS_ERR_TIMEOUT before any factor kernel is launched (the output is
untouched), and the next call with the default limit gives the serial factor
bit for bit.  The matrix is a chain, whose 32-row groups wait for one another
in turn, so that most of them poll far more often than the limit set here.
And ILU(0) of arrays that hold more entries than the matrix."""
import numpy as np
import pytest

import rbs
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def chain(n, lower_only):
    rng = np.random.default_rng(3)
    i = np.arange(n)
    cols = np.stack([i - 1, i, i + 1], 1)[:, : 2 if lower_only else 3]
    keep = (cols >= 0) & (cols < n)
    va = np.where(cols == i[:, None], 3.0, rng.uniform(-1, 1, cols.shape))[keep]
    return np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32), cols[keep].astype(np.int32), va


@pytest.mark.parametrize("ic", [False, True])
def test_level_search_out_of_polls(ic):
    n = 300000
    run, ref = (rbs.ic0_device, oracle.ic0_csr) if ic else (rbs.ilu0_device, oracle.ilu0_csr)
    rp, ci, va = chain(n, ic)
    d = [torch.tensor(a, device="cuda") for a in (rp, ci, va)]
    lu = torch.full_like(d[2], 7.0)
    with pytest.raises(rbs.RbsError) as e:
        run(*d, lu, opts=rbs.options(spin_limit=1))
    assert e.value.code == rbs.ERR_TIMEOUT and "level search" in str(e.value)
    assert bool((lu == 7.0).all())
    run(*d, lu)
    assert np.array_equal(lu.cpu().numpy(), ref(rp, ci, va))


@pytest.mark.parametrize("before,behind", [(3, 0), (0, 5), (2, 2)])
def test_entries_outside_the_rows_are_copied(before, behind):
    # arrays larger than the matrix: the factor's other entries are the matrix's own
    rp, ci, va = chain(5000, False)
    pad = lambda a, v: np.concatenate([np.full(before, v, a.dtype), a, np.full(behind, v, a.dtype)])
    d = [torch.tensor(a, device="cuda") for a in (rp + before, pad(ci, 0), pad(va, -2.5))]
    lu = torch.full_like(d[2], 7.0)
    rbs.ilu0_device(*d, lu)
    assert np.array_equal(lu.cpu().numpy(), pad(oracle.ilu0_csr(rp, ci, va), -2.5))
    rbs.ilu0_device(*d, d[2])
    assert torch.equal(d[2], lu)
