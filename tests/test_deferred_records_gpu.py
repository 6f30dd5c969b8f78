"""Level-chunk records of plans that leave them out until they are asked for:
exports and saves from several threads at once give the records of a plan
that built them at once."""
import threading

import numpy as np
import pytest

import rbs

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def test_exports_and_saves_from_several_threads(tmp_path):
    L = rbs.gen_lower_csr(rbs.GEN_BAND_POISSON, n=120000, lam=8, band=1024, seed=3)
    kw = dict(substitution=rbs.FORWARD, lv=1, fmt=rbs.FMT_CSR)
    names = ("lc_rec64", "lc_rec32", "lc_tab", "lc_segs")
    want = rbs.analyse(*L, opts=rbs.options(host_only=1), **kw)
    want = {q: want.export(q) for q in names}
    assert all(len(v) for v in want.values())
    plan = rbs.analyse(*L, **kw)
    assert plan.export("walk")[0] == 1
    start, bad = threading.Barrier(6), []

    def work(i):
        start.wait()
        try:
            if i % 3 == 2:
                plan.save(tmp_path / f"p{i}")
            else:
                bad.extend((i, q) for q in names if not np.array_equal(plan.export(q), want[q]))
        except Exception as e:  # reported by the assertion below
            bad.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    assert (tmp_path / "p2").read_bytes() == (tmp_path / "p5").read_bytes()
    loaded = rbs.load_plan(tmp_path / "p2", opts=rbs.options(host_only=1))
    assert all(np.array_equal(loaded.export(q), want[q]) for q in names)
