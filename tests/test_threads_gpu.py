"""Two threads, each with graphs and work lists of its own, whose launches of one
kernel need different amounts of shared memory: neither one's limit is the
other's."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _both(a, b):
    """a and b on a thread each, at once; whatever they raised."""
    errs, start = [], threading.Barrier(2)

    def run(f):
        try:
            start.wait()
            f()
        except BaseException as e:  # noqa: BLE001
            errs.append(e)

    ts = [threading.Thread(target=run, args=(f,)) for f in (a, b)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errs, errs


def _repeat_list(g, roots, times):
    dg = ab.Graph(g)
    dg.sell_build()
    wl = ab.Worklist()
    wl.add(dg, np.asarray(roots, np.int32))
    want = [oracle.bfs(g.rowptr, g.col, int(r))[0] for r in roots]

    def run():
        for _ in range(times):
            levels, _ = wl.run(256)
            assert all(np.array_equal(lv, w) for lv, w in zip(levels, want))
    return run


def test_work_lists_of_large_and_small_graphs():
    _both(_repeat_list(ab.gen_er(500_000, 4.0, seed=1), [0, 9], 60),
          _repeat_list(ab.gen_rmat(12, 8, seed=1), [1, 5], 2000))


def test_searches_with_large_and_small_output_tiles():
    def search(sigma, times):
        g = ab.gen_er(100_003, 6.0, seed=sigma)
        dg = ab.Graph(g)
        dg.sell_build(32, sigma)
        olv, opa, _ = oracle.bfs(g.rowptr, g.col, 3)

        def run():
            for _ in range(times):
                lv, pa, _ = dg.bfs(3)
                assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
            assert ab.last_error() == ""  # (the thread's own)
        return run
    _both(search(16384, 300), search(8192, 300))
