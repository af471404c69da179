"""The work-list kernel's three thread counts, graphs around a bitmap word and
the largest that fits, hub rows, and long rows without a source in the frontier
in their first 1024: every item's levels equal the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _run(parts, block):
    wl, csrs = ab.Worklist(), []
    for g, roots, opts in parts:
        dg = ab.Graph(g)
        dg.sell_build(*opts)
        wl.add(dg, np.asarray(roots, np.int32))
        csrs.append(g)
    levels, st = wl.run(block)
    assert st.kernels == 1
    for lv, (gi, root, _) in zip(levels, wl.layout):
        ref = oracle.bfs(csrs[gi].rowptr, csrs[gi].col, root)[0]
        assert np.array_equal(lv, ref), (gi, root)


def _random(n, seed):
    rng = np.random.default_rng(seed)
    return ab.csr_from_edges(n, rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n))


def test_small_graphs_256_threads():
    _run([(_random(n, n), [0, n - 1], (32, 1024, 16)) for n in (1, 2, 31, 32, 33, 1000, 1024)], 256)


def test_many_items_512_threads():
    _run([(_random(40 + 37 * i, i), range(8), (32, 256, 8)) for i in range(77)], 256)


@pytest.mark.parametrize("opts", [(32, 1024, 1024), (16, 64, 40), (64, 16384, 0)])
def test_hubs_and_long_rows_1024_threads(opts):
    n = 30011
    rng = np.random.default_rng(3)
    u, v = [rng.integers(100, n - 5000, 60000)], [rng.integers(100, n - 5000, 60000)]
    for h in (0, 1):
        t = rng.choice(np.arange(100, n - 5000), 15000, replace=False)
        u.append(np.full(t.shape, h))
        v.append(t)
    # vertex 2: 4,000 leaves and one way in, over its largest neighbour
    u += [np.full(4001, 2), np.array([n - 1])]
    v += [np.concatenate([np.arange(n - 5000, n - 1000), [n - 1]]), np.array([100])]
    g = ab.csr_from_edges(n, np.concatenate(u), np.concatenate(v))
    _run([(g, [0, 100, n - 1, n - 4000, n - 500], opts), (_random(4097, 1), [5], opts)], 128)


def test_largest_graph_that_fits():
    g = ab.gen_er(530_000, 6.0, seed=2)
    _run([(g, g.pick_roots(2, 1), (32, 1024, 1024))], 512)


def test_frontiers_around_the_push_list_and_reuse_of_the_work_list():
    """Top-down frontiers just under and over what the push lists at once (2,048
    rows), spread over a large graph's words, and runs of one list one after
    the other while items are added."""
    n = 60_000
    rng = np.random.default_rng(9)
    wl, csrs = ab.Worklist(), []
    for k in (2047, 2048, 2049, 5000):
        # a star of k spokes with a leaf on each, ids shuffled
        ids = rng.permutation(n)
        spokes, leaves = ids[1:k + 1], ids[k + 1:2 * k + 1]
        g = ab.csr_from_edges(n, np.concatenate([np.full(k, ids[0]), spokes]),
                              np.concatenate([spokes, leaves]))
        dg = ab.Graph(g)
        dg.sell_build()
        wl.add(dg, np.array([ids[0], leaves[0]], np.int32), alpha=1e-3)  # (top-down throughout)
        csrs.append(g)
        for _ in range(2):
            levels, _ = wl.run(256)
            for lv, (gi, root, _) in zip(levels, wl.layout):
                assert np.array_equal(lv, oracle.bfs(csrs[gi].rowptr, csrs[gi].col, int(root))[0])
