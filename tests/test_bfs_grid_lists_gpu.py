"""Searches of the cooperative kernel that go from lists straight to a
bottom-up level on graphs with long rows: two counts (words with an unvisited
row, unvisited long rows) then follow each other within one level. Levels,
parents, and the directions of the host-driven loop, many times over."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def grid_only():
    # (a level past any depth: keeps small graphs off the cluster kernel)
    ab.debug_device_waits(withhold_level=1 << 29)
    yield
    ab.debug_device_waits()


@pytest.mark.parametrize("n,deg,long_row", [(20_011, 12, 8), (300_007, 20, 16), (1_700_003, 8, 6)])
def test_lists_then_a_pull_with_long_rows(n, deg, long_row):
    rng = np.random.default_rng(n)
    g = ab.csr_from_edges(n, rng.integers(0, n, n * deg // 2), rng.integers(0, n, n * deg // 2))
    roots = rng.integers(0, n, 2)
    with ab.Graph(g) as dg:
        dg.sell_build(32, 1024, long_row)
        for root in roots:
            olv, opa, nl = oracle.bfs(g.rowptr, g.col, int(root))
            # the first pull after one, two, or more list levels
            for opts in ({"policy": "bottomup"}, {"policy": "beamer", "alpha": 1e4, "beta": 1e4},
                         {"policy": "beamer", "alpha": 500.0}, {"policy": "beamer"}):
                want = dg.bfs(int(root), ab.bfs_opts(loop="host", **opts))[2]
                for _ in range(10):
                    lv, pa, st = dg.bfs(int(root), ab.bfs_opts(loop="graph", **opts))
                    assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
                    assert (st.num_levels, st.levels_topdown, st.levels_bottomup) == \
                        (nl, want.levels_topdown, want.levels_bottomup)
