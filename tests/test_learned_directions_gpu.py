"""The learned policy with weights installed, on every one-kernel search. On the
default loop its features are the same numbers whichever form a frontier has,
so the directions it takes are those of the host-driven loop, which decides
from the counters of every level. (The persistent loop counts the words with an
unvisited row when it leaves its lists.) Levels and parents against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle
from albba_gb300 import selector

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def weights():
    selector.install()
    yield
    ab.selector_clear(0)
    ab.selector_clear(1)


GRAPHS = {
    "rmat10": lambda: ab.gen_rmat(10, 16, seed=26), "rmat12": lambda: ab.gen_rmat(12, 4, seed=16),
    "rmat16": lambda: ab.gen_rmat(16, 16, seed=32), "rmat18": lambda: ab.gen_rmat(18, 8, seed=3),
    "er3000": lambda: ab.gen_er(3000, 8.0, seed=5), "er60000": lambda: ab.gen_er(60_000, 3.0, seed=5),
    "er200003": lambda: ab.gen_er(200_003, 3.0, seed=5),
    "grid100": lambda: ab.gen_grid(100, 100, 0.1, 1e-4, seed=100),
    "grid250": lambda: ab.gen_grid(250, 250, 0.1, 1e-4, seed=250),
    "grid600": lambda: ab.gen_grid(600, 600, 0.1, 1e-4, seed=600),
    "path": lambda: ab.csr_from_edges(3001, np.arange(3000), np.arange(1, 3001)),
}


def _directions(dg, root, loop):
    lv, pa, st = dg.bfs(int(root), ab.bfs_opts("learned", loop))
    return lv, pa, (st.num_levels, st.levels_topdown, st.levels_bottomup, st.reached, st.edges)


@pytest.mark.parametrize("kernel", ["by size", "cooperative"])
@pytest.mark.parametrize("name", GRAPHS)
def test_single_root(name, kernel):
    g = GRAPHS[name]()
    if kernel == "cooperative":
        # a level past any depth keeps small graphs off the cluster kernel
        ab.debug_device_waits(withhold_level=1 << 29)
    try:
        with ab.Graph(g) as dg:
            dg.sell_build()
            for root in g.pick_roots(4, 1):
                olv, opa, _ = oracle.bfs(g.rowptr, g.col, int(root))
                want = _directions(dg, root, "host")[2]
                for loop in ("graph", "persistent"):
                    lv, pa, got = _directions(dg, root, loop)
                    assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
                    assert got == want if loop == "graph" else got[0::3] == want[0::3]
    finally:
        ab.debug_device_waits()


@pytest.mark.parametrize("name", GRAPHS)
def test_batched(name):
    g = GRAPHS[name]()
    roots = g.pick_roots(19, 3)
    with ab.Graph(g) as dg:
        dg.sell_build()
        got = {}
        for loop in ("host", "graph"):
            lv, st = dg.msbfs64(roots, ab.bfs_opts("learned", loop))
            got[loop] = (st.num_levels, st.levels_topdown, st.levels_bottomup, st.pushed_roots)
            for i in (0, 18):
                assert np.array_equal(lv[:, i], oracle.bfs(g.rowptr, g.col, int(roots[i]))[0])
        assert got["host"] == got["graph"]
