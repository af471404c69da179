"""The cooperative kernel where it pulls for a frontier that few rows have a
source in (bottom-up throughout, frontiers too large to stage in shared
memory), and where it pushes many edges of a small graph, from hubs and
leaves: levels and parents against the oracle."""
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


def _check(g, dg, root, policy):
    lv, pa, st = dg.bfs(int(root), ab.bfs_opts(policy))
    olv, opa, nl = oracle.bfs(g.rowptr, g.col, int(root))
    assert np.array_equal(lv, olv) and np.array_equal(pa, opa) and st.num_levels == nl


# (bitmaps are staged up to 1,572,864 vertices)
@pytest.mark.parametrize("C_,sigma,long_row", [(32, 1024, 1024), (8, 64, 40), (64, 4096, 0)])
@pytest.mark.parametrize("kind", ["rmat", "er", "edge"])
def test_bottom_up_throughout(kind, C_, sigma, long_row):
    g = {"rmat": lambda: ab.gen_rmat(21, 4, seed=5), "er": lambda: ab.gen_er(1_700_003, 6.0, seed=5),
         "edge": lambda: ab.gen_er(1_572_865, 3.0, seed=6)}[kind]()
    deg = np.diff(g.rowptr)
    leaf = int(np.flatnonzero(deg == 1)[7])
    with ab.Graph(g) as dg:
        dg.sell_build(C_, sigma, long_row)
        for root in (leaf, int(deg.argmax())):
            _check(g, dg, root, "bottomup")


@pytest.mark.parametrize("n,m", [(2000, 400_000), (33, 400), (20_001, 3_000_000), (70_001, 4_000_000)])
def test_pushes_of_many_edges(n, m):
    rng = np.random.default_rng(n)
    g = ab.csr_from_edges(n, rng.integers(0, n, m), rng.integers(0, n, m))
    with ab.Graph(g) as dg:
        dg.sell_build()
        for root in rng.integers(0, n, 3):
            for _ in range(4):
                _check(g, dg, root, "topdown")
