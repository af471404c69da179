"""Small graphs of many edges, either side of the entries per vertex at which
pushing policies leave the cluster kernel: levels, parents and statistics
against the oracle, and a search that is not left to a tenth of the SMs."""
from __future__ import annotations

import statistics

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


def _regular(n, d):
    """Every vertex joined to the d / 2 after it: d entries a row."""
    k = d // 2
    u = np.repeat(np.arange(n), k)
    return ab.csr_from_edges(n, u, (u + np.tile(np.arange(1, k + 1), n)) % n)


@pytest.mark.parametrize("n,d", [(1500, 98), (1500, 100), (1500, 102), (300, 298), (4000, 600)])
def test_around_the_line(n, d):
    g = _regular(n, d)
    with ab.Graph(g) as dg:
        dg.sell_build()
        for root in (0, n - 1):
            olv, opa, nl = oracle.bfs(g.rowptr, g.col, root)
            for policy in ("topdown", "learned", "beamer", "bottomup"):
                for loop in ("graph", "persistent"):
                    lv, pa, st = dg.bfs(root, ab.bfs_opts(policy, loop))
                    assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
                    assert (st.num_levels, st.reached, st.edges) == (nl, n, g.nnz)


def test_dense_pushes_use_the_whole_gpu():
    rng = np.random.default_rng(1)
    n, m = 8000, 6_400_000
    g = ab.csr_from_edges(n, rng.integers(0, n, m), rng.integers(0, n, m))
    with ab.Graph(g) as dg:
        dg.sell_build()
        us = {}
        for policy in ("topdown", "beamer"):
            t = [dg.bfs(3, ab.bfs_opts(policy), want_level=False, want_parent=False)[2].ms
                 for _ in range(9)]
            us[policy] = 1e3 * statistics.median(t)
    # about 130 us against the pulling policy's 70; on 16 SMs 510
    assert us["topdown"] < 4 * us["beamer"], us
