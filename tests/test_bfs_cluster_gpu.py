"""Graphs small enough for the one-launch cluster BFS: levels, parents and
statistics bit-exact against the oracle, at the edges of its shapes -- vertex
counts around a bitmap word, around each cluster size, the largest one taken
and the first one not taken -- and at the branches inside a level: hub rows
split over the CTAs or shared by one, wide frontiers, long rows with and
without a hit in their head, directed graphs."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _check(g, dg, root, opts, push=None):
    lv, pa, st = dg.bfs(int(root), opts)
    olv, opa, nl = oracle.bfs(g.rowptr, g.col, int(root)) if push is None else \
        oracle.bfs(push.rowptr, push.col, int(root), g.rowptr, g.col)
    assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
    assert st.num_levels == nl and st.reached == int((olv >= 0).sum())
    deg = np.diff((push or g).rowptr)
    assert st.edges == int(deg[olv >= 0].sum())
    return st


def _random(n, m, seed, hubs=0):
    """n vertices, m random undirected edges, and `hubs` vertices joined to
    half of all."""
    rng = np.random.default_rng(seed)
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    for h in range(hubs):
        t = rng.choice(n, n // 2, replace=False)
        u, v = np.concatenate([u, np.full(t.shape, h)]), np.concatenate([v, t])
    return ab.csr_from_edges(n, u, v)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 1024, 1025, 2049, 4097, 8191, 16385, 40001,
                               (1 << 16) - 1, 1 << 16, (1 << 16) + 1])
def test_sizes_every_policy(n):
    g = _random(n, 4 * n, n, hubs=2 if n > 4000 else 0)
    roots = [0, n // 2, n - 1]
    with ab.Graph(g) as dg:
        dg.sell_build()
        for policy in ("beamer", "topdown", "bottomup", "ref004", "learned"):
            for loop in ("graph", "persistent"):
                for r in roots[:1 if n > 40000 else 3]:
                    st = _check(g, dg, r, ab.bfs_opts(policy, loop))
                    if policy == "topdown":
                        assert st.levels_bottomup == 0
        # the loops that were there before give the same directions
        a = dg.bfs(roots[0], ab.bfs_opts("beamer", "graph"))[2]
        b = dg.bfs(roots[0], ab.bfs_opts("beamer", "host"))[2]
        assert (a.levels_topdown, a.levels_bottomup) == (b.levels_topdown, b.levels_bottomup)


@pytest.mark.parametrize("C_,sigma,long_row", [(32, 1024, 64), (8, 64, 8), (64, 16384, 300),
                                               (16, 1, 0)])
def test_hub_and_long_rows(C_, sigma, long_row):
    # two hubs of 15,000 and paths of long rows: heads without a hit (a hub is
    # reached only over its last source) and rows over the CTA's list
    n = 30011
    rng = np.random.default_rng(3)
    u, v = [rng.integers(100, n - 5000, 60000)], [rng.integers(100, n - 5000, 60000)]
    for h in (0, 1):
        t = rng.choice(np.arange(100, n - 5000), 15000, replace=False)
        u.append(np.full(t.shape, h))
        v.append(t)
    # vertex 2: 4,000 leaves and one way in, over its largest neighbour
    u.append(np.full(4001, 2))
    v.append(np.concatenate([np.arange(n - 5000, n - 1000), [n - 1]]))
    u.append(np.array([n - 1]))
    v.append(np.array([100]))
    g = ab.csr_from_edges(n, np.concatenate(u), np.concatenate(v))
    with ab.Graph(g) as dg:
        dg.sell_build(C_, sigma, long_row)
        for root in (0, 100, n - 1, n - 4000, n - 500):
            for policy in ("beamer", "topdown", "bottomup"):
                _check(g, dg, root, ab.bfs_opts(policy))


def test_directed_and_device_outputs():
    import torch
    n = 5000
    rng = np.random.default_rng(9)
    src, dst = rng.integers(0, n, 30000), rng.integers(0, n, 30000)
    keep = src != dst
    key = np.unique(src[keep].astype(np.int64) * n + dst[keep])
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    push = ab.Csr(rp, (key % n).astype(np.int32))
    with ab.Graph(push, ab.CSR_OUT) as dg:
        dg.sell_build()
        pull = dg.export_csr(0)
        for policy in ("beamer", "topdown", "bottomup"):
            st = _check(pull, dg, 7, ab.bfs_opts(policy), push)
        lv = torch.empty(n, dtype=torch.int32, device="cuda")
        st2 = dg.bfs_device(7, lv, None)  # no parents wanted
        olv = oracle.bfs(push.rowptr, push.col, 7, pull.rowptr, pull.col)[0]
        assert np.array_equal(lv.cpu().numpy(), olv) and st2.reached == st.reached
        assert dg.bfs_device(7).reached == st.reached  # nothing wanted
