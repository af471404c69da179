"""The cooperative single-root kernel (graphs past the cluster kernel's size)
against the oracle, bit for bit, at the sizes where it can go wrong: fewer
words than warps or blocks, both bottom-up shapes, the frontier staged in
shared memory and not, every change of a frontier's form, hub and long rows,
output tiles of every window size. A barrier-withholding level past any
depth keeps small graphs off the cluster kernel without changing a run."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def grid_only():
    ab.debug_device_waits(withhold_level=1 << 29)
    yield
    ab.debug_device_waits()


def _check(g, dg, root, opts, push=None):
    lv, pa, st = dg.bfs(int(root), opts)
    olv, opa, nl = oracle.bfs(g.rowptr, g.col, int(root)) if push is None else \
        oracle.bfs(push.rowptr, push.col, int(root), g.rowptr, g.col)
    assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
    assert st.num_levels == nl and st.reached == int((olv >= 0).sum())
    assert st.edges == int(np.diff((push or g).rowptr)[olv >= 0].sum())
    return st


def _random(n, m, seed, hubs=0):
    rng = np.random.default_rng(seed)
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    for h in range(hubs):
        t = rng.choice(n, n // 2, replace=False)
        u, v = np.concatenate([u, np.full(t.shape, h)]), np.concatenate([v, t])
    return ab.csr_from_edges(n, u, v)


@pytest.mark.parametrize("n", [1, 33, 1000, 5003, 40001, 300007, 1 << 20, 1572864])
def test_sizes_every_policy(n):
    g = _random(n, 4 * n, n, hubs=2 if 4000 < n < 500000 else 0)
    with ab.Graph(g) as dg:
        dg.sell_build()
        for policy in ("beamer", "topdown", "bottomup", "ref004", "learned"):
            for loop in ("graph", "persistent"):
                for r in [0, n // 2][:1 if n > 100000 else 2]:
                    _check(g, dg, r, ab.bfs_opts(policy, loop))
        a = dg.bfs(0, ab.bfs_opts("beamer", "graph"))[2]
        b = dg.bfs(0, ab.bfs_opts("beamer", "host"))[2]
        assert (a.levels_topdown, a.levels_bottomup) == (b.levels_topdown, b.levels_bottomup)


@pytest.mark.parametrize("kind", ["grid", "er", "rmat"])
def test_unstaged_and_long_searches(kind):
    """Past the staging limit (1,572,864 vertices); the grid's hundreds of
    list levels, evened out over the blocks."""
    g = {"grid": lambda: ab.gen_grid(1300, 1300, 0.1, 1e-4, seed=5),
         "er": lambda: ab.gen_er(1_700_003, 8.0, seed=5),
         "rmat": lambda: ab.gen_rmat(21, 8, seed=5)}[kind]()
    with ab.Graph(g) as dg:
        dg.sell_build()
        for r in g.pick_roots(2, 3):
            for policy in ("beamer", "topdown", "learned"):
                _check(g, dg, r, ab.bfs_opts(policy, "persistent"))


@pytest.mark.parametrize("C_,sigma,long_row", [(32, 1, 64), (8, 3, 8), (64, 1000, 300),
                                               (16, 16384, 0), (32, 4096, 40)])
def test_windows_hub_and_long_rows(C_, sigma, long_row):
    n = 30011
    rng = np.random.default_rng(3)
    u, v = [rng.integers(100, n - 5000, 60000)], [rng.integers(100, n - 5000, 60000)]
    for h in (0, 1):
        t = rng.choice(np.arange(100, n - 5000), 15000, replace=False)
        u.append(np.full(t.shape, h))
        v.append(t)
    u += [np.full(4001, 2), np.array([n - 1])]
    v += [np.concatenate([np.arange(n - 5000, n - 1000), [n - 1]]), np.array([100])]
    g = ab.csr_from_edges(n, np.concatenate(u), np.concatenate(v))
    with ab.Graph(g) as dg:
        dg.sell_build(C_, sigma, long_row)
        for root in (0, 100, n - 1, n - 4000, n - 500):
            for policy in ("beamer", "topdown", "bottomup"):
                _check(g, dg, root, ab.bfs_opts(policy))


def test_directed_and_unaligned_outputs():
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
            _check(pull, dg, 7, ab.bfs_opts(policy), push)
        olv, opa, _ = oracle.bfs(push.rowptr, push.col, 7, pull.rowptr, pull.col)
        out = torch.full((2 * n + 3,), 77, dtype=torch.int32, device="cuda")
        dg.bfs_device(7, out[1:n + 1], out[n + 2:2 * n + 2])
        h = out.cpu().numpy()
        assert np.array_equal(h[1:n + 1], olv) and np.array_equal(h[n + 2:2 * n + 2], opa)
        assert h[0] == h[n + 1] == h[-1] == 77
        assert dg.bfs_device(7).reached == int((olv >= 0).sum())


@pytest.mark.parametrize("sizes", [(5000, 300, 257, 256, 255, 3), (257, 5000, 256, 1000, 258)])
def test_big_rows_known_before_their_push(sizes):
    """A chain of hubs either side of the length that is pushed in chunks
    (256), reached from lists, queues and bottom-up levels' bitmaps."""
    n = 20_011
    ids = np.random.default_rng(4).permutation(n)
    hubs, rest, u, v = ids[:len(sizes)], ids[len(sizes):], [], []
    for i, k in enumerate(sizes):
        u.append(np.full(k, hubs[i]))
        v.append(rest[:k])
        rest = rest[k:]
    u.append(hubs[:-1])
    v.append(hubs[1:])
    g = ab.csr_from_edges(n, np.concatenate(u), np.concatenate(v))
    with ab.Graph(g) as dg:
        dg.sell_build()
        for root in (hubs[0], hubs[-1], int(v[0][0])):
            _check(g, dg, root, ab.bfs_opts("topdown"))
            _check(g, dg, root, ab.bfs_opts("ref004"))
            for alpha, beta in ((14.0, 24.0), (1e6, 0.5), (200.0, 2.0)):
                _check(g, dg, root, ab.bfs_opts("beamer", alpha=alpha, beta=beta))


@pytest.mark.parametrize("arity,depth", [(2, 17), (3, 11), (15, 4), (15, 5)])
def test_claims_past_a_lists_rows(arity, depth):
    """Trees: a block's list of up to 5,952 edges (rows of at most 16) claims as
    many rows, three times what the next list has room for."""
    n = (arity ** (depth + 1) - 1) // (arity - 1)
    child = np.arange(1, n)
    ids = np.random.default_rng(6).permutation(n)
    for perm in (np.arange(n), ids):
        g = ab.csr_from_edges(n, perm[(child - 1) // arity], perm[child])
        with ab.Graph(g) as dg:
            dg.sell_build()
            for root in (perm[0], perm[1], perm[n - 1]):
                for policy in ("topdown", "beamer", "learned", "ref004"):
                    _check(g, dg, root, ab.bfs_opts(policy, "persistent"))
