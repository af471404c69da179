"""The cooperative batched search against the oracle, bit for bit, at the sizes
where it can go wrong: fewer words than warps, wide slices shared by teams of
warps and slices narrower than those, long rows, frontier rows pushed in
chunks, directed graphs, more levels than the output tiles or the snapshot
store hold, and a barrier whose wait runs out."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _check(g, dg, roots, opts=None):
    lv, st = dg.msbfs64(roots, opts)
    ref = np.stack([oracle.bfs(g.rowptr, g.col, int(r))[0] for r in roots], axis=1)
    assert np.array_equal(lv[:, :len(roots)], ref) and np.all(lv[:, len(roots):] == -1)
    deg = np.diff(g.rowptr)
    assert st.reached == int((ref >= 0).sum())
    assert st.edges == int(sum(deg[ref[:, i] >= 0].sum() for i in range(len(roots))))
    return st


def _hubs(n, m, seed, sizes=()):
    """Random graph with one vertex of each given degree (about)."""
    rng = np.random.default_rng(seed)
    u, v = [rng.integers(0, n, m)], [rng.integers(0, n, m)]
    for h, k in enumerate(sizes):
        u.append(np.full(k, h * 97 % n))
        v.append(rng.choice(n, k, replace=False))
    return ab.csr_from_edges(n, np.concatenate(u), np.concatenate(v))


@pytest.mark.parametrize("n", [1, 31, 33, 1025, 5003, 150_001, 170_000])
@pytest.mark.parametrize("k", [1, 37, 64])
def test_sizes(n, k):
    # 170,000 vertices: more words than the launch has warps
    g = _hubs(n, 3 * n, n, (n // 3, n // 5) if n > 4000 else ())
    roots = np.random.default_rng(k).integers(0, n, k).astype(np.int32)  # (duplicates too)
    with ab.Graph(g) as dg:
        dg.sell_build()
        for policy in ("beamer", "bottomup") if n > 100_000 else \
                ("beamer", "topdown", "bottomup", "bottomup_nobypass", "learned"):
            st = _check(g, dg, roots, ab.bfs_opts(policy))
            assert st.kernels == 2
        host = dg.msbfs64(roots, ab.bfs_opts("beamer", "host"))[1]
        st = dg.msbfs64(roots, ab.bfs_opts("beamer"))[1]
        assert (st.num_levels, st.levels_topdown, st.levels_bottomup, st.pushed_roots) == \
            (host.num_levels, host.levels_topdown, host.levels_bottomup, host.pushed_roots)


@pytest.mark.parametrize("C_,sigma,long_row", [(32, 1024, 1024), (64, 1024, 0), (32, 96, 130),
                                               (16, 256, 1024), (32, 1, 64)])
def test_wide_slices_and_long_rows(C_, sigma, long_row, monkeypatch):
    # rows either side of the widths that teams share (128) and of the chunks
    # that long rows (1024) and long frontier rows (256) are cut into
    sizes = (127, 128, 129, 132, 255, 257, 512, 1000, 1023, 1025, 3000, 9000)
    g = _hubs(20_011, 30_000, 3, sizes)
    roots = g.pick_roots(64, 5)
    with ab.Graph(g) as dg:
        dg.sell_build(C_, sigma, long_row)
        for div in ("64", "1", "0"):
            monkeypatch.setenv("ALB_MS_PUSH_DIV", div)
            for policy in ("beamer", "bottomup", "ref004"):
                for r in (roots, roots[:9]):
                    _check(g, dg, r, ab.bfs_opts(policy))


def test_directed():
    g = _hubs(9000, 20_000, 8, (4000, 600))
    keep = np.random.default_rng(1).random(g.col.size) < 0.6
    src = np.repeat(np.arange(g.n), np.diff(g.rowptr))[keep]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=g.n))]).astype(np.int64)
    out = ab.Csr(rowptr, g.col[keep].astype(np.int32))
    roots = np.arange(0, 9000, 150, dtype=np.int32)
    with ab.Graph(out, ab.CSR_OUT) as dg:
        dg.sell_build()
        want, _ = dg.msbfs64(roots, ab.bfs_opts("beamer", "host"))
        for policy in ("beamer", "topdown", "bottomup"):
            assert np.array_equal(dg.msbfs64(roots, ab.bfs_opts(policy))[0], want)


@pytest.mark.parametrize("n", [15, 17, 32, 33, 34, 65])
def test_level_counts_of_output_and_store(n):
    # a path: 16 levels fit the output tiles, 32 the snapshot store
    u = np.arange(n - 1)
    g = ab.csr_from_edges(n, u, u + 1)
    with ab.Graph(g) as dg:
        dg.sell_build()
        for roots in ([0], [0, n - 1], [n // 2]):
            for policy in ("beamer", "topdown", "bottomup"):
                _check(g, dg, np.array(roots, np.int32), ab.bfs_opts(policy))


def test_a_wait_that_runs_out():
    g = _hubs(5000, 15_000, 2)
    roots = g.pick_roots(64, 1)
    with ab.Graph(g) as dg:
        dg.sell_build()
        for level, block in ((-1, 0), (0, 3), (1, 0), (2, 151)):
            if level >= 0:
                ab.debug_device_waits(withhold_level=level, withhold_block=block, timeout_us=50_000)
                try:
                    with pytest.raises(ab.AlbError) as ei:
                        dg.msbfs64(roots)
                finally:
                    ab.debug_device_waits()
                assert ei.value.code == ab.ERR_TIMEOUT
            _check(g, dg, roots)
