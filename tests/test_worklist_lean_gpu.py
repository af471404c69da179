"""Work-list graphs whose bitmaps fill a CTA's shared memory (about 540,000 to
617,000 vertices): few items run one by one on the single-root path, many in
the kernel without the push's lists, beside items of smaller graphs. Levels
against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _run(parts):
    wl, csrs = ab.Worklist(), []
    for g, roots, opts in parts:
        dg = ab.Graph(g)
        dg.sell_build(*opts)
        wl.add(dg, np.asarray(roots, np.int32))
        csrs.append(g)
    levels, st = wl.run(256)
    want = {}
    for lv, (gi, root, _) in zip(levels, wl.layout):
        if (gi, root) not in want:
            want[gi, root] = oracle.bfs(csrs[gi].rowptr, csrs[gi].col, root)[0]
        assert np.array_equal(lv, want[gi, root]), (gi, root)
    return st


def _hubs(n, seed):
    """Uniform random with two hubs and, for one, a way in over its last neighbour."""
    rng = np.random.default_rng(seed)
    u, v = [rng.integers(100, n - 9000, 2 * n)], [rng.integers(100, n - 9000, 2 * n)]
    for h, k in ((0, 60_000), (1, 3000)):
        u.append(np.full(k, h))
        v.append(rng.choice(np.arange(100, n - 9000), k, replace=False))
    u += [np.full(4001, 2), np.array([n - 1])]
    v += [np.concatenate([np.arange(n - 9000, n - 5000), [n - 1]]), np.array([100])]
    return ab.csr_from_edges(n, np.concatenate(u), np.concatenate(v))


@pytest.mark.parametrize("opts", [(32, 1024, 1024), (16, 64, 40), (64, 16384, 0)])
def test_many_items_in_the_kernel(opts):
    n = 600_011
    g = _hubs(n, 3)
    roots = [0, 2, 100, n - 1, n - 5500]
    st = _run([(g, np.resize(roots, 60), opts), (ab.gen_rmat(10, 8, seed=1), range(8), opts)])
    assert st.kernels == 2  # with and without the lists


def test_the_largest_graphs_and_few_items():
    # 617,120 vertices: the most that fit, the next word does not
    for n, kernels in ((617_120, 1), (617_121, None)):
        g = ab.gen_er(n, 4.0, seed=2)
        st = _run([(g, np.resize(g.pick_roots(3, 1), 50), (32, 1024, 1024))])
        assert st.kernels == kernels if kernels else st.kernels >= 50
    g = ab.gen_er(560_000, 4.0, seed=2)
    st = _run([(g, g.pick_roots(3, 1), (32, 1024, 1024)), (ab.gen_rmat(8, 8, seed=1), [3], (32, 1024, 1024))])
    assert st.kernels > 3  # one by one, and the kernel
