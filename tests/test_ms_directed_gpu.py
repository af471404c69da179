"""The batched search of directed graphs against the oracle (push rows and pull
rows differ, in length too), on the kernel of the default loop and the host's."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _directed(n, m, seed, hubs):
    rng = np.random.default_rng(seed)
    u, v = [rng.integers(0, n, m)], [rng.integers(0, n, m)]
    for h, (out, into) in enumerate(hubs):
        u += [np.full(out, h), rng.choice(n, into, replace=False)]
        v += [rng.choice(n, out, replace=False), np.full(into, h)]
    u, v = np.concatenate(u), np.concatenate(v)
    key = np.unique((u * n + v)[u != v])
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return ab.Csr(rp, (key % n).astype(np.int32))


@pytest.mark.parametrize("long_row", [1024, 40])
@pytest.mark.parametrize("n,m", [(9000, 30_000), (170_003, 500_000)])
def test_directed(n, m, long_row):
    push = _directed(n, m, n, ((4000, 3), (2, 5000), (300, 1500)))
    roots = np.concatenate([[0, 1, 2], np.arange(3, n, n // 30)])[:33].astype(np.int32)
    with ab.Graph(push, ab.CSR_OUT) as dg:
        dg.sell_build(32, 1024, long_row)
        pull = dg.export_csr(0)
        want = np.stack([oracle.bfs(push.rowptr, push.col, int(r), pull.rowptr, pull.col)[0]
                         for r in roots], axis=1)
        deg = np.diff(push.rowptr)
        for policy, loop in (("beamer", "graph"), ("topdown", "graph"), ("bottomup", "graph"),
                             ("beamer", "host")):
            lv, st = dg.msbfs64(roots, ab.bfs_opts(policy, loop))
            assert np.array_equal(lv[:, :len(roots)], want) and np.all(lv[:, len(roots):] == -1)
            assert st.reached == int((want >= 0).sum())
            assert st.edges == int(sum(deg[want[:, i] >= 0].sum() for i in range(len(roots))))
