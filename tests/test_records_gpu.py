"""The push rows' records of the cooperative search are optional: without
memory for them a search runs without, and says nothing of it."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def test_a_search_without_memory_for_records_leaves_no_message():
    g = ab.gen_er(100_003, 8.0, seed=4)  # (no row over 64: searched with records)
    olv, opa, _ = oracle.bfs(g.rowptr, g.col, 5)
    with ab.Graph(g) as dg:
        dg.sell_build()
        # everything but the records is allocated here
        dg.bfs(5, ab.bfs_opts("beamer", "graph", trace=True))
        with pytest.raises(ab.AlbError):
            dg.bfs(g.n)
        said = ab.last_error()
        assert said and "records" not in said
        for fail in (1, 0):
            ab.debug_fail_alloc_after(fail)
            try:
                lv, pa, _ = dg.bfs(5)
            finally:
                ab.debug_fail_alloc_after(0)
            assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
            assert ab.last_error() == said
