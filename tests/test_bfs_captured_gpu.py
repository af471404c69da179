"""A search asked for while its stream is being captured into a CUDA graph is
refused (every call waits for its stream), and leaves nothing behind that a
later search on the same graph would take for made: neither the push rows'
records nor the barrier counter's zero, whose kernel and memset were captured
and have not run."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _refused(dg, n, stream):
    """One search while `stream` is being captured."""
    import torch
    level = torch.empty(n, dtype=torch.int32, device="cuda")
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="relaxed")
        try:
            with pytest.raises(ab.AlbError):
                dg.bfs_device(0, level, None)
        finally:
            with pytest.raises(RuntimeError):  # (the wait ended the capture)
                graph.capture_end()
    torch.cuda.synchronize()


@pytest.mark.parametrize("scratch", [True, False])
def test_a_search_under_capture_is_refused_and_the_next_is_right(scratch):
    """scratch: the graph has been searched before, by a kernel without records."""
    import torch
    g = ab.gen_er(100_003, 8.0, seed=4)  # (no row over 64: searched with records)
    stream = torch.cuda.Stream()
    with ab.Graph(g) as dg:
        dg.sell_build()
        if scratch:
            dg.bfs(0, ab.bfs_opts("beamer", "graph", trace=True))
        dg.set_stream(stream.cuda_stream)
        _refused(dg, g.n, stream)
        dg.set_stream(None)
        for root in (0, 77, g.n - 1):
            lv, pa, _ = dg.bfs(root)
            olv, opa, _ = oracle.bfs(g.rowptr, g.col, root)
            assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
