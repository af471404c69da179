"""A search asked for while its stream is being captured into a CUDA graph is
refused (every call waits for its stream), and leaves nothing behind that a
later search on the same graph would take for made: neither the push rows'
records nor the barrier counter's zero, whose kernel and memset were captured
and have not run."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


RELAXED = 2  # (CU_STREAM_CAPTURE_MODE_RELAXED)


def _refused(dg, n, stream):
    """One search while `stream` is being captured (by the driver's API: a capture
    of torch's that fails leaves its random numbers unusable)."""
    import torch
    cu = C.CDLL("libcuda.so.1")
    level = torch.empty(n, dtype=torch.int32, device="cuda")
    h, graph = C.c_void_p(stream.cuda_stream), C.c_void_p()
    torch.cuda.synchronize()
    assert cu.cuStreamBeginCapture_v2(h, RELAXED) == 0
    try:
        with pytest.raises(ab.AlbError):
            dg.bfs_device(0, level, None)
    finally:
        # (the wait ended the capture)
        assert cu.cuStreamEndCapture(h, C.byref(graph)) != 0
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
