"""A search on the caller's stream under the default loop leaves the stream's own
L2 access-policy window as it was (read back through the driver's API)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu

ACCESS_POLICY_WINDOW = 1


class Window(C.Structure):
    _fields_ = [("base", C.c_void_p), ("bytes", C.c_size_t), ("hit_ratio", C.c_float),
                ("hit_prop", C.c_int), ("miss_prop", C.c_int)]


class Attr(C.Union):
    _fields_ = [("window", Window), ("pad", C.c_char * 64)]


def test_the_callers_window_stays():
    import torch
    cu = C.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    mine = torch.empty(1 << 20, dtype=torch.int32, device="cuda")
    want = Attr()
    want.window = Window(mine.data_ptr(), 1 << 20, 0.5, 1, 0)  # (hits streaming)
    h = C.c_void_p(stream.cuda_stream)
    assert cu.cuStreamSetAttribute(h, ACCESS_POLICY_WINDOW, C.byref(want)) == 0
    # (frontier bitmaps too large to stage have a window in L2)
    g = ab.gen_er(1_700_003, 4.0, seed=2)
    with ab.Graph(g) as dg:
        dg.sell_build()
        dg.set_stream(stream.cuda_stream)
        lv, pa, _ = dg.bfs(5)
        olv, opa, _ = oracle.bfs(g.rowptr, g.col, 5)
        assert np.array_equal(lv, olv) and np.array_equal(pa, opa)
        got = Attr()
        assert cu.cuStreamGetAttribute(h, ACCESS_POLICY_WINDOW, C.byref(got)) == 0
        assert (got.window.base, got.window.bytes) == (mine.data_ptr(), 1 << 20)
