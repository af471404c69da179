"""Matrices whose long rows are all about as long, more of them than get a CTA
each: y bit for bit the in-order chain's, and no longer to wait for than when
they were few (a CTA per row once took ten times as long as a lane per row)."""
from __future__ import annotations

import statistics

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _matrix(rows, length, rng, low=-1):
    lens = np.full(rows, length) + rng.integers(0, 9, rows)
    n = max(rows, 2 * length)
    rp = np.zeros(n + 1, np.int64)
    rp[1:rows + 1] = np.cumsum(lens)
    rp[rows + 1:] = rp[rows]
    return rp, rng.integers(0, n, rp[-1]).astype(np.int32), rng.uniform(low, 1, rp[-1])


# two CTAs an SM, just over, many more; up to 1,000 entries a row's signs count
@pytest.mark.parametrize("low", [-1, 0])
@pytest.mark.parametrize("rows,length", [(300, 300), (304, 700), (305, 700), (305, 5000), (40, 992),
                                         (40, 993), (1000, 260), (3000, 900), (40, 9000)])
def test_bit_exact(rows, length, low):
    rng = np.random.default_rng(rows)
    rp, col, val = _matrix(rows, length, rng, low)
    x = rng.standard_normal(len(rp) - 1)
    with ab.SellMatrix(rp, col, val) as m:
        assert np.array_equal(m.spmv(x).view(np.uint64), oracle.spmv(rp, col, val, x).view(np.uint64))


def test_many_similar_rows_take_no_longer_than_their_chains():
    import torch
    rng = np.random.default_rng(2)
    us = {}
    for rows in (200, 20_000):
        rp, col, val = _matrix(rows, 1000, rng)
        x = torch.randn(len(rp) - 1, dtype=torch.float64, device="cuda")
        y = torch.empty_like(x)
        with ab.SellMatrix(rp, col, val) as m:
            m.spmv_device(x, y)
            us[rows] = statistics.median(m.spmv_device(x, y) for _ in range(9))
    # a chain of 1,000 entries takes about 60 us, 20,000 of them side by side
    # 100 on one GPU, in CTAs of their own 3,000
    assert us[20_000] < 10 * us[200], us
