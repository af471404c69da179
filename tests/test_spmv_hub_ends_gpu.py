"""The ends of the binades in which the CTA-per-row SpMV adds integers: sums
that leave the subnormals slowly, and that stay zero for whole tiles before the
smallest normal terms come. y equals the oracle's in-order chain bit for bit
(tolerance zero)."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu

N = 5000  # one row: longer than any bound below which a row is summed by a lane


def _spmv(rows):
    """rows: (values, x) pairs, one matrix row each with its own columns."""
    lens = [len(v) for v, _ in rows]
    n = sum(lens)
    rp = np.zeros(n + 1, np.int64)
    rp[1:len(lens) + 1] = np.cumsum(lens)
    rp[len(lens) + 1:] = rp[len(lens)]
    val, x = np.concatenate([v for v, _ in rows]), np.concatenate([w for _, w in rows])
    col = np.arange(n, dtype=np.int32)
    want = oracle.spmv(rp, col, val, x)
    with ab.SellMatrix(rp, col, val) as m:
        # other rows' tiles have been in the shared memory before
        for _ in range(2):
            got = m.spmv(x)
            assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), \
                np.flatnonzero(got.view(np.uint64) != want.view(np.uint64))
    return want


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("first", [0, 1, 7, 255, 256, 513, 1024, 1500])
def test_sums_that_leave_the_subnormals_slowly(first, sign):
    """Zeros up to entry `first`, then equal terms of which 64 to 2,000 make the
    smallest normal number: the sum is subnormal, or zero, when a tile's scans
    are made, and normal when they are used."""
    rows = []
    for k in (64, 100, 256, 511, 512, 513, 777, 2000):
        v = np.full(N, sign)
        v[:first] = 0.0
        rows.append((v, np.full(N, 2.0**-1022 / k)))
    assert np.all(_spmv(rows)[:len(rows)] * sign > 0)


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("exp", [-1023, -1022, -1021, -1020])
def test_zeros_for_tiles_then_the_smallest_normals(exp, sign):
    rng = np.random.default_rng(3)
    rows = []
    for first in (511, 512, 513, 600, 767, 768, 1024):
        v = sign * rng.uniform(1, 2, N)
        v[:first] = 0.0
        x = np.full(N, 2.0**exp)
        x[first + 3:first + 500] = 2.0**-1060  # stays in the lowest binades for a while
        rows.append((v, x))
    _spmv(rows)
