"""The ends of the binades in which the CTA-per-row SpMV adds integers: sums
that leave the subnormals slowly, that stay zero for whole tiles before the
smallest normal terms come, and that round to infinity and meet terms of the
other sign. y equals the oracle's in-order chain bit for bit (tolerance zero)."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu

N = 5000  # one row: longer than any bound below which a row is summed by a lane
MAX = np.finfo(np.float64).max


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


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("at", [20, 250, 256, 300, 700, 2000])
def test_a_sum_that_rounds_to_infinity_stays_there(at, sign):
    """The largest finite number, zeros, one last place up (infinity), and terms
    of the other sign, which an infinite sum no longer feels."""
    rows = []
    for up, down, gap in ((2.0**971, 2.0**975, 1), (2.0**971, 2.0**975, 40), (2.0**971, 2.0**1000, 1),
                          (1.5 * 2.0**970, 2.0**971, 1), (2.0**970, 2.0**971, 1), (2.0**969, 2.0**971, 1)):
        v = np.zeros(N)
        v[0] = MAX
        v[at] = up
        v[at + gap] = -down
        v[at + gap + 200] = -2.0**1000
        rows.append((sign * v, np.ones(N)))
    want = _spmv(rows)
    assert np.all(np.isinf(want[:5])) and np.isfinite(want[5])
