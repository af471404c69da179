"""Rows long enough for the CTA-per-row SpMV, whose chain of fused
multiply-adds is evaluated as integer prefix sums: y equals the oracle's
in-order chain bit for bit (tolerance zero; a NaN only has to be a NaN, its
payload is the processor's)."""
from __future__ import annotations

import numpy as np
import pytest

import albba_gb300 as ab
import oracle

pytestmark = pytest.mark.gpu


def _values(kind, m, rng):
    """Entry values of a row and the x they meet (x has one column each)."""
    sign = rng.choice([-1.0, 1.0], m)
    if kind == "signed":
        return rng.uniform(-1, 1, m), rng.standard_normal(m)
    if kind == "positive":
        return rng.uniform(0, 1, m), rng.uniform(0, 1, m)
    if kind == "ties":  # few-bit products over 110 binades: halves are common
        return sign * (1 + rng.integers(0, 8, m) / 8) * np.exp2(rng.integers(-55, 55, m)), np.ones(m)
    if kind == "power":  # the sum sits on powers of two, terms at half its last place
        v = np.where(rng.random(m) < 0.5, 0.5, -0.25)
        v[0] = 2.0**52
        return v, np.ones(m)
    if kind == "integers":  # passes through zero, every step exact
        return np.ones(m), rng.integers(-4, 5, m).astype(float)
    if kind == "zeros":
        return np.where(rng.random(m) < 0.9, 0.0, sign), np.where(rng.random(m) < 0.5, -0.0, 1.0)
    if kind == "tiny":  # subnormal products and sums
        return sign * np.exp2(-rng.uniform(480, 1020, m)), np.exp2(-rng.uniform(0, 540, m))
    if kind == "huge":  # overflows to infinity on the way
        return rng.uniform(0, 1, m) * np.exp2(rng.uniform(900, 1023, m)), np.ones(m)
    v, x = rng.uniform(-1, 1, m), rng.standard_normal(m)  # "special"
    v[m // 2] = np.inf
    x[m // 2 + 40] = np.nan
    return v, x


# longest row N: rows above max(256, 12 sqrt(N)) have a CTA each, others above
# 256 a lane each; lengths on both sides of those lines, of a tile of 256 and
# of a lane's 8 entries
LENS = {"long": [1024, 1697, 1698, 3537, 3583, 3584, 3585, 3591, 3592, 5000, 20011, 0, 3, 256, 257],
        "short": [431, 432, 511, 512, 513, 1279, 1280, 1281, 1288, 0, 7, 255, 256, 257, 263, 264]}


@pytest.mark.parametrize("lens", LENS.values(), ids=LENS)
@pytest.mark.parametrize("kind", ["signed", "positive", "ties", "power", "integers", "zeros",
                                  "tiny", "huge", "special"])
def test_gpu_spmv_hub_rows_bit_exact(kind, lens):
    rng = np.random.default_rng(17)
    n = sum(lens)
    rp = np.zeros(n + 1, np.int64)
    rp[1:len(lens) + 1] = np.cumsum(lens)
    rp[len(lens) + 1:] = rp[len(lens)]
    val, x = np.empty(n), np.empty(n)
    for r, m in enumerate(lens):
        if m:
            v, w = _values(kind, max(m, 128), rng)
            val[rp[r]:rp[r + 1]], x[rp[r]:rp[r + 1]] = v[:m], w[:m]
    col = np.arange(n, dtype=np.int32)
    want = oracle.spmv(rp, col, val, x)
    with ab.SellMatrix(rp, col, val) as m:
        got = m.spmv(x)
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))
