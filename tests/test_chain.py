"""The integer steps of the in-order fused multiply-add chain (chain.cuh),
compiled for the host, against exact rational arithmetic."""
from __future__ import annotations

import ctypes as C
import struct
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "albba_gb300" / "csrc"
DRIVER = """
#include <cstdint>
#define __host__
#define __device__
#include "chain.cuh"
extern "C" int64_t step(uint64_t v, uint64_t x, int E, int *stop) {
    const alb::ChainTerm t = alb::chain_term(v, x);
    bool s;
    const int64_t k = alb::chain_round(t.h, (int16_t)t.e, E, s);
    *stop = s;
    return k;
}
extern "C" int runs(int E) { return alb::chain_runs(E); }
"""


@pytest.fixture(scope="module")
def chain(tmp_path_factory):
    d = tmp_path_factory.mktemp("chain")
    (d / "c.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "c.cpp"),
                    "-o", str(d / "c.so")], check=True)
    lib = C.CDLL(str(d / "c.so"))
    lib.step.restype = C.c_int64
    lib.step.argtypes = [C.c_uint64, C.c_uint64, C.c_int, C.POINTER(C.c_int)]
    return lib


def _bits(v):
    return struct.unpack("<Q", struct.pack("<d", v))[0]


def _round(q):
    """The fp64 number nearest q (ties to even)."""
    try:
        return float(q)
    except OverflowError:
        return np.inf if q > 0 else -np.inf


def _steps(chain, acc, terms):
    """The terms that a run from acc takes, each against the exact sum."""
    took, stop = 0, C.c_int()
    E = (_bits(acc) >> 52) & 0x7FF
    assert chain.runs(E)
    u = Fraction(2) ** (E - 1075)
    A, sg = abs(Fraction(acc)) / u, 1 if acc > 0 else -1
    for v, x in terms:
        k = chain.step(_bits(v), _bits(x), E, C.byref(stop))
        nxt = A + sg * k
        if stop.value or not 2**52 < nxt <= 2**53:
            break
        want = _round(sg * A * u + Fraction(v) * Fraction(x))
        assert want == float(sg * nxt * u), (acc, v, x)
        A, took = nxt, took + 1
    return took


# the lowest normal binade, ordinary ones, and the last whose upper end is finite
@pytest.mark.parametrize("E", [1, 2, 53, 1023, 2044, 2045])
def test_a_run_rounds_as_the_chain_does(chain, E):
    rng = np.random.default_rng(E)
    took = 0
    for _ in range(300):
        acc = float(np.ldexp(rng.integers(1 << 52, 1 << 53) * rng.choice([-1.0, 1.0]), E - 1075))
        for acc in (acc, float(np.copysign(np.ldexp(1.0, E - 1023), acc)),
                    float(np.copysign(np.ldexp(2.0**53 - 1, E - 1075), acc))):
            mag = np.exp2(rng.uniform(-60, 51, 8))
            t = rng.choice([-1.0, 1.0], 8) * mag
            t[rng.random(8) < 0.2] = 0.0
            half = rng.integers(0, 2) * 0.5 + rng.integers(0, 4, 8) * 0.25
            t[rng.random(8) < 0.3] = half[0]
            # (v in units of the sum's last place, x the rest)
            e1 = (E - 1075) // 2
            took += _steps(chain, acc, [(float(np.ldexp(q, e1)), float(np.ldexp(1.0, E - 1075 - e1)))
                                        for q in t])
    assert took > 500


def test_no_run_from_zero_subnormal_last_binade_infinity_or_nan(chain):
    assert [chain.runs(E) for E in (0, 1, 2045, 2046, 2047)] == [0, 1, 1, 0, 0]


def test_ties_and_special_operands_end_a_run(chain):
    stop = C.c_int()
    one = _bits(1.0)
    for v, want in ((0.5, 1), (1.5, 1), (-0.5, 1), (0.25, 0), (0.75, 0), (0.0, 0), (np.inf, 1), (-np.inf, 1),
                    (np.nan, 1), (2.0**53, 1)):
        chain.step(_bits(np.ldexp(v, -52)), one, 1023, C.byref(stop))
        assert stop.value == want, v
