// The in-order fp64 fused multiply-add chain acc = fma(v[i], x[i], acc),
// evaluated many entries at a time with the same bits.
//
// While |acc| stays inside one binade [2^e, 2^(e+1)), every result is a
// multiple of the same u = 2^(e-52), so one step is acc + round(p / u) * u
// with p the exact product v * x: acc itself is already a multiple of u, and
// what rounding adds does not depend on it -- unless p lies exactly halfway
// between two multiples, where ties-to-even looks at acc. The chain is then
// a sum of integers k[i] = round(p[i] / u), whose prefix sums are found in
// parallel, exact in 64 bits. A prefix that leaves the binade, a tie, or a
// product too large for the bound below ends the run: entries before it are
// committed and that entry is done by fma itself.
//
// Products are formed with integer multiplies: a warp's fp64 operation holds
// its quarter of the SM for about 64 cycles on GB300, a dependent one for
// about 115. 62 bits of the product and a sticky bit are kept, enough to round
// to the at most 53 bits of k and to tell a tie.
//
// The binade's ends: with A = |acc| / u a step's result is taken for
// 2^52 < A <= 2^53. Above 2^52 the exact sum lies at or above 2^52 - with A
// exactly 2^52 it may lie below, where the grid is finer - and a sum within
// u / 2 of 2^53 rounds to 2^53 on either side's grid; from there a step down
// is on this grid again, and one up leaves the interval. In the last binade
// 2^53 u is infinity, from which no step leads back: sums in it, like zero and
// subnormal ones, are not run this way (chain_runs).
#pragma once

#include <cstdint>

namespace alb {

constexpr int64_t kChainOne = 1ll << 52;

// Whether a sum of biased exponent E may be run on integers.
__host__ __device__ inline bool chain_runs(int E) { return E > 0 && E < 0x7FE; }

// High half of a 64 x 64-bit product.
__host__ __device__ inline uint64_t chain_mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// p = v * x as h * 2^(e - 2106), |h| < 2^62, the last bit of |h| sticky; from
// the operands' bits. An infinite or NaN operand gives an e that chain_round
// refuses.
struct ChainTerm {
    int64_t h;
    int32_t e;
};
__host__ __device__ inline ChainTerm chain_term(uint64_t v, uint64_t x) {
    const int ev = (int)(v >> 52) & 0x7FF, ex = (int)(x >> 52) & 0x7FF;
    const uint64_t mask = (uint64_t)kChainOne - 1;
    const uint64_t mv = ((v & mask) | (ev ? (uint64_t)kChainOne : 0)) << 11;
    const uint64_t mx = ((x & mask) | (ex ? (uint64_t)kChainOne : 0)) << 11;
    const uint64_t hi = chain_mulhi(mv, mx), lo = mv * mx;
    const uint64_t m = (hi >> 2) | ((hi & 3) != 0 || lo != 0 ? 1u : 0u);
    const int64_t sg = (int64_t)(v ^ x) >> 63;
    ChainTerm t;
    t.h = ((int64_t)m ^ sg) - sg;
    t.e = ev == 0x7FF || ex == 0x7FF ? 1 << 14 : (ev ? ev : 1) + (ex ? ex : 1);
    return t;
}

// k = round(p / u) for acc of biased exponent E (1 .. 2046). stop: p / u may
// reach 2^53 (256 of them still add up in 64 bits), or p is halfway between two
// multiples of u. No branch: the shift held at 63 sends every |p| below u / 2
// to 0.
__host__ __device__ inline int64_t chain_round(int64_t h, int32_t e, int E, bool &stop) {
    int d = E + 1031 - e;
    stop = d < 9;
    d = d < 9 ? 9 : d > 63 ? 63 : d;
    const int64_t sg = h >> 63;
    const uint64_t s = (uint64_t)((h ^ sg) - sg) + (1ull << (d - 1));
    stop |= (s << (64 - d)) == 0;
    return ((int64_t)(s >> d) ^ sg) - sg;
}

}  // namespace alb
