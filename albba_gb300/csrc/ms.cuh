// Batched BFS: its state, and the steps of a level as device functions. The
// host loop launches them one by one (msbfs.cu: LOOP_HOST and the profile);
// the cooperative kernel runs a whole search (ms_grid.cu).
//
// Arrays that a level writes are read with ordinary loads, never through the
// non-coherent path: inside the cooperative kernel the next level reads them.
#pragma once

#include <cstring>

#include "dev.cuh"
#include "selector.cuh"

namespace alb {

constexpr uint64_t kAll = ~0ull;
// Packed list counters (rows << kMsBigShift | chunks), as in bfs.cu.
constexpr int kMsBigShift = 38;
constexpr unsigned long long kMsBigMask = (1ull << kMsBigShift) - 1;

struct MsCtl {
    int32_t level, dir, prev_dir, q_valid, done, err, policy, base;  // base: level of S[0]
    float alpha, beta;
    int32_t levels_td, levels_bu;
    int64_t n, nwords;
    int64_t nf, mf, prev_nf, nu, mu, active_words;
    int64_t pairs, edges;  // (vertex, root) pairs reached; sum of their push degrees
    // the host loop's counters, by level modulo 3 (the cooperative kernel's: MsSlots)
    unsigned long long acc_n[3], acc_mo[3], acc_mi[3], acc_full[3], acc_bits[3], acc_edges[3],
        qn[3], acc_bytes[3], acc_done[3], nbig[3], work[3];
    float feat_mean_deg, feat_skew;
    // set for the next level at the end of one: frontier-nonzero filter on or
    // off, and whether the snapshot store must be flushed before the level runs
    int32_t filt, need_flush, level_cap, pad;
    int64_t m_in;
    // Roots whose frontier is small (or empty) at a bottom-up level: the pull
    // does not wait for their bits (a row stops once every other root is
    // accounted for) and a push over their frontier finds their new rows.
    // Chosen by ms_decide from per-root frontier counts sampled on every
    // kSampleStride-th bitmap word (MsSample, filled by ms_sample).
    unsigned long long tmask;
    int32_t grab;  // words per run of the bottom-up pull (1 .. 32)
    // budget of estimated push edges for all tmask roots together (0: off)
    int64_t push_budget;
    unsigned long long used;  // root bits in use
    int32_t pushed_roots;     // sum of popc(tmask) over the levels
    int32_t gtrace_on;        // cooperative kernel: record each level in MsArgs::gtrace
};
static_assert(sizeof(MsCtl) % 8 == 0, "the control block is copied in 8-byte words");

// Level records of the cooperative kernel, written by its first block: start
// and end %globaltimer stamps, the level's algorithmic bytes, its direction,
// and the frontier and unvisited counts it started from.
constexpr int kGTraceCap = 1 << 14;
constexpr int kGTraceW = 8;

// Push degrees of each root's sampled frontier. Kept beside the control block
// (same allocation) so that copies of that stay small.
struct MsSample {
    unsigned long long deg[64];
};

// Per-root frontier sampling: one bitmap word (32 rows) in kSampleStride.
constexpr int kSampleStride = 32;
constexpr int kSampleMinDiv = 1024;
// Default push budget (all tmask roots together): m_in / kPushDiv estimated
// push edges.
constexpr int kPushDiv = 64;

struct MsArgs {
    int64_t n, nwords, npad;
    int32_t C, log2C, K;
    int32_t sigma;  // sort window: perm maps each aligned window of sigma rows to itself
    unsigned wpw, nwin;  // words of a sort window (1: not whole words), windows
    const int32_t *perm, *inv, *ideg, *odeg, *width;
    const uint32_t *vinit;  // rows without sources, and padding: one bit a position
    const int64_t *slice_off;
    const int4 *col4;
    const int64_t *prow;
    const int32_t *pcol;
    int64_t nlong;  // rows kept out of the slices, pulled in chunks
    const int32_t *lrow;
    const int64_t *lptr;
    const int32_t *lcol;
    uint64_t *V;
    uint64_t *S;  // K slots of npad words
    uint32_t *D;
    uint32_t *A;  // 2 x nwords: frontier-nonzero bitmaps by level parity
    int32_t *q0, *q1;
    int32_t *big;  // frontier rows longer than kBigRow (top-down)
    int64_t *big_base;
    int32_t *pbig;  // the same of the pushed roots' rows: the long rows' list is in use
    int64_t *pbig_base;
    MsCtl *ctl;
    MsSample *smp;  // directly after *ctl
    int32_t any_big;   // some push row is longer than kBigRow
    int32_t long_row;  // rows with more sources than this are the long rows
    const float *mlp;
    long long *gtrace;  // kGTraceCap x kGTraceW level records (MsCtl::gtrace_on)
};

__device__ __forceinline__ uint32_t *nz_bits(const MsArgs &a, int L) { return a.A + (int64_t)(L & 1) * a.nwords; }
__device__ __forceinline__ uint64_t *slot(const MsArgs &a, int j) { return a.S + (int64_t)j * a.npad; }

struct MsInit {
    int32_t roots[64];
    int32_t nroots, policy, level_cap;
    float alpha, beta, mean_deg, skew;
    int64_t n_live, m_in, active0, push_budget;
    int32_t grab;
    int32_t gtrace;  // record the levels (MsArgs::gtrace)
    uint64_t unused;  // root bits not in use
};

// What a step found, per thread.
struct MsCounts {
    unsigned n = 0, bits = 0, full = 0, done = 0;
    unsigned long long mo = 0, mi = 0, edges = 0, bytes = 0;
};

// One level as a step sees it, and the calling warp's place in the launch:
// the first warps of all blocks come first, so that work for fewer warps than
// there are is spread over all SMs (64 K vertices have 2,048 words for 4,864
// warps), and each next one turned by five blocks, so that every 4th, 16th or
// 32nd piece of work -- a sort window's widest rows -- is not always the same
// blocks' (152 SMs; the first pull of 2^22 took 633 us instead of 532).
struct MsStep {
    int L;
    const uint64_t *F;   // this level's frontier and the next one's
    uint64_t *N;
    const uint32_t *Az;  // their nonzero bitmaps
    uint32_t *An;
    uint64_t tm;         // roots that are pushed at a bottom-up level
    int64_t gw, nwarps;
    bool numbered;  // the pull's first runs by warp number, not from the counter
};

__device__ __forceinline__ MsStep ms_step(const MsArgs &a, int L, int j, uint64_t tm,
                                          bool numbered) {
    const unsigned wib = threadIdx.x >> 5;
    return MsStep{L, slot(a, j), slot(a, j + 1), nz_bits(a, L), nz_bits(a, L + 1), tm,
                  (int64_t)wib * gridDim.x + (blockIdx.x + 5 * wib) % gridDim.x,
                  (int64_t)gridDim.x * (blockDim.x >> 5), numbered};
}

// The control block before level 0, from what the roots came to.
__device__ __forceinline__ void ms_start(const MsArgs &a, const MsInit &in, int64_t nf, int64_t mf,
                                         int64_t pairs, int64_t edges, int64_t done, int64_t done_mi,
                                         int64_t full, MsCtl &c) {
    memset(&c, 0, sizeof(c));
    c.dir = -1;
    c.prev_dir = -1;
    c.policy = in.policy;
    c.alpha = in.alpha;
    c.beta = in.beta;
    c.n = a.n;
    c.nwords = a.nwords;
    c.nf = nf;
    c.mf = mf;
    c.nu = in.n_live - done;
    c.mu = in.m_in - done_mi;
    c.active_words = in.active0 - full;
    c.pairs = pairs;
    c.edges = edges;
    c.feat_mean_deg = in.mean_deg;
    c.feat_skew = in.skew;
    c.m_in = in.m_in;
    c.level_cap = in.level_cap;
    c.push_budget = in.push_budget;
    c.grab = in.grab;
    c.used = in.nroots >= 64 ? kAll : (1ull << in.nroots) - 1;
    c.gtrace_on = in.gtrace;
    c.done = c.nf == 0;
    // level 0's direction: the rule of later levels (the learned policy
    // falls back to Beamer here: no level has run yet)
    BfsCtl fc;
    memset(&fc, 0, sizeof(fc));
    fc.n = c.n;
    fc.nwords = c.nwords;
    fc.nf = c.nf;
    fc.mf = c.mf;
    fc.nu = c.nu;
    fc.mu = c.mu;
    fc.prev_dir = -1;
    fc.policy = in.policy == ALB_POLICY_LEARNED ? ALB_POLICY_BEAMER : in.policy;
    fc.alpha = in.alpha;
    fc.beta = in.beta;
    c.dir = rule_dir(fc);
    c.filt = c.mf < c.m_in / 8;
}

// Words of a bottom-up level in runs of `run` words (1 to 32, set by the
// host from the word count: about three runs per warp) from the level's
// counter (dynamic distribution, as WordRuns); where x.numbered is set a warp's
// first run goes by its number, which saves a round trip. The done words of a
// run are loaded together, one per lane, a run ahead of use. kSkip: words whose
// rows are all done are not yielded; their next-frontier words and nonzero bits
// are cleared when the run comes up, one coalesced store per word, so a warp
// does not walk them one dependent round trip at a time (at late levels most
// words are such). Words of slices wider than `split` are left to ms_pull_wide.
// Call from all lanes of a warp.
template <bool kSkip>
struct MsWords {
    int32_t cur, nxt;     // first word of the current run and of the next one
    uint32_t dcur, dnxt;  // lane l < step: done word of word cur + l / nxt + l
    unsigned left;        // words of the current run not yet yielded
    unsigned ncur, nnxt;  // words of the runs that are not left out
    int step, split;
    // (words past the last are taken for a.nwords)
    __device__ __forceinline__ int32_t grab(const MsArgs &a, const MsStep &x,
                                            unsigned long long *ctr) const {
        unsigned long long v = 0;
        if ((threadIdx.x & 31) == 0) v = atomicAdd(ctr, (unsigned long long)step);
        return (int32_t)min(a.nwords, (x.numbered ? x.nwarps * step : 0) +
                                          (int64_t)__shfl_sync(kFull, v, 0));
    }
    __device__ __forceinline__ void load(const MsArgs &a, int32_t r, uint32_t &d, unsigned &n) const {
        const int l = threadIdx.x & 31;
        bool mine = l < step && r + l < a.nwords;
        d = mine ? a.D[r + l] : kFull;
        if (mine && split != INT32_MAX) mine = __ldg(a.width + (((int64_t)(r + l) * 32) >> a.log2C)) <= split;
        n = __ballot_sync(kFull, mine);
    }
    __device__ __forceinline__ unsigned prep(uint64_t *N, uint32_t *An) const {
        if (!kSkip) return ncur;
        const int l = threadIdx.x & 31;
        const unsigned full = __ballot_sync(kFull, dcur == kFull) & ncur;
        for (unsigned f = full; f; f &= f - 1) {
            const int q = __ffs(f) - 1;
            N[(int64_t)(cur + q) * 32 + l] = 0;
            if (l == 0) An[cur + q] = 0;
        }
        return ncur & ~full;
    }
    __device__ __forceinline__ void start(const MsArgs &a, const MsStep &x, int run, int wide,
                                          unsigned long long *ctr) {
        step = run;
        split = wide;
        cur = x.numbered ? (int32_t)min(a.nwords, x.gw * step) : grab(a, x, ctr);
        nxt = grab(a, x, ctr);
        load(a, cur, dcur, ncur);
        load(a, nxt, dnxt, nnxt);
        left = prep(x.N, x.An);
    }
    // the next word (a.nwords when the level's words are exhausted) and its
    // done word
    __device__ __forceinline__ int32_t next(const MsArgs &a, const MsStep &x,
                                            unsigned long long *ctr, uint32_t &d) {
        while (!left) {
            if (cur >= a.nwords) {
                d = kFull;
                return (int32_t)a.nwords;
            }
            cur = nxt;
            dcur = dnxt;
            ncur = nnxt;
            if (cur < a.nwords) {
                nxt = grab(a, x, ctr);
                load(a, nxt, dnxt, nnxt);
            }
            left = prep(x.N, x.An);
        }
        const int q = __ffs(left) - 1;
        left &= left - 1;
        d = __shfl_sync(kFull, dcur, q);
        return cur + q;
    }
};

template <class T>
__device__ __forceinline__ T ms_ld(const T *p) { return *p; }

// What a word's 32 rows found (acc) into the state: next frontier, nonzero
// bits, visited and done words, counts. vis, d: its visited and done words.
// Returns the lane's bytes.
__device__ __forceinline__ unsigned ms_pull_fold(const MsArgs &a, const MsStep &x, int64_t w,
                                                 uint64_t vis, uint64_t acc, uint32_t d,
                                                 MsCounts &cnt) {
    const int lane = threadIdx.x & 31;
    const int64_t p = w * 32 + lane;
    const uint64_t nb = acc & ~vis;
    x.N[p] = nb;
    const unsigned nzm = __ballot_sync(kFull, nb != 0);
    if (lane == 0) x.An[w] = nzm;
    bool done_now = false;
    if (nb) {
        const uint64_t nv = vis | nb;
        a.V[p] = nv;
        const int pc = __popcll(nb);
        const int32_t od = __ldg(a.odeg + p);
        cnt.n++;
        cnt.bits += pc;
        cnt.mo += od;
        cnt.edges += (unsigned long long)pc * od;
        if (nv == kAll) {
            done_now = true;
            cnt.done++;
            cnt.mi += __ldg(a.ideg + p);
        }
    }
    const unsigned dm = __ballot_sync(kFull, done_now);
    if (lane == 0 && dm) {
        a.D[w] = d | dm;
        cnt.full += (d != kFull && (d | dm) == kFull);
    }
    return nb ? 12 : 0;  // V[p] written, push degree
}

// Bottom-up over S[j] -> S[j+1]. kBypass: skip words whose 32 positions are
// done; kEarly: stop a row once every root is accounted for, or at padding.
// kFilt: test the nonzero bitmap before each 8-byte frontier fetch. It pays
// when few sources are in the frontier (the fetches it saves miss L2) and
// costs a dependent round trip per group when most are, so the host picks it
// from the frontier's share of all entries.
// kWide (with !kFilt): two column groups per step, eight frontier fetches in
// flight per lane, at 32 warps per SM.
template <bool kBypass, bool kEarly, bool kFilt, bool kWide = false>
__device__ __forceinline__ void ms_pull(const MsArgs &a, const MsStep &x, int run, int split,
                                        unsigned long long *ctr, MsCounts &cnt) {
    const uint64_t *F = x.F;
    uint64_t *N = x.N;
    const int lane = threadIdx.x & 31;
    const uint64_t tm = x.tm;
    const uint32_t *Az = x.Az;
    uint32_t *An = x.An;
    unsigned bytes = 0;
    const uint64_t pol = l2_evict_first();
    // words come in runs from the level's counter (MsWords, done words
    // skipped when kBypass). Software pipeline over words: the visited words
    // and slice geometry are requested one word ahead, so their latency
    // overlaps the current word's column loads and gathers.
    MsWords<kBypass> it;
    it.start(a, x, run, split, ctr);
    auto geometry = [&](int32_t ww, uint32_t dd, uint64_t &vv, int32_t &wdv, int64_t &sov) {
        vv = kAll;
        wdv = 0;
        sov = 0;
        if (ww < a.nwords && !(kBypass && dd == kFull)) {
            const int64_t pw = (int64_t)ww * 32 + lane;
            // rows past n (padding of the last word) are preset visited;
            // their slice index is clamped so the loads stay in bounds
            const int64_t sw = (pw < a.n ? pw : a.n - 1) >> a.log2C;
            vv = a.V[pw];
            wdv = __ldg(a.width + sw);
            sov = __ldg(a.slice_off + sw);
        }
    };
    uint32_t d, d1 = kFull;
    const int32_t nwords = (int32_t)a.nwords;
    int32_t w = it.next(a, x, ctr, d);
    int32_t w1 = w < nwords ? it.next(a, x, ctr, d1) : nwords;
    uint64_t vis_c;
    int32_t wd_c;
    int64_t so_c;
    geometry(w, d, vis_c, wd_c, so_c);
    while (w < nwords) {
        uint64_t vis1;
        int32_t wd1;
        int64_t so1;
        geometry(w1, d1, vis1, wd1, so1);
        const int64_t p = (int64_t)w * 32 + lane;
        if (kBypass && d == kFull) {  // not reached: MsWords clears these words
            N[p] = 0;
            if (lane == 0) An[w] = 0;
        } else {
            bytes += 8;  // V[p]
            const uint64_t vis = vis_c;
            // roots in tmask are found by the push over their frontier
            const uint64_t visx = vis | tm;
            bool active = visx != kAll;
            int32_t ng = active ? (wd_c + 3) >> 2 : 0;
            const int4 *cp = a.col4 + (so_c >> 2) + (p & (a.C - 1));
            uint64_t acc = 0;
            // group g+1 is requested before group g's frontier fetches, so each
            // lane keeps a column load in flight while it waits on the gathers
            const int32_t pp = (int32_t)p;
            if (kWide && !kFilt) {
                const int4 pad = make_int4(pp, pp, pp, pp);
                int4 c0 = pad, c1 = pad;
                if (active && ng > 0) c0 = ld_stream(cp, pol);
                if (active && ng > 1) c1 = ld_stream(cp + a.C, pol);
                for (int32_t g = 0;; g += 2) {
                    active = active && g < ng;
                    if (!__any_sync(kFull, active)) break;
                    if (!active) continue;
                    int4 n0 = pad, n1 = pad;
                    if (g + 2 < ng) n0 = ld_stream(cp + (int64_t)(g + 2) * a.C, pol);
                    if (g + 3 < ng) n1 = ld_stream(cp + (int64_t)(g + 3) * a.C, pol);
                    ALB_CHECK_ID4(c0, a.npad, pp, &a.ctl->err);
                    ALB_CHECK_ID4(c1, a.npad, pp, &a.ctl->err);
                    // past the row's last group c1 is padding (p itself)
                    acc |= ms_ld(F + c0.x) | ms_ld(F + c0.y) | ms_ld(F + c0.z) | ms_ld(F + c0.w) |
                           ms_ld(F + c1.x) | ms_ld(F + c1.y) | ms_ld(F + c1.z) | ms_ld(F + c1.w);
                    bytes += g + 1 < ng ? 96 : 48;
                    if (kEarly && (c1.w == pp || (acc | visx) == kAll)) active = false;
                    c0 = n0;
                    c1 = n1;
                }
                ng = 0;  // the single-group loop below has nothing left
            }
            int4 c = make_int4(pp, pp, pp, pp);
            if (active && ng > 0) c = ld_stream(cp, pol);
            for (int32_t g = 0;; g++) {
                active = active && g < ng;
                if (!__any_sync(kFull, active)) break;
                if (!active) continue;
                int4 nx = make_int4(pp, pp, pp, pp);
                if (g + 1 < ng) nx = ld_stream(cp + (int64_t)(g + 1) * a.C, pol);
                // padding entries hold p itself: S[j][p] only has bits already in
                // V[p], so OR-ing it changes nothing
                ALB_CHECK_ID4(c, a.npad, pp, &a.ctl->err);
                if (kFilt) {
                    const uint32_t z0 = ms_ld(Az + (c.x >> 5)), z1 = ms_ld(Az + (c.y >> 5)),
                                   z2 = ms_ld(Az + (c.z >> 5)), z3 = ms_ld(Az + (c.w >> 5));
                    const bool h0 = (z0 >> (c.x & 31)) & 1u, h1 = (z1 >> (c.y & 31)) & 1u,
                               h2 = (z2 >> (c.z & 31)) & 1u, h3 = (z3 >> (c.w & 31)) & 1u;
                    if (h0) acc |= ms_ld(F + c.x);
                    if (h1) acc |= ms_ld(F + c.y);
                    if (h2) acc |= ms_ld(F + c.z);
                    if (h3) acc |= ms_ld(F + c.w);
                    // four columns, four bitmap words, the frontier words fetched
                    bytes += 32 + 8 * (h0 + h1 + h2 + h3);
                } else {
                    acc |= ms_ld(F + c.x) | ms_ld(F + c.y) | ms_ld(F + c.z) | ms_ld(F + c.w);
                    bytes += 48;  // four columns and their four frontier words
                }
                if (kEarly && (c.w == pp || (acc | visx) == kAll)) active = false;
                c = nx;
            }
            bytes += ms_pull_fold(a, x, w, vis, acc, d, cnt);
        }
        w = w1;
        d = d1;
        vis_c = vis1;
        wd_c = wd1;
        so_c = so1;
        w1 = w1 < nwords ? it.next(a, x, ctr, d1) : nwords;
    }
    cnt.bytes += bytes;
}

// The words of slices wider than `split`, by teams of kTeam warps that share
// a word's column groups. One warp takes a slice of 1024 columns 128 dependent
// steps (90 us on R-MAT scale 20, whose whole level moves in less), so where a
// level is not many times longer than that, its widest words are spread. A
// team's words lie `teams` apart in the order of rank in the sort window (the
// first word of every window, then the second, ...): the wide ones are among
// the first ranks. room: 32 words a team.
constexpr int kTeam = 8;

__device__ __forceinline__ void team_sync(int team) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kTeam * 32) : "memory");
}

__device__ __forceinline__ void ms_pull_wide(const MsArgs &a, const MsStep &x, int split,
                                             uint64_t *room, MsCounts &cnt) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int team = wib / kTeam, k = wib % kTeam;
    const int64_t teams = x.nwarps / kTeam, t = (int64_t)team * gridDim.x + blockIdx.x;
    const int64_t all = (int64_t)a.nwin * a.wpw;
    unsigned *acc_lo = reinterpret_cast<unsigned *>(room + team * 32) + 2 * lane, *acc_hi = acc_lo + 1;
    for (int64_t i0 = t; i0 < all; i0 += 32 * teams) {
        // lane l: the team's word l from here on
        const int64_t i = i0 + lane * teams;
        int32_t mw = (int32_t)a.nwords, wd_l = 0;
        if (i < all) {
            const unsigned rank = (unsigned)i / a.nwin;
            mw = (int32_t)min((int64_t)((unsigned)i - rank * a.nwin) * a.wpw + rank, a.nwords);
            if (mw < a.nwords) wd_l = __ldg(a.width + (((int64_t)mw * 32) >> a.log2C));
        }
        for (unsigned m = __ballot_sync(kFull, wd_l > split); m; m &= m - 1) {
            const int q = __ffs(m) - 1;
            const int64_t w = __shfl_sync(kFull, mw, q);
            const int32_t ng = (__shfl_sync(kFull, wd_l, q) + 3) >> 2;
            const int64_t p = w * 32 + lane;
            const int32_t pp = (int32_t)p;
            const uint64_t vis = ms_ld(a.V + p), visx = vis | x.tm;
            const uint32_t d = a.D[w];
            if (k == 0) *acc_lo = *acc_hi = 0;
            team_sync(team);
            bool active = visx != kAll;
            const int4 *cp = a.col4 + (__ldg(a.slice_off + (p >> a.log2C)) >> 2) + (p & (a.C - 1));
            const int4 pad = make_int4(pp, pp, pp, pp);
            uint64_t acc = 0;
            for (int32_t g = 2 * k; g < ng; g += 2 * kTeam) {
                if (!__any_sync(kFull, active)) break;
                if (!active) continue;
                int4 c0 = __ldg(cp + (int64_t)g * a.C), c1 = pad;
                if (g + 1 < ng) c1 = __ldg(cp + (int64_t)(g + 1) * a.C);
                ALB_CHECK_ID4(c0, a.npad, pp, &a.ctl->err);
                ALB_CHECK_ID4(c1, a.npad, pp, &a.ctl->err);
                const uint64_t f = ms_ld(x.F + c0.x) | ms_ld(x.F + c0.y) | ms_ld(x.F + c0.z) |
                                   ms_ld(x.F + c0.w) | ms_ld(x.F + c1.x) | ms_ld(x.F + c1.y) |
                                   ms_ld(x.F + c1.z) | ms_ld(x.F + c1.w);
                cnt.bytes += 96;
                if (f & ~acc) {  // to the team's other warps, and from them
                    acc |= f;
                    acc |= (uint64_t)atomicOr(acc_lo, (unsigned)acc) |
                           ((uint64_t)atomicOr(acc_hi, (unsigned)(acc >> 32)) << 32);
                }
                if (c1.w == pp || (acc | visx) == kAll) active = false;
            }
            team_sync(team);
            if (k == 0) {
                cnt.bytes += 8;
                cnt.bytes += ms_pull_fold(a, x, w, vis,
                                          (uint64_t)*acc_lo | ((uint64_t)*acc_hi << 32), d, cnt);
            }
            // (the words are cleared by the warp that folds, whose team waits
            // for it at the next word's first barrier)
        }
    }
}

__device__ __forceinline__ uint64_t warp_or64(uint64_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v |= __shfl_xor_sync(kFull, v, o);
    return v;
}

// Long rows (kept out of the slices), head pass: one warp per long row some
// root has not visited ORs the frontier words of its first kLongChunk
// sources, 32 per step (fetched where the nonzero bitmap has a bit when filt
// is set), and stops once every root is accounted for. New bits go into N[p]
// by atomicOr (the slice pass wrote 0 there). A row still missing roots with
// sources left joins the continuation list (nbig[L % 3], big, big_base) for
// k_ms_bu_long_tail; k_ms_bu_long_fin folds N[p] into the state.
// Sources [st, en) of one long row, 128 per step: each lane loads four
// source ids, then their four frontier words, all before using any of them,
// and keeps a private OR; the warp combines the lanes once per step.
template <bool kEarly>
__device__ __forceinline__ uint64_t ms_long_scan(const MsArgs &a, const uint64_t *F,
                                                 const uint32_t *Az, int filt, int64_t st,
                                                 int64_t en, uint64_t acc, uint64_t vis,
                                                 unsigned long long &bytes) {
    const int lane = threadIdx.x & 31;
    uint64_t mine = 0;
    for (int64_t e0 = st; e0 < en; e0 += 128) {
        int32_t c[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t e = e0 + 32 * u + lane;
            c[u] = e < en ? __ldg(a.lcol + e) : -1;
            if (c[u] >= 0) ALB_CHECK_ID(c[u], a.n, -1, &a.ctl->err);
        }
        int fetched = 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (c[u] >= 0 && (!filt || ((ms_ld(Az + (c[u] >> 5)) >> (c[u] & 31)) & 1u))) {
                mine |= ms_ld(F + c[u]);
                fetched++;
            }
        }
        // columns (and bitmap words when filtering), frontier words fetched
        const int64_t ne = min((int64_t)128, en - e0);
        bytes += (filt ? 8 : 4) * ne + 8 * (unsigned long long)warp_sum(fetched);
        if (kEarly && ((acc | warp_or64(mine)) | vis) == kAll) break;
    }
    return acc | warp_or64(mine);
}

// Long row p reached by the roots nb (not in vis) this level: visited word,
// nonzero and done bitmaps, counters. One thread per row.
__device__ __forceinline__ void ms_long_fold(const MsArgs &a, int32_t p, uint64_t nb, uint64_t vis,
                                             uint32_t *An, MsCounts &c) {
    const uint64_t nv = vis | nb;
    a.V[p] = nv;
    const uint32_t bit = 1u << (p & 31);
    atomicOr(An + (p >> 5), bit);
    const int pc = __popcll(nb);
    const int32_t od = __ldg(a.odeg + p);
    c.n++;
    c.bits += pc;
    c.mo += od;
    c.edges += (unsigned long long)pc * od;
    if (nv == kAll) {
        c.done++;
        c.mi += __ldg(a.ideg + p);
        const uint32_t od2 = atomicOr(a.D + (p >> 5), bit);
        c.full += (od2 != kFull && (od2 | bit) == kFull);
    }
}

// Head pass over the long rows: a warp loads the position, visited word and
// offsets of 32 of its rows at once (one per lane), then scans the first
// kLongChunk sources of every one some root has not visited. A row settled
// by its head (every root accounted for, or no sources left) is folded in
// here; the rest go on the continuation list for ms_long_tail with their
// new bits ORed into N[p], and ms_long_fin folds them in.
template <bool kEarly>
__device__ __forceinline__ void ms_long_head(const MsArgs &a, const MsStep &x, int filt,
                                             unsigned long long *cont, MsCounts &cnt) {
    const uint64_t *F = x.F;
    uint64_t *N = x.N;
    const int lane = threadIdx.x & 31;
    const uint64_t tm = x.tm;  // roots the push handles: not waited for
    const int64_t gw = x.gw, nwarps = x.nwarps;
    unsigned long long bytes = 0;
    // rows stay strided over the warps (row gw + k * nwarps goes to warp gw),
    // but a warp loads the metadata of its next 32 rows at once, one per lane
    for (int64_t i0 = gw; i0 < a.nlong; i0 += 32 * nwarps) {
        const int64_t i = i0 + lane * nwarps;
        int32_t p_l = 0;
        uint64_t vis_l = kAll;
        int64_t st_l = 0, en_l = 0;
        if (i < a.nlong) {
            p_l = __ldg(a.lrow + i);
            st_l = __ldg(a.lptr + i);
            en_l = __ldg(a.lptr + i + 1);
            vis_l = ms_ld(a.V + p_l);
        }
        unsigned todo = __ballot_sync(kFull, (vis_l | tm) != kAll);
        while (todo) {
            const int b = __ffs(todo) - 1;
            todo &= todo - 1;
            const int32_t p = __shfl_sync(kFull, p_l, b);
            const uint64_t vis = __shfl_sync(kFull, vis_l, b);
            const int64_t st = __shfl_sync(kFull, st_l, b), en = __shfl_sync(kFull, en_l, b);
            const int64_t hen = min(en, st + kLongChunk);
            bytes += 24;
            const uint64_t acc =
                ms_long_scan<kEarly>(a, F, x.Az, filt, st, hen, 0ull, vis | tm, bytes);
            const uint64_t nb = acc & ~vis;
            if (lane == 0) {
                if ((acc | vis | tm) != kAll && hen < en) {
                    if (nb) atomicOr((unsigned long long *)N + p, (unsigned long long)nb);
                    const unsigned long long nch =
                        (unsigned long long)((en - hen + kLongChunk - 1) / kLongChunk);
                    const unsigned long long old = atomicAdd(cont, (1ull << kMsBigShift) | nch);
                    const int64_t idx = (int64_t)(old >> kMsBigShift);
                    a.big[idx] = (int32_t)(i0 + b * nwarps);
                    a.big_base[idx] = (int64_t)(old & kMsBigMask);
                } else if (nb) {
                    N[p] = nb;  // the slice pass wrote 0 here
                    ms_long_fold(a, p, nb, vis, x.An, cnt);
                }
            }
        }
    }
    if (lane == 0) cnt.bytes += bytes;
}

// Tail pass: chunk k of continuation entry jj covers sources
// [lptr[i] + (1 + k - big_base[jj]) * kLongChunk, ...) of long row i = big[jj];
// the scan starts from the bits N[p] already holds so it can stop early.
template <bool kEarly>
__device__ __forceinline__ void ms_long_tail(const MsArgs &a, const MsStep &x, int filt,
                                             unsigned long long ctr, MsCounts &cnt) {
    const int64_t nrows = (int64_t)(ctr >> kMsBigShift);
    const int64_t total = (int64_t)(ctr & kMsBigMask);
    const uint64_t *F = x.F;
    uint64_t *N = x.N;
    const int lane = threadIdx.x & 31;
    const uint64_t tm = x.tm;  // roots the push handles: not waited for
    unsigned long long bytes = 0;
    for (int64_t k = x.gw; k < total; k += x.nwarps) {
        int64_t lo = 0, hi = nrows - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if (a.big_base[mid] <= k) lo = mid;
            else hi = mid - 1;
        }
        const int32_t i = a.big[lo];
        const int32_t p = __ldg(a.lrow + i);
        const uint64_t vis = ms_ld(a.V + p);
        const uint64_t have = __ldcg((const unsigned long long *)N + p);
        if ((have | vis | tm) == kAll) continue;
        const int64_t st = __ldg(a.lptr + i) + (1 + k - a.big_base[lo]) * kLongChunk;
        const int64_t en = min(__ldg(a.lptr + i + 1), st + kLongChunk);
        bytes += 24;
        const uint64_t acc = ms_long_scan<kEarly>(a, F, x.Az, filt, st, en, have, vis | tm, bytes);
        const uint64_t nb = acc & ~vis & ~have;
        if (lane == 0 && nb) atomicOr((unsigned long long *)N + p, (unsigned long long)nb);
    }
    if (lane == 0) cnt.bytes += bytes;
}

// Long rows on the continuation list: thread per entry folds N[p] (head and
// tail bits) into the state.
__device__ __forceinline__ void ms_long_fin(const MsArgs &a, const MsStep &x,
                                            unsigned long long ctr, MsCounts &cnt) {
    const int64_t nrows = (int64_t)(ctr >> kMsBigShift);
    for (int64_t e = x.gw * 32 + (threadIdx.x & 31); e < nrows; e += x.nwarps * 32) {
        const int32_t p = __ldg(a.lrow + a.big[e]);
        const uint64_t nb = __ldcg((const unsigned long long *)x.N + p);
        if (nb) ms_long_fold(a, p, nb, ms_ld(a.V + p), x.An, cnt);
    }
}

// Push of the roots in tmask during a bottom-up level (after the pull): the
// roots nb reach v (nb: the edge's roots not in v's visited word as read).
// The new roots are claimed on V[v] itself (atomicOr), so concurrent pushers
// and the pull's own discoveries are never counted twice, and the level's
// state and counters are updated in place.
__device__ __forceinline__ void ms_tclaim(const MsArgs &a, uint64_t *N, uint32_t *An, int32_t v,
                                          uint64_t nb, MsCounts &c) {
    if (!nb) return;
    const uint32_t bit = 1u << (v & 31);
    const uint64_t oldv = atomicOr((unsigned long long *)a.V + v, (unsigned long long)nb);
    nb &= ~oldv;
    if (!nb) return;
    const uint64_t oldn = atomicOr((unsigned long long *)N + v, (unsigned long long)nb);
    c.bytes += 16;  // V and N words written
    const int pc = __popcll(nb);
    const int32_t od = __ldg(a.odeg + v);
    c.bits += pc;
    c.edges += (unsigned long long)pc * od;
    if (oldn == 0) {  // v enters the next frontier
        c.n++;
        c.mo += od;
        atomicOr(An + (v >> 5), bit);
    }
    if ((oldv | nb) == kAll) {
        c.done++;
        c.mi += __ldg(a.ideg + v);
        const uint32_t od2 = atomicOr(a.D + (v >> 5), bit);
        c.full += (od2 != kFull && (od2 | bit) == kFull);
    }
}

// Four pushed edges per lane (v[k] < 0: none), roots f[k] reaching v[k]
// this level: the done words and the target words of all four are requested
// before the first atomic, so one lane keeps eight loads in flight instead
// of two. Top-down (kPush false): only two small words are read per edge,
// v's done bit (D, 1 bit per row, stays in L2) and N[v] (so that the many
// pushes into a hub stop issuing atomics once its word holds their bits); f
// is ORed in without masking by V[v], and the finish removes the roots
// that had already visited v. A push that finds N[v] empty marks v in the
// next nonzero bitmap An (setting a bit is idempotent, so racing pushers need
// no claim); the next queue is compacted from An afterwards. kPush: the push
// of the tmask roots, ms_tclaim against V (D can change during that kernel
// and is read through L2).
template <bool kPush>
__device__ __forceinline__ void ms_push4(const MsArgs &a, uint64_t *N, uint32_t *An,
                                         const int32_t (&v)[4], const uint64_t (&f)[4],
                                         MsCounts &c) {
    uint32_t dw[4];
    uint64_t cur[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        dw[k] = kFull;
        cur[k] = 0;
        if (v[k] >= 0) {
            dw[k] = kPush ? __ldcg(a.D + (v[k] >> 5)) : ms_ld(a.D + (v[k] >> 5));
            cur[k] = __ldcg((const unsigned long long *)(kPush ? a.V : N) + v[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (v[k] < 0 || ((dw[k] >> (v[k] & 31)) & 1u)) continue;  // every root has visited v
        if (kPush) {
            c.bytes += 16;  // column, done bit, visited probe
            ms_tclaim(a, N, An, v[k], f[k] & ~cur[k], c);
        } else if (f[k] & ~cur[k]) {
            atomicOr((unsigned long long *)N + v[k], (unsigned long long)f[k]);
            if (!cur[k]) atomicOr(An + (v[k] >> 5), 1u << (v[k] & 31));
        }
    }
}

// A row of d > kBigRow edges onto the list that all warps share (ms_push_big).
template <bool kPush>
__device__ __forceinline__ void ms_put_big(const MsArgs &a, unsigned long long *big_slot, int32_t u,
                                           int64_t d) {
    const unsigned long long nch = (unsigned long long)((d + kBigChunk - 1) / kBigChunk);
    const unsigned long long old = atomicAdd(big_slot, (1ull << kMsBigShift) | nch);
    const int64_t idx = (int64_t)(old >> kMsBigShift);
    (kPush ? a.pbig : a.big)[idx] = u;
    (kPush ? a.pbig_base : a.big_base)[idx] = (int64_t)(old & kMsBigMask);
}

// Row u's entry in a queue made at the level that pushes it: a big row is
// listed at once and stands in the queue as ~u, which ms_push_rows passes over,
// so that both kinds can be pushed in one step.
template <bool kPush>
__device__ __forceinline__ int32_t ms_queued(const MsArgs &a, unsigned long long *big_slot, int32_t u) {
    if (!a.any_big) return u;
    const int32_t d = __ldg(a.odeg + u);
    if (d <= kBigRow) return u;
    ms_put_big<kPush>(a, big_slot, u, d);
    return ~u;
}

// Top-down push over the frontier queue. kPush: the push of a bottom-up
// level's tmask roots, over the queue ms_tq built (next-parity queue and
// counters, which that level leaves unused), with the state updated in place.
template <bool kPush>
__device__ __forceinline__ void ms_push_rows(const MsArgs &a, const MsStep &x,
                                             const int32_t *Q, int64_t qlen,
                                             unsigned long long *big_slot, MsCounts &cnt) {
    const uint64_t *F = x.F;
    const uint64_t tm = kPush ? x.tm : kAll;
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = x.nwarps;
    int G = 32;  // frontier rows per warp: enough to keep every warp busy
    while (G > 1 && (int64_t)(G >> 1) * nwarps >= qlen) G >>= 1;
    const int64_t stride = nwarps * G;
    for (int64_t cb = x.gw * G; cb < qlen; cb += stride) {
        const int64_t i = cb + lane;
        int32_t u = (lane < G && i < qlen) ? __ldcg(Q + i) : -1;
        if (u >= 0) ALB_CHECK_ID(u, a.n, -1, &a.ctl->err);
        int64_t st = 0, d = 0;
        uint64_t f = 0;
        if (u >= 0) {
            st = __ldg(a.prow + u);
            d = __ldg(a.prow + u + 1) - st;
            f = ms_ld(F + u) & tm;
            if (kPush) cnt.bytes += 20;  // queue entry, row offsets, frontier word
            if (d > kBigRow) {  // pushed in chunks by all warps
                ms_put_big<kPush>(a, big_slot, u, d);
                d = 0;
            }
        }
        // the rows' edges flattened over the lanes (at most 32 * kBigRow): row
        // j's start at ex of lane j, ascending
        const int inc = warp_inclusive_scan((int)d);
        const int T = __shfl_sync(kFull, inc, 31);
        const int ex = inc - (int)d;
        for (int e0 = 0; e0 < T; e0 += 128) {  // (the same for all lanes: they exchange rows)
            int32_t v[4];
            uint64_t ff[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int e = e0 + 32 * k + lane;
                int jj = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(kFull, ex, jj + step) <= e) jj += step;
                const int64_t at = __shfl_sync(kFull, st - ex, jj) + e;
                ff[k] = __shfl_sync(kFull, f, jj);
                v[k] = -1;
                if (e < T) {
                    v[k] = __ldg(a.pcol + at);
                    ALB_CHECK_ID(v[k], a.n, -1, &a.ctl->err);
                }
            }
            ms_push4<kPush>(a, x.N, x.An, v, ff, cnt);
        }
    }
}

// Long frontier rows in kBigChunk-edge chunks over all warps. Each warp
// takes a contiguous run of chunks: it finds the row of its first chunk by
// binary search over the chunk bases (monotone in the list index) and walks
// forward from there.
template <bool kPush>
__device__ __forceinline__ void ms_push_big(const MsArgs &a, const MsStep &x,
                                            unsigned long long ctr, MsCounts &cnt) {
    const uint64_t tm = kPush ? x.tm : kAll;
    const int32_t *big = kPush ? a.pbig : a.big;
    const int64_t *big_base = kPush ? a.pbig_base : a.big_base;
    const int64_t nbig = (int64_t)(ctr >> kMsBigShift);
    const int64_t total = (int64_t)(ctr & kMsBigMask);
    const uint64_t *F = x.F;
    const int lane = threadIdx.x & 31;
    const int64_t per = (total + x.nwarps - 1) / x.nwarps;
    const int64_t k0 = x.gw * per, k1 = min(total, k0 + per);
    if (k0 >= k1) return;  // warp-uniform: whole warps leave
    int64_t lo = 0, hi = nbig - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (big_base[mid] <= k0) lo = mid;
        else hi = mid - 1;
    }
    int64_t base = big_base[lo];
    int64_t next = lo + 1 < nbig ? big_base[lo + 1] : total;
    int32_t u = big[lo];
    int64_t st = __ldg(a.prow + u), d = __ldg(a.prow + u + 1) - st;
    uint64_t f = ms_ld(F + u) & tm;
    for (int64_t k = k0; k < k1; k++) {
        while (k >= next) {  // the run crosses into the next long row
            lo++;
            base = next;
            next = lo + 1 < nbig ? big_base[lo + 1] : total;
            u = big[lo];
            st = __ldg(a.prow + u);
            d = __ldg(a.prow + u + 1) - st;
            f = ms_ld(F + u) & tm;
        }
        const int64_t c = k - base;
        const int64_t e1 = min(d, (c + 1) * kBigChunk);
        static_assert(kBigChunk == 128, "four edges per lane per chunk");
        int32_t v[4];
        uint64_t ff[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int64_t e = c * kBigChunk + 32 * q + lane;
            v[q] = e < e1 ? __ldg(a.pcol + st + e) : -1;
            if (v[q] >= 0) ALB_CHECK_ID(v[q], a.n, -1, &a.ctl->err);
            ff[q] = f;
        }
        ms_push4<kPush>(a, x.N, x.An, v, ff, cnt);
    }
}

// The set bits of 32 words (lane l holds word l) as row numbers 0 .. 1023,
// kRowBuf at a time in the warp's buffer.
constexpr int kRowBuf = 64;  // (small: see the shared memory of ms_grid.cu)
struct MsBits {
    uint16_t *buf;
    uint32_t rem;
    int at, tot, base;  // this lane's next row's index; all; those before the buffer's
    __device__ __forceinline__ MsBits(uint16_t *b, uint32_t m) : buf(b), rem(m), base(0) {
        const int inc = warp_inclusive_scan(__popc(m));
        at = inc - __popc(m);
        tot = __shfl_sync(kFull, inc, 31);
    }
    // the next rows into the buffer; how many (0: no more)
    __device__ __forceinline__ int next() {
        __syncwarp();
        const int n = min(kRowBuf, tot - base);
        if (n <= 0) return 0;
        for (; rem && at < base + kRowBuf; rem &= rem - 1)
            buf[at++ - base] = (uint16_t)((threadIdx.x & 31) * 32 + __ffs(rem) - 1);
        base += n;
        __syncwarp();
        return n;
    }
};

// Words a warp takes at a time where it lists bits: 32 keep the atomics on
// the queue's counter few, but a small graph has too few words for that to
// leave every warp something (a whole 32 of R-MAT scale 16's words held one
// warp 32 round trips).
__device__ __forceinline__ int ms_words_at_once(const MsArgs &a, const MsStep &x) {
    const int64_t per = (a.nwords + x.nwarps - 1) / x.nwarps;
    return per >= 32 ? 32 : per < 1 ? 1 : (int)per;
}

// Frontier-nonzero bitmap Az -> queue, before a top-down level that follows a
// bottom-up one (or none). Big rows are listed (big_slot).
__device__ __forceinline__ void ms_compact(const MsArgs &a, const MsStep &x, int32_t *Q,
                                           unsigned long long *qslot,
                                           unsigned long long *big_slot) {
    const int lane = threadIdx.x & 31, per = ms_words_at_once(a, x);
    for (int64_t w0 = x.gw * per; w0 < a.nwords; w0 += x.nwarps * per) {
        const int64_t w = w0 + lane;
        uint32_t m = lane < per && w < a.nwords ? ms_ld(x.Az + w) : 0u;
        const int cnt = __popc(m);
        const int inc = warp_inclusive_scan(cnt);
        const int total = __shfl_sync(kFull, inc, 31);
        if (total == 0) continue;
        unsigned long long base = 0;
        if (lane == 31) base = atomicAdd(qslot, (unsigned long long)total);
        base = __shfl_sync(kFull, base, 31);
        int64_t o = (int64_t)base + inc - cnt;
        for (; m; m &= m - 1) Q[o++] = ms_queued<false>(a, big_slot, (int32_t)(w * 32 + __ffs(m) - 1));
    }
}

// Before a top-down level: the next slot and its nonzero bitmap cleared.
__device__ __forceinline__ void ms_zero_next(const MsArgs &a, const MsStep &x) {
    const int64_t tid = x.gw * 32 + (threadIdx.x & 31), str = x.nwarps * 32;
    for (int64_t i = tid; i < a.npad / 2; i += str)
        reinterpret_cast<uint4 *>(x.N)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int64_t w = tid; w < a.nwords; w += str) x.An[w] = 0u;
}

// After a top-down level's pushes, which only marked the nonzero bitmap: its
// rows fold the new frontier words into V, are counted and go on the next
// queue; rows reached only by roots that had visited them leave the frontier
// (their queue entry is -1).
__device__ __forceinline__ void ms_finish(const MsArgs &a, const MsStep &x, uint16_t *buf,
                                          int32_t *NQ, unsigned long long *qslot, MsCounts &c) {
    const int lane = threadIdx.x & 31, per = ms_words_at_once(a, x);
    for (int64_t w0 = x.gw * per; w0 < a.nwords; w0 += x.nwarps * per) {
        MsBits bits(buf, lane < per && w0 + lane < a.nwords ? __ldcg(x.An + w0 + lane) : 0u);
        if (bits.tot == 0) continue;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(qslot, (unsigned long long)bits.tot);
        base = __shfl_sync(kFull, base, 0);
        while (const int k = bits.next()) {
            for (int i = lane; i < k; i += 32) {
                const int32_t v = (int32_t)(w0 * 32) + buf[i];
                const uint64_t raw = __ldcg((const unsigned long long *)x.N + v);
                const uint64_t old = ms_ld(a.V + v);  // only this thread writes V[v] here
                const uint64_t nb = raw & ~old;       // the pushes did not mask by V
                const uint32_t bit = 1u << (v & 31);
                NQ[base + i] = nb ? v : -1;
                if (nb != raw) x.N[v] = nb;
                if (!nb) {
                    atomicAnd(x.An + (v >> 5), ~bit);
                    continue;
                }
                const uint64_t nv = old | nb;
                a.V[v] = nv;
                const int pc = __popcll(nb);
                const int32_t od = __ldg(a.odeg + v);
                c.n++;
                c.bits += pc;
                c.mo += od;
                c.edges += (unsigned long long)pc * od;
                if (nv == kAll) {  // (old was not: nb is not empty)
                    c.done++;
                    c.mi += __ldg(a.ideg + v);
                    const uint32_t od2 = atomicOr(a.D + (v >> 5), bit);
                    c.full += (od2 != kFull && (od2 | bit) == kFull);
                }
            }
            base += k;
        }
    }
}

// Queue of the rows in the level's frontier that hold a tmask root, for the
// push after a bottom-up level's pull, big rows listed. A warp takes 32 bitmap
// words at a time and reads the frontier words of the set bits only.
__device__ __forceinline__ void ms_tq(const MsArgs &a, const MsStep &x, int32_t *Q,
                                      unsigned long long *qslot, unsigned long long *big_slot,
                                      MsCounts &c) {
    const int lane = threadIdx.x & 31, per = ms_words_at_once(a, x);
    for (int64_t w0 = x.gw * per; w0 < a.nwords; w0 += x.nwarps * per) {
        const uint32_t mine = lane < per && w0 + lane < a.nwords ? ms_ld(x.Az + w0 + lane) : 0u;
        c.bytes += 4 + 8 * __popc(mine);  // bitmap word, the frontier words it selects
        uint32_t hits = 0;                // lane q: the rows of word q
        for (unsigned words = __ballot_sync(kFull, mine != 0); words; words &= words - 1) {
            const int q = __ffs(words) - 1;
            const uint32_t m = __shfl_sync(kFull, mine, q);
            const bool hit = ((m >> lane) & 1u) && (ms_ld(x.F + (w0 + q) * 32 + lane) & x.tm);
            const unsigned hm = __ballot_sync(kFull, hit);
            if (lane == q) hits = hm;
        }
        const int inc = warp_inclusive_scan(__popc(hits));
        const int tot = __shfl_sync(kFull, inc, 31);
        if (tot == 0) continue;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(qslot, (unsigned long long)tot);
        base = __shfl_sync(kFull, base, 0);
        int64_t o = (int64_t)base + inc - __popc(hits);
        c.bytes += 4 * __popc(hits);  // queue entries
        for (; hits; hits &= hits - 1)
            Q[o++] = ms_queued<true>(a, big_slot, (int32_t)((w0 + lane) * 32 + __ffs(hits) - 1));
    }
}

// Per-root size of the frontier level L produced (S[j+1]) for ms_decide's
// choice of pushed roots, in push degrees (MsSample). The long rows
// are counted exactly (they carry most of the degree in a skewed graph); the
// others on one bitmap word in every kSampleStride, scaled by the stride. The
// sampled word's offset inside its stride cycles with the stride index: rows
// are sorted by length inside sigma windows, and a fixed offset would sample
// one rank of length only. Warp per sampled word or per 32 long rows; lane i
// keeps roots i and i + 32.
struct MsSampleRoom {
    unsigned long long deg[64];
};
// Only a top-down level can be followed by a level with pushed roots. A
// frontier under n / kSampleMinDiv rows is not sampled: every root's estimate
// stays 0, and a bottom-up level after it pushes all of them (a push over so
// few rows is cheaper than any pull).
__device__ __forceinline__ bool ms_samples(const MsArgs &a, int64_t budget, int dir, int64_t nf) {
    return budget > 0 && dir == ALB_DIR_TOPDOWN && nf * kSampleMinDiv >= a.n;
}

// All threads of a block.
__device__ __forceinline__ void ms_sample(const MsArgs &a, const MsStep &x, MsSampleRoom &s,
                                          unsigned long long *bytes_out) {
    const uint64_t *N = x.N;
    const uint32_t *An = x.An;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 64) s.deg[threadIdx.x] = 0;
    __syncthreads();
    unsigned long long d0 = 0, d1 = 0, bytes = 0;
    const int64_t nsamp = (a.nwords + kSampleStride - 1) / kSampleStride;
    const int64_t ntask = nsamp + (a.nlong + 31) / 32;
    for (int64_t t = x.gw; t < ntask; t += x.nwarps) {
        uint64_t f = 0;
        int32_t od = 0;
        unsigned wt;
        if (t < nsamp) {
            const int64_t w = min(t * kSampleStride + ((t * 13) & (kSampleStride - 1)), a.nwords - 1);
            const uint32_t m = ms_ld(An + w);
            if (lane == 0) bytes += 4;
            if (!m) continue;  // warp-uniform
            const int64_t p = w * 32 + lane;
            // long rows (long_row > 0) are counted below
            if (((m >> lane) & 1u) && (a.long_row <= 0 || __ldg(a.ideg + p) <= a.long_row)) {
                f = __ldcg((const unsigned long long *)N + p);
                od = __ldg(a.odeg + p);
                bytes += 16;  // length, frontier word, push degree
            }
            wt = kSampleStride;
        } else {
            const int64_t e = (t - nsamp) * 32 + lane;
            if (e < a.nlong) {
                const int32_t p = __ldg(a.lrow + e);
                f = __ldcg((const unsigned long long *)N + p);
                if (f) od = __ldg(a.odeg + p);
                bytes += f ? 16 : 12;
            }
            wt = 1;
        }
        unsigned m = __ballot_sync(kFull, f != 0);
        while (m) {
            const int q = __ffs(m) - 1;
            m &= m - 1;
            const uint64_t xq = __shfl_sync(kFull, f, q);
            const unsigned long long oq = (unsigned long long)(unsigned)__shfl_sync(kFull, od, q) * wt;
            if ((xq >> lane) & 1ull) d0 += oq;
            if ((xq >> (lane + 32)) & 1ull) d1 += oq;
        }
    }
    if (d0) atomicAdd(&s.deg[lane], d0);
    if (d1) atomicAdd(&s.deg[lane + 32], d1);
    bytes = warp_sum(bytes);
    if (lane == 0 && bytes) atomicAdd(bytes_out, bytes);
    __syncthreads();
    if (threadIdx.x < 64 && s.deg[threadIdx.x])
        atomicAdd(&a.smp->deg[threadIdx.x], s.deg[threadIdx.x]);
}

__device__ inline void ms_feature_ctl(const MsCtl &m, BfsCtl &c) {
    memset(&c, 0, sizeof(c));
    c.level = m.level;
    c.n = m.n;
    c.nwords = m.nwords;
    c.nf = m.nf;
    c.mf = m.mf;
    c.prev_nf = m.prev_nf;
    c.nu = m.nu;
    c.mu = m.mu;
    c.active_words = m.active_words;
    c.prev_dir = m.prev_dir;
    c.policy = m.policy;
    c.alpha = m.alpha;
    c.beta = m.beta;
    c.feat_mean_deg = m.feat_mean_deg;
    c.feat_skew = m.feat_skew;
}

// What level L came to.
struct MsSums {
    unsigned long long n, bits, full, done, mo, mi, edges, bytes;
};

// The level's end: what it found goes into the control block. dir: the
// direction that it ran.
__device__ __forceinline__ void ms_rollover(MsCtl &c, int dir, const MsSums &k) {
    c.prev_nf = c.nf;
    c.nf = (int64_t)k.n;
    c.mf = (int64_t)k.mo;
    c.nu -= (int64_t)k.done;  // vertices every root has visited
    c.mu -= (int64_t)k.mi;
    c.active_words -= (int64_t)k.full;
    c.pairs += (int64_t)k.bits;
    c.edges += (int64_t)k.edges;
    c.q_valid = dir == ALB_DIR_TOPDOWN;
    c.prev_dir = dir;
    c.dir = dir;
    if (dir == ALB_DIR_TOPDOWN) c.levels_td++; else c.levels_bu++;
    c.level++;
    if (k.n == 0) c.done = 1;
    if (!c.done && c.level >= c.level_cap) {  // cannot happen in a BFS: refuse
        c.done = 1;
        c.err = ALB_ERR_DEVICE;
    }
}

// The next level's settings but for the pushed roots (one thread). next: its
// direction.
__device__ __forceinline__ void ms_set_next(const MsArgs &a, MsCtl &c, int next) {
    c.dir = next;
    // nonzero-bitmap filter when under 1/8 of all entries point into the frontier
    c.filt = c.mf < c.m_in / 8;
    c.need_flush = !c.done && (c.level - c.base + 1 >= a.K);
}

// Roots pushed instead of pulled, at the first bottom-up level after a
// top-down one (where the roots' frontiers differ most in size: some are
// still a few rows wide when most cover a good part of the graph): the
// roots with the smallest estimated push edges, in ascending order while
// their running sum stays within the budget. Later bottom-up levels pull
// every root. A full warp; room: 128 words of shared memory; e0, e1: the
// estimates of roots lane and lane + 32.
__device__ __forceinline__ unsigned long long ms_pushed_roots(unsigned long long e0,
                                                              unsigned long long e1,
                                                              unsigned long long lim,
                                                              unsigned long long used,
                                                              unsigned long long *room) {
    const int i = threadIdx.x & 31;
    unsigned long long *val = room, *cum = room + 64;
    // rank of roots i and i + 32 by (estimate, root index)
    int r0 = 0, r1 = 0;
    for (int q = 0; q < 32; q++) {
        const unsigned long long a0 = __shfl_sync(kFull, e0, q), a1 = __shfl_sync(kFull, e1, q);
        r0 += (a0 < e0 || (a0 == e0 && q < i)) + (a1 < e0);
        r1 += (a0 <= e1) + (a1 < e1 || (a1 == e1 && q < i));
    }
    val[r0] = e0;
    val[r1] = e1;
    __syncwarp();
    // running sums in rank order: lane i holds ranks 2i and 2i + 1
    const unsigned long long v0 = val[2 * i], v1 = val[2 * i + 1];
    const unsigned long long inc = warp_inclusive_scan(v0 + v1);
    cum[2 * i] = inc - v1;
    cum[2 * i + 1] = inc;
    __syncwarp();
    const unsigned lo = __ballot_sync(kFull, cum[r0] <= lim && ((used >> i) & 1ull));
    const unsigned hi = __ballot_sync(kFull, cum[r1] <= lim && ((used >> (i + 32)) & 1ull));
    return (unsigned long long)lo | ((unsigned long long)hi << 32);
}

}  // namespace alb
