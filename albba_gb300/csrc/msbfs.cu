// Bit-parallel multi-source BFS: up to 64 roots per uint64 word, one pass
// over the SELL-C-sigma matrix per level for all roots. No counterpart in the
// reference (bfs/src/bfs_SELLCSv2.c runs one root from row 0).
//
// Per position p (sorted-position space, as in bfs.cu):
//   V[p]     roots that have visited p (unused root bits preset)
//   S[l][p]  roots whose level-l frontier contains p. S[l] is both the
//            frontier of level l and the record of level l: a root's level at
//            p is the l whose S[l][p] holds its bit, so the int32 output is
//            written once, at the end, as full 256-byte rows.
//   D        one bit per position: V[p] == ~0 (the bypass test)
//   A[l & 1] one bit per position: S[l][p] != 0. The 2 MB-per-2^24-vertex
//            bitmap stays in L2 where the 8-byte frontier words do not, and a
//            bottom-up gather fetches S[l][c] only when c's bit is set.
//
// bottom-up (ms_pull): warp per 32 positions; a full D word is skipped; each
//   lane ORs S[l] over its row with 16-byte column loads and stops when every
//   root has visited or reached it ((acc | V) == ~0) or at the row padding.
// top-down (ms_push_rows): warp-cooperative push over the frontier queue; targets
//   receive atomicOr(S[l+1][v], S[l][u]) (64-bit atomics) and are marked in
//   A[l + 1], from which ms_finish takes the roots that had visited them out
//   again, counts them and lists the next queue.
// The whole search runs as one cooperative kernel (ms_grid.cu); here are the
// level kernels of the host-driven loop and of the profile, the level output
// and the entry points.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "graph.h"
#include "ms.cuh"
#include "ms_grid.h"
#include "selector.cuh"

namespace alb {

// Bound of the cooperative kernel's barrier waits, as the single-root kernels'.
constexpr uint64_t kMsBarrierNs = 4ull * 1000 * 1000 * 1000;

// --------------------------------------- the host loop's kernels, a step each

__device__ __forceinline__ MsStep ms_step(const MsArgs &a, int j) {
    return ms_step(a, a.ctl->level, j, a.ctl->tmask, false);
}

// Adds what the warps found to the level's counters.
__device__ __forceinline__ void ms_count(const MsArgs &a, int L, const MsCounts &c) {
    const int k = (L + 1) % 3;
    const unsigned long long n = warp_sum((unsigned long long)c.n), bits = warp_sum((unsigned long long)c.bits),
                             full = warp_sum((unsigned long long)c.full),
                             done = warp_sum((unsigned long long)c.done), mo = warp_sum(c.mo),
                             mi = warp_sum(c.mi), edges = warp_sum(c.edges), bytes = warp_sum(c.bytes);
    if ((threadIdx.x & 31) != 0) return;
    if (bytes) atomicAdd(&a.ctl->acc_bytes[k], bytes);
    if (!(n | bits | done | full)) return;
    atomicAdd(&a.ctl->acc_n[k], n);
    atomicAdd(&a.ctl->acc_bits[k], bits);
    atomicAdd(&a.ctl->acc_mo[k], mo);
    atomicAdd(&a.ctl->acc_mi[k], mi);
    atomicAdd(&a.ctl->acc_edges[k], edges);
    if (done) atomicAdd(&a.ctl->acc_done[k], done);
    if (full) atomicAdd(&a.ctl->acc_full[k], full);
}

// Initial state, thread per position: a warp covers one bitmap word (npad and
// the grid stride are multiples of 32), so the done word comes from a ballot.
__global__ void k_ms_init(MsArgs a, uint64_t unused) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t str = (int64_t)gridDim.x * blockDim.x;
    uint64_t *S0 = a.S;
    for (int64_t p = tid; p < a.npad; p += str) {
        const bool live = p < a.n && __ldg(a.ideg + p) > 0;
        a.V[p] = live ? unused : kAll;
        S0[p] = 0;
        const unsigned dead = __ballot_sync(kFull, !live);
        if ((threadIdx.x & 31) == 0) {
            const int64_t w = p >> 5;
            a.D[w] = dead;
            a.A[w] = 0;
            a.A[a.nwords + w] = 0;
        }
    }
}

// One block of 64 threads: thread i seeds root i; thread 0 fills the control block.
__global__ void k_ms_roots(MsArgs a, MsInit in) {
    __shared__ unsigned long long s_nf, s_mf, s_pairs, s_edges, s_done_mi, s_full, s_done_v;
    const int i = threadIdx.x;
    if (i == 0) s_nf = s_mf = s_pairs = s_edges = s_done_mi = s_full = s_done_v = 0;
    a.smp->deg[i] = 0;
    __syncthreads();
    if (i < in.nroots) {
        const int32_t p = a.inv[in.roots[i]];
        const uint64_t bit = 1ull << i;
        const unsigned long long oldv = atomicOr((unsigned long long *)a.V + p, bit);
        const unsigned long long olds = atomicOr((unsigned long long *)a.S + p, bit);
        if (olds == 0) {
            a.q0[atomicAdd(&s_nf, 1ull)] = p;
            atomicAdd(&s_mf, (unsigned long long)a.odeg[p]);
            atomicOr(a.A + (p >> 5), 1u << (p & 31));  // level 0: A[0]
        }
        // bit i belongs to root i alone, so every root counts once (its bit
        // may already be set in V when p has no sources: V starts full there)
        (void)oldv;
        atomicAdd(&s_pairs, 1ull);
        atomicAdd(&s_edges, (unsigned long long)a.odeg[p]);
    }
    __syncthreads();
    // positions whose every root bit is now set
    if (i < in.nroots) {
        const int32_t p = a.inv[in.roots[i]];
        if (a.V[p] == kAll) {
            const unsigned long long old = atomicOr(&a.D[p >> 5], 1u << (p & 31));
            if (!(old & (1u << (p & 31)))) {
                atomicAdd(&s_done_v, 1ull);
                atomicAdd(&s_done_mi, (unsigned long long)a.ideg[p]);
                if ((old | (1u << (p & 31))) == kFull) atomicAdd(&s_full, 1ull);
            }
        }
    }
    __syncthreads();
    if (i == 0) {
        MsCtl c;
        ms_start(a, in, (int64_t)s_nf, (int64_t)s_mf, (int64_t)s_pairs, (int64_t)s_edges,
                 (int64_t)s_done_v, (int64_t)s_done_mi, (int64_t)s_full, c);
        c.q_valid = 1;
        c.qn[0] = s_nf;
        *a.ctl = c;
    }
}

// (four blocks an SM, three for the two-group pull: at five and four the loops
// spill: R-MAT scale 19's first pull 198 against 227 us)
constexpr int kMsBuBlock = 256;

template <bool kBypass, bool kEarly, bool kFilt, bool kWide = false>
__global__ void __launch_bounds__(kMsBuBlock, kWide ? 3 : 4) k_ms_bu(MsArgs a, int j) {
    const MsStep x = ms_step(a, j);
    MsCounts cnt;
    ms_pull<kBypass, kEarly, kFilt, kWide>(a, x, a.ctl->grab, INT32_MAX, &a.ctl->work[x.L % 3], cnt);
    ms_count(a, x.L, cnt);
}

template <bool kEarly>
__global__ void k_ms_bu_long(MsArgs a, int j, int filt) {
    if (a.nlong == 0) return;
    const MsStep x = ms_step(a, j);
    MsCounts cnt;
    ms_long_head<kEarly>(a, x, filt, &a.ctl->nbig[x.L % 3], cnt);
    ms_count(a, x.L, cnt);
}

template <bool kEarly>
__global__ void k_ms_bu_long_tail(MsArgs a, int j, int filt) {
    const MsStep x = ms_step(a, j);
    const unsigned long long ctr = a.ctl->nbig[x.L % 3];
    if (ctr == 0) return;
    MsCounts cnt;
    ms_long_tail<kEarly>(a, x, filt, ctr, cnt);
    ms_count(a, x.L, cnt);
}

__global__ void k_ms_bu_long_fin(MsArgs a, int j) {
    const MsStep x = ms_step(a, j);
    const unsigned long long ctr = a.ctl->nbig[x.L % 3];
    if (ctr == 0) return;
    MsCounts cnt;
    ms_long_fin(a, x, ctr, cnt);
    ms_count(a, x.L, cnt);
}

// The queue of the running level's frontier.
__global__ void k_ms_compact(MsArgs a, int j) {
    const MsStep x = ms_step(a, j);
    ms_compact(a, x, (x.L & 1) ? a.q1 : a.q0, &a.ctl->qn[x.L % 3], &a.ctl->nbig[x.L % 3]);
}

__global__ void k_ms_zero_next(MsArgs a, int j) { ms_zero_next(a, ms_step(a, j)); }

// kPush: the push of a bottom-up level's tmask roots over the queue that
// k_ms_tq built (next-parity queue and counters, which that level leaves
// unused), with the state updated in place.
template <bool kPush>
__global__ void k_ms_td(MsArgs a, int j) {
    const MsStep x = ms_step(a, j);
    if (kPush && !x.tm) return;
    const int qp = kPush ? x.L + 1 : x.L;
    MsCounts cnt;
    ms_push_rows<kPush>(a, x, (qp & 1) ? a.q1 : a.q0,
                        (int64_t)a.ctl->qn[qp % 3], &a.ctl->nbig[qp % 3], cnt);
    if (kPush) ms_count(a, x.L, cnt);
}

template <bool kPush>
__global__ void k_ms_td_big(MsArgs a, int j) {
    const MsStep x = ms_step(a, j);
    const unsigned long long ctr = a.ctl->nbig[(kPush ? x.L + 1 : x.L) % 3];
    if (ctr == 0) return;
    MsCounts cnt;
    ms_push_big<kPush>(a, x, ctr, cnt);
    if (kPush) ms_count(a, x.L, cnt);
}

__global__ void k_ms_td_finish(MsArgs a, int j) {
    __shared__ uint16_t buf[32][kRowBuf];
    const MsStep x = ms_step(a, j);
    MsCounts cnt;
    ms_finish(a, x, buf[threadIdx.x >> 5], (x.L & 1) ? a.q0 : a.q1, &a.ctl->qn[(x.L + 1) % 3], cnt);
    ms_count(a, x.L, cnt);
}

// dir: the direction that the level ran.
constexpr int kSampleBlock = 256;
__global__ void __launch_bounds__(kSampleBlock) k_ms_sample(MsArgs a, int j, int dir) {
    __shared__ MsSampleRoom room;
    const MsStep x = ms_step(a, j);
    const int k = (x.L + 1) % 3;
    if (!ms_samples(a, a.ctl->push_budget, dir, (int64_t)a.ctl->acc_n[k])) return;
    ms_sample(a, x, room, &a.ctl->acc_bytes[k]);
}

__global__ void k_ms_tq(MsArgs a, int j) {
    const MsStep x = ms_step(a, j);
    if (!x.tm) return;
    MsCounts cnt;
    ms_tq(a, x, ((x.L + 1) & 1) ? a.q1 : a.q0, &a.ctl->qn[(x.L + 1) % 3],
          &a.ctl->nbig[(x.L + 1) % 3], cnt);
    ms_count(a, x.L, cnt);
}

// Rollover of level L's counters and the device-side decision for L+1.
// dir: the direction level L ran.
__global__ void k_ms_end(MsArgs a, int dir) {
    if (threadIdx.x >= 32) return;
    __shared__ MsCtl s;
    __shared__ unsigned long long room[128];
    // the control block moves between global and shared memory with all 32
    // lanes (8-byte words), not one thread's serial copy
    constexpr int kCtlWords = (int)(sizeof(MsCtl) / 8);
    for (int w = threadIdx.x; w < kCtlWords; w += 32)
        reinterpret_cast<unsigned long long *>(&s)[w] =
            reinterpret_cast<const unsigned long long *>(a.ctl)[w];
    __syncwarp();
    if (threadIdx.x == 0) {
        MsCtl &c = s;
        const int k = (c.level + 1) % 3;
        ms_rollover(c, dir, MsSums{c.acc_n[k], c.acc_bits[k], c.acc_full[k], c.acc_done[k],
                                   c.acc_mo[k], c.acc_mi[k], c.acc_edges[k], c.acc_bytes[k]});
        // zero the slots level L+1 accumulates into after the next rollover
        const int z = (c.level + 1) % 3;
        c.acc_n[z] = c.acc_mo[z] = c.acc_mi[z] = c.acc_full[z] = c.acc_bits[z] = 0;
        c.acc_edges[z] = c.qn[z] = c.acc_bytes[z] = c.acc_done[z] = c.nbig[z] = c.work[z] = 0;
        // a bottom-up level's push of its tmask roots used the new level's
        // long-row counter and, after a bottom-up level, its queue count
        c.nbig[c.level % 3] = 0;
        if (!c.q_valid) c.qn[c.level % 3] = 0;
    }
    __syncwarp();
    // decide the next level (one warp; the MLP runs here when loaded)
    BfsCtl fc;
    ms_feature_ctl(s, fc);
    int next;
    if (s.policy == ALB_POLICY_LEARNED && a.mlp && a.mlp[kMlpParams] != 0.0f) {
        float f[kMlpIn];
        level_features(fc, f);
        next = mlp_select_warp(a.mlp, f);
    } else {
        next = rule_dir(fc);
    }
    const int i = threadIdx.x;
    unsigned long long tm = 0;
    if (next != ALB_DIR_TOPDOWN && s.dir == ALB_DIR_TOPDOWN && !s.done && s.push_budget > 0)
        tm = ms_pushed_roots(a.smp->deg[i], a.smp->deg[i + 32], (unsigned long long)s.push_budget,
                             s.used, room);
    a.smp->deg[i] = a.smp->deg[i + 32] = 0;
    if (i == 0) {
        s.tmask = tm;
        s.pushed_roots += __popcll(tm);
        ms_set_next(a, s, next);
    }
    __syncwarp();
    for (int w = threadIdx.x; w < kCtlWords; w += 32)
        reinterpret_cast<unsigned long long *>(a.ctl)[w] =
            reinterpret_cast<const unsigned long long *>(&s)[w];
}

// After a flush of the snapshot store: slot 0 now holds level `base`.
__global__ void k_ms_set_base(MsArgs a, int base) {
    a.ctl->base = base;
    a.ctl->need_flush = 0;
}

// Writes the levels held by snapshot slots [0, nslots) (levels base ..) into
// the vertex-major n x 64 output. Half a warp per position: lane q of the
// half owns roots 4q .. 4q+3 and writes them as one 16-byte store, so a
// position's 256-byte output row is one contiguous burst. The slots are read
// once per position (lane q loads slot q and q+16) and shared with shuffles.
// Each warp takes kExpandUnroll pairs of positions per step and issues all
// their loads before the first shuffle, to keep enough bytes in flight.
// A root's bit is set in exactly one slot, so the slots can be scanned in any
// order. kFirst: the first flush writes every entry (-1 where unreached and
// for root columns >= nroots); later flushes write only the levels found.
constexpr int kExpandUnroll = 4;

template <bool kFirst, bool kVec>
__global__ void k_ms_expand(MsArgs a, int nslots, int base, int nroots, int32_t *out) {
    const int lane = threadIdx.x & 31, q = lane & 15;
    const int64_t total = a.n * 16;
    const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int first_cnt = min(16, nslots);
    // the loop bound is warp-uniform so that every lane reaches the shuffles
    for (int64_t t0 = gw * 32 * kExpandUnroll; t0 < total; t0 += nw * 32 * kExpandUnroll) {
        uint64_t mine[kExpandUnroll];
        int32_t vid[kExpandUnroll];
#pragma unroll
        for (int u = 0; u < kExpandUnroll; u++) {
            const int64_t t = t0 + u * 32 + lane;
            const bool ok = t < total;
            const int64_t p = ok ? t >> 4 : 0;
            mine[u] = (ok && q < nslots) ? __ldcs(a.S + (int64_t)q * a.npad + p) : 0ull;
            vid[u] = ok ? __ldg(a.perm + p) : 0;
        }
#pragma unroll
        for (int u = 0; u < kExpandUnroll; u++) {
            const int64_t t = t0 + u * 32 + lane;
            const bool ok = t < total;
            const int64_t p = ok ? t >> 4 : 0;
            int32_t l[4] = {-1, -1, -1, -1};
            for (int k = 0; k < first_cnt; k++) {
                const uint64_t sv = __shfl_sync(kFull, mine[u], k, 16);
                const uint32_t b = (uint32_t)(sv >> (4 * q)) & 0xFu;
                if (b) {
#pragma unroll
                    for (int r = 0; r < 4; r++)
                        if ((b >> r) & 1u) l[r] = base + k;
                }
            }
            for (int c0 = 16; c0 < nslots; c0 += 16) {  // more than 16 levels held
                const int js = c0 + q;
                const uint64_t m2 =
                    (ok && js < nslots) ? __ldcs(a.S + (int64_t)js * a.npad + p) : 0ull;
                const int cnt = min(16, nslots - c0);
                for (int k = 0; k < cnt; k++) {
                    const uint64_t sv = __shfl_sync(kFull, m2, k, 16);
                    const uint32_t b = (uint32_t)(sv >> (4 * q)) & 0xFu;
                    if (b) {
#pragma unroll
                        for (int r = 0; r < 4; r++)
                            if ((b >> r) & 1u) l[r] = base + c0 + k;
                    }
                }
            }
            if (!ok) continue;
#pragma unroll
            for (int r = 0; r < 4; r++)
                if (4 * q + r >= nroots) l[r] = -1;
            int32_t *o = out + (int64_t)vid[u] * 64 + 4 * q;
            if (kFirst && kVec) {
                __stcs(reinterpret_cast<int4 *>(o), make_int4(l[0], l[1], l[2], l[3]));
            } else {
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if (kFirst || l[r] >= 0) o[r] = l[r];
            }
        }
    }
}

// The same output, one CTA per aligned tile of kExpandTile rows. The sort
// permutes rows only inside sigma windows, so when sigma divides the tile the
// positions of the tile's original ids are the tile's own positions. The CTA
// first reads the tile's slot words (coalesced) and folds them, per
// position, into five words: R = OR of all slots (roots that reached it) and
// M_t = OR of the slots whose index has bit t set, so that root i's slot
// index is the number whose bit t is bit i of M_t. It then writes the tile's
// 256-byte output rows in original-id order, a sequential stream: lane q of a
// half warp turns nibble q of the five words into the levels of roots
// 4q .. 4q+3 with a few integer operations, independent of the slot count.
// First flush, 16-byte aligned output, at most kExpandMaxSlots slots.
// parts CTAs share a tile, each folding it and writing its part of the rows:
// R-MAT scale 16 has but 64 tiles. (Reading a slot's words only where its
// nonzero bitmap has any, and CTAs that take one tile after another, each cost
// 40 to 80 us of 870 at scale 24: a round trip more before a tile's loads, and
// fewer tiles in flight.)
// nslots < 0: launched behind the search, which says how many levels it had;
// nothing is written where it has not ended or had too many.
constexpr int kExpandTile = 1024;
constexpr int kExpandMaxSlots = 16;
constexpr int kExpandThreads = 512;
__host__ __device__ inline bool ms_output_ready(const MsCtl &c) {
    return c.done && !c.err && c.base == 0 && c.level <= kExpandMaxSlots;
}
constexpr size_t kExpandSmem = (5 * sizeof(uint64_t) + sizeof(int32_t)) * kExpandTile;

// Bit k of the nibble n moves to bit 8k (copies shifted by 0, 7, 14, 21 do
// not overlap for n < 16, so the product has no carries).
__device__ __forceinline__ uint32_t nibble_to_bytes(uint32_t n) {
    return (n * 0x00204081u) & 0x01010101u;
}

__global__ void __launch_bounds__(kExpandThreads) k_ms_expand_tile(MsArgs a, int nslots, int base,
                                                                   int nroots, int parts,
                                                                   int32_t *h_err, int32_t *out) {
    extern __shared__ uint64_t s_fold[];  // 5 x kExpandTile words, then kExpandTile positions
    int32_t *s_pos = reinterpret_cast<int32_t *>(s_fold + 5 * kExpandTile);
    if (nslots < 0) {
        if (!ms_output_ready(*a.ctl)) return;
        nslots = a.ctl->level;
        base = 0;
    }
    const int part = (int)(blockIdx.x % (unsigned)parts);
    const int64_t t0 = (int64_t)(blockIdx.x / (unsigned)parts) * kExpandTile;
    const int rows = (int)min((int64_t)kExpandTile, a.n - t0);
    for (int r = threadIdx.x; r < kExpandTile; r += blockDim.x) {
        uint64_t m0 = 0, m1 = 0, m2 = 0, m3 = 0, all = 0;
        if (r < rows) {
#pragma unroll 4
            for (int jj = 0; jj < nslots; jj++) {
                const uint64_t w = __ldcs(a.S + (int64_t)jj * a.npad + t0 + r);
                all |= w;
                if (jj & 1) m0 |= w;
                if (jj & 2) m1 |= w;
                if (jj & 4) m2 |= w;
                if (jj & 8) m3 |= w;
            }
            s_pos[r] = (int32_t)((int64_t)__ldg(a.inv + t0 + r) - t0);  // position in the tile
        }
        s_fold[r] = all;
        s_fold[kExpandTile + r] = m0;
        s_fold[2 * kExpandTile + r] = m1;
        s_fold[3 * kExpandTile + r] = m2;
        s_fold[4 * kExpandTile + r] = m3;
    }
    __syncthreads();
    const int q = threadIdx.x & 15;
    const int sh = 4 * q;
    const int r1 = rows * (part + 1) / parts;
    for (int r = rows * part / parts + (threadIdx.x >> 4); r < r1; r += blockDim.x >> 4) {
        const int64_t v = t0 + r;  // original id
        const int pl = s_pos[r];
        if ((unsigned)pl >= (unsigned)rows) {  // not a window permutation: refuse, loudly
            a.ctl->err = ALB_ERR_DEVICE;
            *h_err = ALB_ERR_DEVICE;
            continue;
        }
        const uint32_t reach =
            nibble_to_bytes((uint32_t)(s_fold[pl] >> sh) & 0xFu);
        const uint32_t idx =
            nibble_to_bytes((uint32_t)(s_fold[kExpandTile + pl] >> sh) & 0xFu) |
            (nibble_to_bytes((uint32_t)(s_fold[2 * kExpandTile + pl] >> sh) & 0xFu) << 1) |
            (nibble_to_bytes((uint32_t)(s_fold[3 * kExpandTile + pl] >> sh) & 0xFu) << 2) |
            (nibble_to_bytes((uint32_t)(s_fold[4 * kExpandTile + pl] >> sh) & 0xFu) << 3);
        int32_t l[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool hit = ((reach >> (8 * k)) & 1u) && (sh + k < nroots);
            l[k] = hit ? base + (int32_t)((idx >> (8 * k)) & 0xFu) : -1;
        }
        __stcs(reinterpret_cast<int4 *>(out + v * 64 + 4 * q), make_int4(l[0], l[1], l[2], l[3]));
    }
}

struct MsScratch {
    bool ready = false;
    int32_t K = 0;
    uint64_t *V = nullptr, *S = nullptr;
    uint32_t *D = nullptr, *A = nullptr;
    int32_t *q0 = nullptr, *q1 = nullptr, *big = nullptr;
    int64_t *big_base = nullptr;
    int32_t *pbig = nullptr;
    int64_t *pbig_base = nullptr;
    MsCtl *ctl = nullptr, *h_ctl = nullptr;
    int32_t *out = nullptr;
    long long *gtrace = nullptr;  // the cooperative kernel's level records
    MsSlots *slots = nullptr;     // its counters; clean: as a finished launch leaves them
    bool slots_clean = false;
};

}  // namespace alb

namespace alb {

static MsScratch &ms_scratch(alb_graph *g) {
    if (!g->ms) g->ms = new MsScratch();
    return *(MsScratch *)g->ms;
}

void ms_scratch_free(alb_graph *g) {
    if (!g->ms) return;
    MsScratch &m = *(MsScratch *)g->ms;
    dfree(m.V);
    dfree(m.S);
    dfree(m.D);
    dfree(m.A);
    dfree(m.q0);
    dfree(m.q1);
    dfree(m.big);
    dfree(m.big_base);
    dfree(m.pbig);
    dfree(m.pbig_base);
    dfree(m.ctl);
    dfree(m.out);
    dfree(m.gtrace);
    if (m.h_ctl) cudaFreeHost(m.h_ctl);
    dfree(m.slots);
    delete (MsScratch *)g->ms;
    g->ms = nullptr;
}

namespace {

// Whether the first flush into out takes whole tiles.
bool expand_tiles(const MsArgs &a, const int32_t *out) {
    return ((uintptr_t)out & 15) == 0 && a.sigma >= 1 && a.sigma <= kExpandTile &&
           kExpandTile % a.sigma == 0;
}

// h_err: page-locked, told of a row outside its tile.
alb_status launch_expand_tiles(const MsArgs &a, int nslots, int base, int nroots, int32_t *h_err,
                               int32_t *out, int num_sms, cudaStream_t st) {
    ALB_CK(cudaFuncSetAttribute(k_ms_expand_tile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kExpandSmem));
    const int64_t tiles = (a.n + kExpandTile - 1) / kExpandTile;
    const int parts = (int)std::max<int64_t>(1, std::min<int64_t>(4, 2 * num_sms / tiles));
    k_ms_expand_tile<<<(unsigned)(tiles * parts), kExpandThreads, kExpandSmem, st>>>(
        a, nslots, base, nroots, parts, h_err, out);
    ALB_CK(cudaGetLastError());
    return ALB_OK;
}

alb_status launch_expand(const MsArgs &a, int nslots, int base, bool first, int nroots,
                         int32_t *h_err, int32_t *out, int num_sms, cudaStream_t st) {
    const bool vec = ((uintptr_t)out & 15) == 0;
    auto grid = [&](const void *f) {
        const int per = resident_blocks(f, 256);
        return (unsigned)(num_sms * (per > 0 ? per : 8));
    };
    if (first && nslots <= kExpandMaxSlots && expand_tiles(a, out))
        return launch_expand_tiles(a, nslots, base, nroots, h_err, out, num_sms, st);
    if (first && vec)
        k_ms_expand<true, true><<<grid((const void *)k_ms_expand<true, true>), 256, 0, st>>>(
            a, nslots, base, nroots, out);
    else if (first)
        k_ms_expand<true, false><<<grid((const void *)k_ms_expand<true, false>), 256, 0, st>>>(
            a, nslots, base, nroots, out);
    else
        k_ms_expand<false, false><<<grid((const void *)k_ms_expand<false, false>), 256, 0, st>>>(
            a, nslots, base, nroots, out);
    ALB_CK(cudaGetLastError());
    return ALB_OK;
}

alb_status ms_alloc(alb_graph *g, MsScratch &m) {
    if (m.ready) return ALB_OK;
    const Sell &s = g->sell;
    const int64_t npad = s.nwords * 32;
    m.K = 32;
    ALB_TRY(dmalloc((void **)&m.V, sizeof(uint64_t) * npad, "msbfs visited"));
    ALB_TRY(dmalloc((void **)&m.S, sizeof(uint64_t) * npad * m.K, "msbfs frontier snapshots"));
    ALB_TRY(dmalloc((void **)&m.D, sizeof(uint32_t) * s.nwords, "msbfs done bitmap"));
    ALB_TRY(dmalloc((void **)&m.A, sizeof(uint32_t) * 2 * s.nwords, "msbfs frontier-nonzero bitmaps"));
    ALB_TRY(dmalloc((void **)&m.q0, sizeof(int32_t) * npad, "msbfs queue"));
    ALB_TRY(dmalloc((void **)&m.q1, sizeof(int32_t) * npad, "msbfs queue"));
    ALB_TRY(dmalloc((void **)&m.big, sizeof(int32_t) * npad, "msbfs long-row list"));
    ALB_TRY(dmalloc((void **)&m.big_base, sizeof(int64_t) * npad, "msbfs long-row chunk bases"));
    // (rows of more than kBigRow edges: there cannot be more)
    const size_t nbig = (size_t)std::min<int64_t>(npad, s.m_out / kBigRow + 1);
    ALB_TRY(dmalloc((void **)&m.pbig, sizeof(int32_t) * nbig, "msbfs pushed rows"));
    ALB_TRY(dmalloc((void **)&m.pbig_base, sizeof(int64_t) * nbig, "msbfs pushed rows' chunk bases"));
    ALB_TRY(dmalloc((void **)&m.ctl, sizeof(MsCtl) + sizeof(MsSample), "msbfs control"));
    ALB_TRY(dmalloc((void **)&m.gtrace, sizeof(long long) * kGTraceCap * kGTraceW,
                    "msbfs level records"));
    ALB_TRY(dmalloc((void **)&m.slots, sizeof(MsSlots), "msbfs counters"));
    ALB_CK(cudaMallocHost((void **)&m.h_ctl, sizeof(MsCtl)));
    m.ready = true;
    return ALB_OK;
}

MsArgs ms_args(alb_graph *g, MsScratch &m) {
    const Sell &s = g->sell;
    MsArgs a;
    std::memset(&a, 0, sizeof(a));
    a.n = g->n;
    a.nwords = s.nwords;
    a.npad = s.nwords * 32;
    a.C = s.C;
    a.log2C = s.log2C;
    a.K = m.K;
    a.sigma = s.sigma;
    a.wpw = s.sigma >= 32 && s.sigma % 32 == 0 ? (unsigned)s.sigma / 32 : 1u;
    a.nwin = (unsigned)((s.nwords + a.wpw - 1) / a.wpw);
    a.perm = s.perm;
    a.inv = s.inv;
    a.ideg = s.ideg;
    a.odeg = s.odeg;
    a.width = s.width;
    a.vinit = s.vinit;
    a.slice_off = s.slice_off;
    a.col4 = (const int4 *)s.col;
    a.prow = s.prow;
    a.pcol = s.pcol;
    a.nlong = s.nlong;
    a.long_row = s.long_row;
    a.any_big = s.max_deg > kBigRow;
    a.lrow = s.lrow;
    a.lptr = s.lptr;
    a.lcol = s.lcol;
    a.V = m.V;
    a.S = m.S;
    a.D = m.D;
    a.A = m.A;
    a.q0 = m.q0;
    a.q1 = m.q1;
    a.big = m.big;
    a.big_base = m.big_base;
    a.pbig = m.pbig;
    a.pbig_base = m.pbig_base;
    a.ctl = m.ctl;
    a.smp = reinterpret_cast<MsSample *>(m.ctl + 1);
    a.gtrace = m.gtrace;
    return a;
}

}  // namespace

extern const float *selector_device_params(int which);

// Device copies of the state one level mutates (restored between variants).
struct MsSnapshot {
    uint64_t *V = nullptr;
    uint32_t *D = nullptr;
    MsCtl *ctl = nullptr;
    ~MsSnapshot() {
        dfree(V);
        dfree(D);
        dfree(ctl);
    }
};

alb_status ms_snapshot(const MsArgs &a, MsSnapshot &s, cudaStream_t st, bool restore) {
    auto cp = [&](void *dst, const void *src, size_t bytes) {
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st);
    };
    cudaError_t e = restore ? cp(a.V, s.V, 8 * a.npad) : cp(s.V, a.V, 8 * a.npad);
    if (e == cudaSuccess) e = restore ? cp(a.D, s.D, 4 * a.nwords) : cp(s.D, a.D, 4 * a.nwords);
    const size_t cb = sizeof(MsCtl) + sizeof(MsSample);
    if (e == cudaSuccess) e = restore ? cp(a.ctl, s.ctl, cb) : cp(s.ctl, a.ctl, cb);
    if (e != cudaSuccess) return fail(ALB_ERR_CUDA, "msbfs snapshot: %s", cudaGetErrorString(e));
    return ALB_OK;
}

alb_status msbfs_impl(alb_graph *g, const int32_t *roots, int32_t nroots, const alb_bfs_opts &o,
                      int32_t *d_levels, alb_stats *st, std::vector<alb_level_rec> *trace,
                      std::vector<alb_level_profile> *prof = nullptr) {
    MsScratch &m = ms_scratch(g);
    PhaseLog ph("msbfs64_device");
    ALB_TRY(ms_alloc(g, m));
    ph.mark("scratch", g->stream);
    MsArgs a = ms_args(g, m);
    a.mlp = selector_device_params(1);
    const Sell &s = g->sell;
    cudaStream_t stream = g->stream;
    const int block = o.block;
    const unsigned wide = (unsigned)(g->num_sms * std::max(1, 2048 / block));
    // the cooperative kernel; a run of it traced under ALB_LOOP_GRAPH records
    // its levels on the device, so that the trace times the benchmarked form
    // itself (one under ALB_LOOP_PERSISTENT has the active words too, which only
    // the host-driven loop records)
    const bool coop = o.loop != ALB_LOOP_HOST && !prof && !(trace && o.loop == ALB_LOOP_PERSISTENT);
    MsInit in;
    std::memset(&in, 0, sizeof(in));
    for (int i = 0; i < nroots; i++) in.roots[i] = roots[i];
    in.nroots = nroots;
    in.policy = o.policy;
    in.alpha = o.alpha;
    in.beta = o.beta;
    in.mean_deg = g->n > 0 ? (float)((double)s.m_in / (double)g->n) : 0.f;
    in.skew = skew_of(s, g->n);
    in.n_live = g->n - s.zero_in;
    in.m_in = s.m_in;
    in.active0 = s.active0;
    in.push_budget = s.m_in / kPushDiv;
    {
        // words per run of the pull: about three runs per resident warp, up to
        // 32 (RMAT s22: 8 beats 32 by 7 %; s24: 32 beats 8 by 2 %, where longer
        // runs save counter round trips and still leave every warp busy). The
        // cooperative kernel, whose teams take the widest words first, goes
        // down to 1; the host loop's kernels to 8: with fewer words a run a
        // window's wide first word comes up late (s19: a level 205 -> 295 us).
        const int per = resident_blocks((const void *)k_ms_bu<true, true, false>, kMsBuBlock);
        const int64_t warps = coop ? (int64_t)32 * g->num_sms
                                   : (int64_t)std::max(per, 1) * (kMsBuBlock / 32) * g->num_sms;
        in.grab = (int32_t)std::max<int64_t>(coop ? 1 : kGrabWords,
                                             std::min<int64_t>(32, s.nwords / (3 * warps)));
    }
    if (const char *e = std::getenv("ALB_MS_PUSH_DIV")) {  // tuning: 0 turns the push off
        const long long dv = std::atoll(e);
        in.push_budget = dv > 0 ? s.m_in / dv : 0;
    }
    const int32_t level_cap = (int32_t)std::min<int64_t>(g->n + 1, INT32_MAX - 1);
    in.level_cap = level_cap;
    const bool gtrace = trace && coop;
    in.gtrace = gtrace ? 1 : 0;
    in.unused = nroots >= 64 ? 0ull : ~((1ull << nroots) - 1);
    ALB_CK(cudaEventRecord(g->ev0, stream));
    int64_t launches = 0;
    MsCtl *h = m.h_ctl;
    int base = 0;      // level held by slot 0
    bool first_flush = true;
    bool written = false;  // the output was launched behind the search
    // flush of the snapshot store: write out levels [base, base + K - 1) and
    // restart the store from the current frontier
    auto flush = [&]() -> alb_status {
        if (d_levels) {
            ALB_TRY(launch_expand(a, m.K - 1, base, first_flush, nroots, &h->err, d_levels,
                                  g->num_sms, stream));
            launches++;
        }
        first_flush = false;
        ALB_CK(cudaMemcpyAsync(a.S, a.S + (int64_t)(m.K - 1) * a.npad, sizeof(uint64_t) * a.npad,
                               cudaMemcpyDeviceToDevice, stream));
        base += m.K - 1;
        k_ms_set_base<<<1, 1, 0, stream>>>(a, base);
        launches++;
        return ALB_OK;
    };
    if (coop) {
        // the host only steps in for flushes
        const DeviceWaits dw = device_waits(kMsBarrierNs, 0);
        MsGridArgs x{m.slots, h, 0, dw.barrier_ns, dw.withhold_level, dw.withhold_block};
        while (true) {
            if (!m.slots_clean) ALB_CK(cudaMemsetAsync(m.slots, 0, sizeof(MsSlots), stream));
            m.slots_clean = false;
            h->done = h->need_flush = 0;
            h->err = ALB_OK;
            ALB_TRY(ms_grid_launch(g, a, in, x, stream));
            launches++;
            // the output right behind it, for the usual search of few levels
            // (its launch then costs no trip to the host between the two)
            const bool behind = d_levels && !x.resume && expand_tiles(a, d_levels);
            if (behind) {
                ALB_TRY(launch_expand_tiles(a, -1, 0, nroots, &h->err, d_levels, g->num_sms, stream));
                ALB_CK(cudaEventRecord(g->ev1, stream));
                launches++;
            }
            ALB_CK(cudaStreamSynchronize(stream));
            if (!h->done && !h->need_flush) {  // a wait gave up, perhaps before the result
                ALB_CK(cudaMemcpy(&h->err, &a.ctl->err, sizeof(int32_t), cudaMemcpyDeviceToHost));
                return fail(h->err ? h->err : ALB_ERR_DEVICE, "msbfs: the kernel gave up");
            }
            m.slots_clean = true;
            if (h->err) return fail(h->err, "msbfs: the device refused the traversal");
            written = behind && ms_output_ready(*h);
            if (h->done) break;
            ALB_TRY(flush());
            x.resume = 1;
        }
        if (gtrace) {
            const int nl = std::min<int>(h->level, kGTraceCap);
            std::vector<long long> rec((size_t)nl * kGTraceW);
            if (nl > 0)
                ALB_CK(cudaMemcpyAsync(rec.data(), m.gtrace, sizeof(long long) * rec.size(),
                                       cudaMemcpyDeviceToHost, stream));
            ALB_CK(cudaStreamSynchronize(stream));
            trace->clear();
            for (int L = 0; L < nl; L++) {
                const long long *r = rec.data() + (size_t)L * kGTraceW;
                alb_level_rec t;
                std::memset(&t, 0, sizeof(t));
                t.level = L;
                t.dir = (int32_t)r[3];
                t.nf = r[4];
                t.mf = r[5];
                t.nu = r[6];
                t.mu = r[7];
                t.t_ns = r[0];
                t.step_us = (float)((r[1] - r[0]) / 1e3);
                t.bytes = r[2];
                trace->push_back(t);
            }
        }
    } else {
        k_ms_init<<<wide, 256, 0, stream>>>(a, in.unused);
        k_ms_roots<<<1, 64, 0, stream>>>(a, in);  // also decides level 0's direction
        ALB_CK(cudaGetLastError());
        launches += 2;
        ALB_CK(cudaMemcpyAsync(h, a.ctl, sizeof(MsCtl), cudaMemcpyDeviceToHost, stream));
        ALB_CK(cudaStreamSynchronize(stream));
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        if (trace) trace->clear();
        if (trace || prof) {
            ALB_CK(cudaEventCreate(&e0));
            ALB_CK(cudaEventCreate(&e1));
        }
        MsSnapshot snap;
        if (prof) {
            prof->clear();
            ALB_TRY(dmalloc((void **)&snap.V, 8 * a.npad, "msbfs snapshot"));
            ALB_TRY(dmalloc((void **)&snap.D, 4 * a.nwords, "msbfs snapshot"));
            ALB_TRY(dmalloc((void **)&snap.ctl, sizeof(MsCtl) + sizeof(MsSample), "msbfs snapshot"));
        }
        while (!h->done && h->level < level_cap) {
            const int L = h->level;
            int j = L - base;
            if (j + 1 >= m.K) {
                ALB_TRY(flush());
                j = 0;
            }
            int dir = h->dir;
            alb_level_rec rec;
            std::memset(&rec, 0, sizeof(rec));
            rec.dir = dir;
            rec.level = L;
            rec.nf = h->nf;
            rec.mf = h->mf;
            rec.nu = h->nu;
            rec.mu = h->mu;
            rec.active_slices = h->active_words;
            rec.step_us = -1.f;
            const bool q_valid = h->q_valid != 0;
            // nonzero-bitmap filter when under 1/8 of all entries point into the frontier
            const int filt = (h->mf < s.m_in / 8) ? 1 : 0;
            // the first bottom-up level after a top-down one pulls two groups at a time
            const bool two_groups = h->prev_dir == ALB_DIR_TOPDOWN;
            auto launch_step = [&](int d) -> alb_status {
                if (d == ALB_DIR_TOPDOWN) {
                    if (!q_valid) {
                        k_ms_compact<<<wide, block, 0, stream>>>(a, j);
                        launches++;
                    }
                    k_ms_zero_next<<<wide, block, 0, stream>>>(a, j);
                    launch_resident(k_ms_td<false>, block, g->num_sms, stream, a, j);
                    launch_resident(k_ms_td_big<false>, block, g->num_sms, stream, a, j);
                    launch_resident(k_ms_td_finish, block, g->num_sms, stream, a, j);
                    launches += 4;
                } else if (d == ALB_DIR_BOTTOMUP) {
                    if (filt)
                        launch_resident(k_ms_bu<true, true, true>, kMsBuBlock, g->num_sms, stream, a, j);
                    else if (two_groups)
                        launch_resident(k_ms_bu<true, true, false, true>, kMsBuBlock, g->num_sms, stream, a, j);
                    else
                        launch_resident(k_ms_bu<true, true, false>, kMsBuBlock, g->num_sms, stream, a, j);
                    launch_resident(k_ms_bu_long<true>, block, g->num_sms, stream, a, j, filt);
                    launch_resident(k_ms_bu_long_tail<true>, block, g->num_sms, stream, a, j, filt);
                    launch_resident(k_ms_bu_long_fin, block, g->num_sms, stream, a, j);
                    launches += 4;
                } else {
                    if (filt)
                        launch_resident(k_ms_bu<false, false, true>, kMsBuBlock, g->num_sms, stream, a, j);
                    else
                        launch_resident(k_ms_bu<false, false, false>, kMsBuBlock, g->num_sms, stream, a, j);
                    launch_resident(k_ms_bu_long<false>, block, g->num_sms, stream, a, j, filt);
                    launch_resident(k_ms_bu_long_tail<false>, block, g->num_sms, stream, a, j, filt);
                    launch_resident(k_ms_bu_long_fin, block, g->num_sms, stream, a, j);
                    launches += 4;
                }
                if (d != ALB_DIR_TOPDOWN && h->prev_dir == ALB_DIR_TOPDOWN) {  // push of the roots in tmask
                    k_ms_tq<<<wide, block, 0, stream>>>(a, j);
                    launch_resident(k_ms_td<true>, block, g->num_sms, stream, a, j);
                    launch_resident(k_ms_td_big<true>, block, g->num_sms, stream, a, j);
                    launches += 3;
                }
                launch_resident(k_ms_sample, kSampleBlock, g->num_sms, stream, a, j, d);
                launches++;
                return ALB_OK;
            };
            if (prof) {
                // time every variant from the same state, then take the fastest
                alb_level_profile pr;
                std::memset(&pr, 0, sizeof(pr));
                ALB_TRY(ms_snapshot(a, snap, stream, false));
                for (int v = 0; v < 3; v++) {
                    if (v) ALB_TRY(ms_snapshot(a, snap, stream, true));
                    ALB_CK(cudaEventRecord(e0, stream));
                    ALB_TRY(launch_step(v));
                    ALB_CK(cudaEventRecord(e1, stream));
                    ALB_CK(cudaStreamSynchronize(stream));
                    float ms = 0;
                    ALB_CK(cudaEventElapsedTime(&ms, e0, e1));
                    pr.us[v] = ms * 1000.f;
                }
                int best = 0;
                for (int v = 1; v < 3; v++)
                    if (pr.us[v] < pr.us[best]) best = v;
                ALB_TRY(ms_snapshot(a, snap, stream, true));
                dir = best;
                pr.best = best;
                pr.rec = rec;
                pr.rec.dir = best;
                pr.rec.step_us = pr.us[best];
                BfsCtl fc;
                std::memset(&fc, 0, sizeof(fc));
                fc.level = L;
                fc.n = h->n;
                fc.nwords = h->nwords;
                fc.nf = h->nf;
                fc.mf = h->mf;
                fc.nu = h->nu;
                fc.mu = h->mu;
                fc.active_words = h->active_words;
                fc.feat_mean_deg = h->feat_mean_deg;
                fc.feat_skew = h->feat_skew;
                level_features(fc, pr.feat);
                prof->push_back(pr);
            }
            if (e0) cudaEventRecord(e0, stream);
            ALB_TRY(launch_step(dir));
            if (e1) cudaEventRecord(e1, stream);
            k_ms_end<<<1, 32, 0, stream>>>(a, dir);
            launches++;
            ALB_CK(cudaGetLastError());
            ALB_CK(cudaMemcpyAsync(h, a.ctl, sizeof(MsCtl), cudaMemcpyDeviceToHost, stream));
            ALB_CK(cudaStreamSynchronize(stream));
            if (trace) {
                float ms = 0;
                cudaEventElapsedTime(&ms, e0, e1);
                rec.dir = dir;
                rec.step_us = ms * 1000.f;
                const int k = (L + 1) % 3;
                rec.bytes = dir == ALB_DIR_TOPDOWN
                                ? (int64_t)(20 * rec.nf + 16 * rec.mf + 16 * (int64_t)h->acc_n[k])
                                : (int64_t)h->acc_bytes[k] + 8 * a.npad + 8 * a.nwords;
                trace->push_back(rec);
            }
        }
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
    }
    if (!h->done) return fail(ALB_ERR_DEVICE, "msbfs: level cap reached");
    if (!written) {
        if (d_levels) {
            const int nslots = h->level - base;  // slots 0 .. level-base-1 hold levels
            ALB_TRY(launch_expand(a, std::min(nslots, m.K), base, first_flush, nroots, &h->err,
                                  d_levels, g->num_sms, stream));
            launches++;
        }
        ALB_CK(cudaEventRecord(g->ev1, stream));
        ALB_CK(cudaStreamSynchronize(stream));
    }
    if (h->err) return fail(h->err, "msbfs: level output saw a position outside its tile");
    float ms = 0;
    ALB_CK(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
    if (st) {
        st->num_levels = h->level;
        st->levels_topdown = h->levels_td;
        st->levels_bottomup = h->levels_bu;
        st->pushed_roots = h->pushed_roots;
        st->reached = h->pairs;
        st->edges = h->edges;
        st->ms = ms;
        st->kernels = launches;
    }
    return ALB_OK;
}

}  // namespace alb

using namespace alb;

extern "C" {

alb_status alb_msbfs64_device(alb_graph *g, const int32_t *roots, int32_t nroots,
                              const alb_bfs_opts *o, int32_t *d_levels, alb_stats *st) {
    if (!g || !roots || nroots < 1 || nroots > 64)
        return fail(ALB_ERR_INVALID, "alb_msbfs64: need a graph and 1..64 roots");
    if (!g->sell.built) return fail(ALB_ERR_STATE, "alb_msbfs64: call alb_sell_build first");
    for (int i = 0; i < nroots; i++)
        if (roots[i] < 0 || roots[i] >= g->n)
            return fail(ALB_ERR_INVALID, "alb_msbfs64: root %d outside [0, %lld)", roots[i],
                        (long long)g->n);
    alb_bfs_opts oo;
    alb_bfs_opts_default(&oo);
    if (o) oo = *o;
    if (oo.policy < ALB_POLICY_BEAMER || oo.policy > ALB_POLICY_BOTTOMUP_NOBYPASS)
        return fail(ALB_ERR_INVALID, "alb_msbfs64: unknown policy %d", oo.policy);
    if (!(oo.block == 128 || oo.block == 256 || oo.block == 512 || oo.block == 1024))
        return fail(ALB_ERR_UNSUPPORTED, "alb_msbfs64: block must be 128, 256, 512 or 1024");
    ALB_CK(cudaSetDevice(g->device));
    std::vector<alb_level_rec> tr;
    alb_status rc;
    try {
        rc = msbfs_impl(g, roots, nroots, oo, d_levels, st, oo.trace ? &tr : nullptr);
    } catch (const std::bad_alloc &) {
        rc = fail(ALB_ERR_OOM, "alb_msbfs64: host allocation failed");
    }
    if (rc == ALB_OK && oo.trace) {
        g->last_trace = tr;
        g->last_trace_valid = true;
    }
    return rc;
}

alb_status alb_msbfs64_profile(alb_graph *g, const int32_t *roots, int32_t nroots,
                               const alb_bfs_opts *o, int32_t cap, alb_level_profile *out,
                               int32_t *count) {
    if (!g || !roots || nroots < 1 || nroots > 64 || !count || (cap > 0 && !out))
        return fail(ALB_ERR_INVALID, "alb_msbfs64_profile: bad arguments");
    if (!g->sell.built) return fail(ALB_ERR_STATE, "alb_msbfs64_profile: call alb_sell_build first");
    for (int i = 0; i < nroots; i++)
        if (roots[i] < 0 || roots[i] >= g->n)
            return fail(ALB_ERR_INVALID, "alb_msbfs64_profile: root outside the graph");
    alb_bfs_opts oo;
    alb_bfs_opts_default(&oo);
    if (o) oo = *o;
    ALB_CK(cudaSetDevice(g->device));
    std::vector<alb_level_profile> pr;
    alb_status rc;
    try {
        rc = msbfs_impl(g, roots, nroots, oo, nullptr, nullptr, nullptr, &pr);
    } catch (const std::bad_alloc &) {
        rc = fail(ALB_ERR_OOM, "alb_msbfs64_profile: host allocation failed");
    }
    if (rc != ALB_OK) return rc;
    *count = (int32_t)pr.size();
    for (int32_t i = 0; i < cap && i < (int32_t)pr.size(); i++) out[i] = pr[i];
    return ALB_OK;
}

alb_status alb_msbfs64(alb_graph *g, const int32_t *roots, int32_t nroots, const alb_bfs_opts *o,
                       int32_t *levels, alb_stats *st) {
    if (!g) return fail(ALB_ERR_INVALID, "alb_msbfs64: graph is NULL");
    ALB_CK(cudaSetDevice(g->device));
    PhaseLog ph("msbfs64");
    MsScratch &m = ms_scratch(g);
    // page-locked host levels are written by the expansion itself, across
    // the host link (as fast as a copy, measured: 193 GB/s either way), with
    // no device staging buffer and no separate copy; other host memory goes
    // through a device buffer and one copy
    int32_t *direct = nullptr;
    if (levels) {
        cudaPointerAttributes pa;
        if (cudaPointerGetAttributes(&pa, levels) == cudaSuccess && pa.type == cudaMemoryTypeHost &&
            pa.devicePointer)
            direct = static_cast<int32_t *>(pa.devicePointer);
        cudaGetLastError();
    }
    if (levels && !direct && !m.out) {
        ALB_TRY(dmalloc((void **)&m.out, sizeof(int32_t) * (size_t)g->n * 64, "msbfs levels"));
    }
    ph.mark("out_alloc", g->stream);
    ALB_TRY(alb_msbfs64_device(g, roots, nroots, o, direct ? direct : levels ? m.out : nullptr, st));
    ph.mark("traversal", g->stream);
    if (direct) {
        ALB_CK(cudaStreamSynchronize(g->stream));
    } else if (levels) {
        ALB_CK(cudaMemcpyAsync(levels, m.out, sizeof(int32_t) * (size_t)g->n * 64,
                               cudaMemcpyDeviceToHost, g->stream));
        ALB_CK(cudaStreamSynchronize(g->stream));
    }
    ph.mark("copy_out", g->stream);
    return ALB_OK;
}

}  // extern "C"

