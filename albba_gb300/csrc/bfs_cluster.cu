// Single-root BFS of a small graph in one launch of one thread-block cluster.
//
// The level loops of bfs.cu fill the GPU with every kernel; a graph of a few
// thousand vertices then spends its time on launches (20 to 25 us a level in
// the CUDA graph) and on grid barriers and round trips to L2. Here the whole
// call -- initial state, every level, the outputs in original ids -- is one
// kernel of up to 16 CTAs of 1024 threads on neighbouring SMs, which meet at
// the cluster's hardware barrier. Each CTA keeps the three bitmaps (frontier,
// next frontier, visited; a bit per position) whole in its shared memory, so
// frontier and visited tests never leave the SM, and owns a run of bitmap
// words: it pulls their rows at bottom-up levels and merges the other CTAs'
// pushes into them at top-down ones, writing each finished word into every
// CTA's copy through distributed shared memory. Levels, parents and their
// rules, directions and counters are those of bfs.cu.
//
// Bound: latency. A level costs two to four dependent L2 round trips, one or
// two cluster barriers, and the instruction fetches of code that runs once a
// level (32-bit counters and few unrolled loops for that reason). us a call,
// Beamer, and in brackets what the loops of bfs.cu took (CUDA graph / persistent
// kernel): R-MAT edge factor 16, n = 1,024: 37 (180 / 118), 65,536: 70 (277 / 160);
// uniform random, mean degree 8, n = 10,000: 51 (313 / 186), degree 3, 60,000:
// 114 (682 / 370); grid of 65,025: 833 (6,918 / 2,403).
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>

#include "bfs_cluster.h"
#include "block_push.cuh"
#include "graph.h"
#include "selector.cuh"

namespace alb {
namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 1024, kWarps = kThreads / 32;
constexpr int kMaxCtas = 16;
constexpr int kPullWords = 2;    // words a warp pulls at a time
// Frontiers of at most this many rows are walked by every CTA, each taking
// its share of the rows longer than kBigRow; in larger ones a row's edges
// stay with the CTA that owns it.
constexpr int kSplitRows = 1024;
static_assert(kSplitRows <= kPushRows, "the rows of a split level are listed at once");
// Edges a CTA pushes at most at a list level, one per thread (and so the most
// it can claim for its next list).
constexpr int kListCap = kThreads;
// Lists are evened out over the CTAs when one holds more edges than this:
// scattered accesses of one SM start to queue.
constexpr int kListEven = 256;
// A list's rows and edges in one counter, edges in the low bits: with a row's
// edges counted as kEdgeMask >> 10 at most, kListCap rows cannot carry over,
// and a list that is used (kListCap edges at most) is counted exactly.
constexpr int kRowShift = 21;
constexpr unsigned kEdgeMask = (1u << kRowShift) - 1;

struct __align__(16) Counts {
    unsigned n, mo, mi, full;
};

// Frontier rows of one CTA at list levels: where the row starts, its edges
// before it in the list, its id.
struct List {
    int32_t st[kListCap], d[kListCap], off[kListCap], ou[kListCap];
};

struct Shared {
    int level, dir, done, lists;  // lists: the level runs on lists, not on bitmaps
    unsigned nf, mf;
    Counts cnt[2];                // by level parity: what this CTA found
    unsigned longest[2];          // and its longest row, at list levels
    unsigned next_word;
    unsigned nq[2];               // list counters (rows, edges) by level parity
    int even;                     // the lists are evened out before the level
    unsigned before[kMaxCtas + 1];  // rows in the lists of the CTAs before each
    unsigned hit;                 // a cooperative scan's first hit
    PushLists rows;               // frontier rows; or the long rows left after their head
    MlpCopy mlp;
    List q[2];
};

__device__ __forceinline__ void put_counts(Shared &s, int L, unsigned n, unsigned mo, unsigned mi,
                                           unsigned full) {
    n = __reduce_add_sync(kFull, n);
    mo = __reduce_add_sync(kFull, mo);
    mi = __reduce_add_sync(kFull, mi);
    full = __reduce_add_sync(kFull, full);
    if (lane_id() == 0 && (n | full)) {
        Counts &k = s.cnt[L & 1];
        atomicAdd(&k.n, n);
        atomicAdd(&k.mo, mo);
        atomicAdd(&k.mi, mi);
        atomicAdd(&k.full, full);
    }
}

// ------------------------------------------------------------- bitmap levels

// Four pushed edges per lane (v[k] < 0: none) from sources ou[k]: unvisited
// targets take the smallest source as parent and set their bit in this CTA's
// copy of the next frontier. Parents are read before the atomic: a hub's
// targets meet many pushes, and most can no longer lower the parent.
__device__ __forceinline__ void push4(const BfsArgs &a, const uint32_t *V, uint32_t *N,
                                      const int32_t (&v)[4], const uint32_t (&ou)[4]) {
    uint32_t cur[4];
    bool live[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        live[k] = v[k] >= 0 && !((V[v[k] >> 5] >> (v[k] & 31)) & 1u);
        cur[k] = live[k] ? __ldcg(a.parent_pos + v[k]) : 0u;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (!live[k]) continue;
        const uint32_t bit = 1u << (v[k] & 31);
        if (ou[k] < cur[k]) atomicMin(a.parent_pos + v[k], ou[k]);
        if (!(N[v[k] >> 5] & bit)) atomicOr(N + (v[k] >> 5), bit);
    }
}

// This CTA's pushes of the frontier F into its copy N (all words' rows at once
// when few rows are split over the CTAs).
__device__ void push_level(const BfsArgs &a, Shared &s, const uint32_t *F, const uint32_t *V,
                           uint32_t *N, int w0, int w1, int rank, int nctas, bool split) {
    const int from = split ? 0 : w0, to = split ? (int)a.nwords : w1;
    block_push<kThreads>(
        s.rows, F, from, to, split ? to : kPushWords, a.pcol,
        [&](int32_t u, int32_t &st, int32_t &d, int32_t &ou) {
            ALB_CHECK_ID(u, a.n, 0, &a.ctl->err);
            st = (int32_t)__ldg(a.prow + u);
            d = (int32_t)__ldg(a.prow + u + 1) - st;
            ou = __ldg(a.perm + u);
            if (!split) return;
            if (d > kBigRow) {  // this CTA's share
                const int32_t per = (d + nctas - 1) / nctas, skip = min(d, per * rank);
                st += skip;
                d = min(per, d - skip);
            } else if ((u >> 5) < w0 || (u >> 5) >= w1) {
                d = 0;
            }
        },
        [&](int32_t (&v)[4], const uint32_t (&ou)[4]) {
            for (int k = 0; k < 4; k++)
                if (v[k] >= 0) ALB_CHECK_ID(v[k], a.n, -1, &a.ctl->err);
            push4(a, V, N, v, ou);
        });
}

// After the pushes: the CTAs' copies of this CTA's next-frontier words are
// merged, recorded and written back to every copy.
__device__ void merge_words(const BfsArgs &a, Shared &s, cg::cluster_group &cl, int nctas, int L,
                            const uint32_t *V, uint32_t *N, int w0, int w1) {
    const int lane = lane_id();
    unsigned cn = 0, mo = 0, mi = 0, full = 0;
    for (int wb = w0 + (int)(threadIdx.x & ~31u); wb < w1; wb += kThreads) {
        const int w = wb + lane;
        uint32_t m = 0;
        if (w < w1) {
#pragma unroll
            for (int r = 0; r < kMaxCtas; r++)
                if (r < nctas) m |= cl.map_shared_rank(N, r)[w];
#pragma unroll
            for (int r = 0; r < kMaxCtas; r++)
                if (r < nctas) cl.map_shared_rank(N, r)[w] = m;
            const uint32_t v = V[w];
            full += v != kFull && (v | m) == kFull;
        }
        unsigned todo = __ballot_sync(kFull, m != 0);
        while (todo) {
            const int q = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t mq = __shfl_sync(kFull, m, q);
            if (!((mq >> lane) & 1u)) continue;
            const int32_t p = (wb + q) * 32 + lane;
            a.level_pos[p] = L + 1;
            cn++;
            mo += __ldg(a.odeg + p);
            mi += __ldg(a.ideg + p);
        }
    }
    put_counts(s, L, cn, mo, mi, full);
}

// First source of [st, en) in F, as its offset from st (kFull: none); one
// warp, 128 sources a step.
__device__ unsigned scan_row(const BfsArgs &a, const uint32_t *F, int64_t st, int64_t en) {
    const int lane = lane_id();
    for (int64_t e0 = st; e0 < en; e0 += 128) {
        int32_t c[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t e = e0 + 32 * u + lane;
            c[u] = e < en ? __ldg(a.lcol + e) : -1;
            if (c[u] >= 0) ALB_CHECK_ID(c[u], a.n, -1, &a.ctl->err);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const bool hit = c[u] >= 0 && ((F[c[u] >> 5] >> (c[u] & 31)) & 1u);
            const unsigned m = __ballot_sync(kFull, hit);
            if (m) return (unsigned)(e0 - st) + 32 * u + __ffs(m) - 1;
        }
    }
    return kFull;
}

// The unvisited long rows of this CTA's words: a warp scans the first
// kLongChunk sources of a row, the whole CTA what is left of a row without a
// hit there. A hit's parent goes to parent_pos, where pull_words finds it.
__device__ void pull_long(const BfsArgs &a, Shared &s, const uint32_t *F, const uint32_t *V, int w0,
                          int w1) {
    const int lane = lane_id(), wib = threadIdx.x >> 5;
    // long rows are listed by position: this CTA's are [lo, hi)
    int lo = 0, hi = 0;
    for (int side = 0; side < 2; side++) {
        const int key = (side ? w1 : w0) * 32;
        int b = 0, e = (int)a.nlong;
        while (b < e) {
            const int mid = (b + e) >> 1;
            if (__ldg(a.lrow + mid) < key) b = mid + 1;
            else e = mid;
        }
        (side ? hi : lo) = b;
    }
    if (threadIdx.x == 0) s.rows.nlist = 0;
    __syncthreads();
    for (int i = lo + wib; i < hi; i += kWarps) {
        const int32_t p = __ldg(a.lrow + i);
        if ((V[p >> 5] >> (p & 31)) & 1u) continue;
        const int64_t st = __ldg(a.lptr + i), en = __ldg(a.lptr + i + 1);
        // (a full list: the warp scans the whole row)
        const int64_t head = min(en, st + kLongChunk);
        unsigned f = scan_row(a, F, st, head);
        if (f == kFull && head < en) {
            int q = 0;
            if (lane == 0) q = atomicAdd(&s.rows.nlist, 1);
            q = __shfl_sync(kFull, q, 0);
            if (q < kPushRows) {
                if (lane == 0) {
                    s.rows.list[q] = p;
                    s.rows.list_st[q] = i;
                }
            } else {
                f = scan_row(a, F, head, en);
                if (f != kFull) f += (unsigned)(head - st);
            }
        }
        if (f != kFull && lane == 0) {
            int32_t c = __ldg(a.lcol + st + f);
            ALB_CHECK_ID(c, a.n, 0, &a.ctl->err);
            a.parent_pos[p] = (uint32_t)__ldg(a.perm + c);
        }
    }
    __syncthreads();
    const int nrows = min(s.rows.nlist, kPushRows);
    for (int q = 0; q < nrows; q++) {
        const int i = s.rows.list_st[q];
        const int64_t st = __ldg(a.lptr + i) + kLongChunk, en = __ldg(a.lptr + i + 1);
        if (threadIdx.x == 0) s.hit = kFull;
        __syncthreads();
        // each warp its kLongChunk sources of a CTA-wide step; the smallest
        // offset of the first step with a hit
        for (int64_t e0 = st; e0 < en; e0 += kWarps * kLongChunk) {
            const int64_t b = e0 + wib * kLongChunk;
            if (b < en) {
                const unsigned f = scan_row(a, F, b, min(en, b + kLongChunk));
                if (f != kFull && lane == 0) atomicMin(&s.hit, (unsigned)(b - st) + f);
            }
            __syncthreads();
            const bool found = s.hit != kFull;
            __syncthreads();
            if (found) break;
        }
        if (threadIdx.x == 0 && s.hit != kFull) {
            int32_t c = __ldg(a.lcol + st + s.hit);
            ALB_CHECK_ID(c, a.n, 0, &a.ctl->err);
            a.parent_pos[s.rows.list[q]] = (uint32_t)__ldg(a.perm + c);
        }
        __syncthreads();
    }
}

// Bottom-up pull of this CTA's words, kPullWords at a time per warp: lane l
// scans row l of each, the next column group requested before the current
// one's frontier tests. Finished next-frontier words go into every CTA's copy.
__device__ void pull_words(const BfsArgs &a, Shared &s, cg::cluster_group &cl, int nctas, int L,
                           const uint32_t *F, const uint32_t *V, uint32_t *N, int w0, int w1) {
    const int lane = lane_id();
    const int32_t C = a.C, log2C = a.log2C;
    unsigned cn = 0, mo = 0, mi = 0, full = 0;
    while (true) {
        unsigned g = 0;
        if (lane == 0) g = atomicAdd(&s.next_word, (unsigned)kPullWords);
        const int wa = w0 + (int)__shfl_sync(kFull, g, 0);
        if (wa >= w1) break;
        uint32_t vis[kPullWords];
        int32_t p[kPullWords], ng[kPullWords], found[kPullWords];
        bool act[kPullWords], maybe_long[kPullWords];
        const int4 *cp[kPullWords];
        int4 c[kPullWords];
        int64_t so[kPullWords];
#pragma unroll
        for (int t = 0; t < kPullWords; t++) {
            const int w = wa + t;
            vis[t] = w < w1 ? V[w] : kFull;
            p[t] = w * 32 + lane;
            act[t] = !((vis[t] >> lane) & 1u);
            found[t] = -1;
            const int32_t sl = (act[t] ? p[t] : 0) >> log2C;
            ng[t] = act[t] ? (__ldg(a.width + sl) + 3) >> 2 : 0;
            so[t] = act[t] ? __ldg(a.slice_off + sl) : 0;
        }
#pragma unroll
        for (int t = 0; t < kPullWords; t++) {
            cp[t] = a.col4 + (so[t] >> 2) + (p[t] & (C - 1));
            c[t] = make_int4(p[t], p[t], p[t], p[t]);
            if (ng[t] > 0) c[t] = __ldg(cp[t]);
        }
        // an unvisited row whose first entry is padding is a long row
#pragma unroll
        for (int t = 0; t < kPullWords; t++) maybe_long[t] = act[t] && c[t].x == p[t];
        for (int32_t j = 0;; j++) {
            bool any = false;
#pragma unroll
            for (int t = 0; t < kPullWords; t++) {
                act[t] = act[t] && j < ng[t];
                any = any || act[t];
            }
            if (!__any_sync(kFull, any)) break;
#pragma unroll
            for (int t = 0; t < kPullWords; t++) {
                if (!act[t]) continue;
                int4 nx = make_int4(p[t], p[t], p[t], p[t]);
                if (j + 1 < ng[t]) nx = __ldg(cp[t] + (int64_t)(j + 1) * C);
                ALB_CHECK_ID4(c[t], a.nwords * 32, p[t], &a.ctl->err);
                // padding is the row itself, which is not in the frontier and
                // ends the row: the first hit is the smallest source
                const bool h0 = (F[c[t].x >> 5] >> (c[t].x & 31)) & 1u,
                           h1 = (F[c[t].y >> 5] >> (c[t].y & 31)) & 1u,
                           h2 = (F[c[t].z >> 5] >> (c[t].z & 31)) & 1u,
                           h3 = (F[c[t].w >> 5] >> (c[t].w & 31)) & 1u;
                if (h0 | h1 | h2 | h3) found[t] = h0 ? c[t].x : h1 ? c[t].y : h2 ? c[t].z : c[t].w;
                act[t] = found[t] < 0 && c[t].w != p[t];
                c[t] = nx;
            }
        }
#pragma unroll
        for (int t = 0; t < kPullWords; t++) {
            if (wa + t >= w1) break;
            bool reached = found[t] >= 0, by_long = false;
            if (maybe_long[t] && !reached && a.nlong)
                by_long = reached = __ldcg(a.parent_pos + p[t]) != kFull;
            const unsigned nm = __ballot_sync(kFull, reached);
            if (lane < nctas) cl.map_shared_rank(N, lane)[wa + t] = nm;
            if (lane == 0) full += vis[t] != kFull && (vis[t] | nm) == kFull;
            if (reached) {
                a.level_pos[p[t]] = L + 1;
                if (!by_long) a.parent_pos[p[t]] = (uint32_t)__ldg(a.perm + found[t]);
                cn++;
                mo += __ldg(a.odeg + p[t]);
                mi += __ldg(a.ideg + p[t]);
            }
        }
    }
    put_counts(s, L, cn, mo, mi, full);
}

// --------------------------------------------------------------- list levels
//
// A small frontier (kListCap edges at most in any CTA, an edge per thread) is
// kept as one list per CTA, in shared memory: the CTA that claims a vertex
// pushes it at the next level, and lists that grew apart are evened out. A
// target is claimed by the compare-and-swap that moves its level from -1, and
// its row's bounds and id are requested together with it, so a level is two
// round trips to L2 and one barrier. The bitmaps go stale
// and are rebuilt from the levels when a level needs them (lists_to_maps); under
// the learned policy, to which the words with an unvisited row are a feature,
// the visited words are kept up by the CTAs that own them.

__device__ __forceinline__ void append(List &q, unsigned *nq, int32_t st, int32_t d, int32_t ou) {
    const unsigned at = atomicAdd(nq, (1u << kRowShift) | min((unsigned)d, kEdgeMask >> 10));
    const unsigned i = at >> kRowShift;
    q.st[i] = st;
    q.d[i] = d;
    q.off[i] = (int32_t)(at & kEdgeMask);
    q.ou[i] = ou;
}

__device__ void maps_to_lists(const BfsArgs &a, Shared &s, const uint32_t *F, int par, int w0,
                              int w1) {
    if (threadIdx.x == 0) s.nq[par] = 0;
    __syncthreads();
    for (int w = w0 + (int)threadIdx.x; w < w1; w += kThreads) {
        for (uint32_t m = F[w]; m; m &= m - 1) {
            int32_t u = w * 32 + __ffs(m) - 1;
            ALB_CHECK_ID(u, a.n, 0, &a.ctl->err);
            const int32_t st = (int32_t)__ldg(a.prow + u);
            append(s.q[par], &s.nq[par], st, (int32_t)__ldg(a.prow + u + 1) - st,
                   __ldg(a.perm + u));
        }
    }
    __syncthreads();
}

// Every CTA takes an equal run of the rows of all lists, one row per thread.
__device__ void even_lists(Shared &s, cg::cluster_group &cl, int rank, int nctas, int par) {
    const unsigned tot = s.before[nctas];
    const unsigned g = tot * rank / nctas + threadIdx.x, end = tot * (rank + 1) / nctas;
    int32_t st = 0, d = 0, ou = 0;
    if (g < end) {
        int c = 0;
        while (s.before[c + 1] <= g) c++;
        const List &q = cl.map_shared_rank(&s, c)->q[par];
        const unsigned i = g - s.before[c];
        st = q.st[i];
        d = q.d[i];
        ou = q.ou[i];
    }
    cl.sync();  // every list has been read
    if (threadIdx.x == 0) s.nq[par] = 0;
    __syncthreads();
    if (g < end) append(s.q[par], &s.nq[par], st, d, ou);
    __syncthreads();
}

// V: the visited words, per of them a CTA (kLearned).
template <bool kLearned>
__device__ void list_level(const BfsArgs &a, Shared &s, cg::cluster_group &cl, int L, uint32_t *V,
                           int per) {
    const List &q = s.q[L & 1];
    const unsigned cnt = s.nq[L & 1];
    const int nq = (int)(cnt >> kRowShift), e = (int)threadIdx.x;
    int32_t v = -1, st = 0, len = 0, id = 0, in_len = 0;
    uint32_t word = kFull;  // the target's visited word before
    bool claimed = false;
    if (e < (int)(cnt & kEdgeMask)) {
        int j = 0;  // the last row that starts at or before edge e (rows
                    // without edges share their start with the next one)
        for (int step = kListCap / 2; step > 0; step >>= 1)
            if (j + step < nq && q.off[j + step] <= e) j += step;
        v = __ldg(a.pcol + q.st[j] + (e - q.off[j]));
        ALB_CHECK_ID(v, a.n, -1, &a.ctl->err);
        if (v >= 0) {
            const int32_t old = atomicCAS(a.level_pos + v, -1, L + 1);
            // (visited when the level ends, whoever claims it)
            if (kLearned)
                word = atomicOr(cl.map_shared_rank(V, (v >> 5) / per) + (v >> 5), 1u << (v & 31));
            const uint32_t cur = __ldcg(a.parent_pos + v), ou = (uint32_t)q.ou[j];
            st = (int32_t)__ldg(a.prow + v);
            len = (int32_t)__ldg(a.prow + v + 1) - st;
            id = __ldg(a.perm + v);
            in_len = __ldg(a.ideg + v);
            claimed = old == -1;
            if ((claimed || old == L + 1) && ou < cur) atomicMin(a.parent_pos + v, ou);
        }
    }
    if (claimed) append(s.q[(L + 1) & 1], &s.nq[(L + 1) & 1], st, len, id);
    Counts &k = s.cnt[L & 1];
    if (kLearned) {
        const unsigned full =
            __ballot_sync(kFull, word != kFull && (word | (1u << (v & 31))) == kFull);
        if (lane_id() == 0 && full) atomicAdd(&k.full, __popc(full));
    }
    if (!__any_sync(kFull, claimed)) return;
    const unsigned n = __popc(__ballot_sync(kFull, claimed));
    const unsigned mo = __reduce_add_sync(kFull, claimed ? (unsigned)len : 0u);
    const unsigned mi = __reduce_add_sync(kFull, claimed ? (unsigned)in_len : 0u);
    const unsigned longest = __reduce_max_sync(kFull, claimed ? (unsigned)len : 0u);
    if (lane_id() == 0) {
        atomicAdd(&k.n, n);
        atomicAdd(&k.mo, mo);
        atomicAdd(&k.mi, mi);
        atomicMax(&s.longest[L & 1], longest);
    }
}

// The bitmaps of level L from the levels: this CTA's words, into every copy.
// Returns (in one lane of each warp) the words with an unvisited row.
__device__ void lists_to_maps(const BfsArgs &a, Shared &s, cg::cluster_group &cl, int nctas, int L,
                              uint32_t *F, uint32_t *V, int w0, int w1) {
    const int lane = lane_id();
    unsigned active = 0;
    for (int w = w0 + (int)(threadIdx.x >> 5); w < w1; w += kWarps) {
        const int32_t p = w * 32 + lane;
        const int32_t lp = p < a.n ? __ldcg(a.level_pos + p) : -1;
        const uint32_t v = __ballot_sync(kFull, lp >= 0) | __ldg(a.vinit + w);
        const uint32_t f = __ballot_sync(kFull, lp == L);
        if (lane < nctas) {
            cl.map_shared_rank(F, lane)[w] = f;
            cl.map_shared_rank(V, lane)[w] = v;
        }
        active += v != kFull;
    }
    if (lane == 0 && active) atomicAdd(&s.cnt[L & 1].full, active);
}

// The traversal's state, held by every lane of warp 0 of each CTA alike.
struct State {
    int level, prev_dir, levels_td, levels_bu;
    unsigned nf, prev_nf, mf, nu, mu, active, reached, edges;
};

// The next level's direction and form (warp 0). most: the largest number of
// edges any one CTA's list holds (after a bitmap level, the frontier's edges
// or rows: any CTA might get them all).
template <bool kLearned>
__device__ void next_level(Shared &s, const State &t, const BfsArgs &a, const InitParams &in,
                           unsigned most) {
    BfsCtl c;
    c.level = t.level;
    c.prev_dir = t.prev_dir;
    c.policy = in.policy;
    c.alpha = in.alpha;
    c.beta = in.beta;
    c.n = a.n;
    c.nwords = a.nwords;
    c.nf = t.nf;
    c.prev_nf = t.prev_nf;
    c.mf = t.mf;
    c.nu = t.nu;
    c.mu = t.mu;
    c.active_words = t.active;
    c.feat_mean_deg = in.mean_deg;
    c.feat_skew = in.skew;
    int dir;
    if (kLearned && s.mlp.loaded()) {
        float f[kMlpIn];
        level_features_warp(c, f);
        dir = s.mlp.select(f);
    } else {
        dir = rule_dir(c);
    }
    if (lane_id() == 0) {
        s.level = t.level;
        s.nf = t.nf;
        s.mf = t.mf;
        s.dir = dir;
        s.lists = dir == ALB_DIR_TOPDOWN && most <= kListCap;
        s.next_word = 0;
        s.nq[(t.level + 1) & 1] = 0;
    }
}

// kLearned: the learned policy, and weights may be loaded.
template <bool kLearned>
__global__ void __launch_bounds__(kThreads, 1)
    k_bfs_cluster(BfsArgs a, InitParams in, int32_t *out_level, int32_t *out_parent,
                  BfsCtl *result) {
    extern __shared__ __align__(16) unsigned char smem[];
    Shared &s = *reinterpret_cast<Shared *>(smem);
    uint32_t *maps = reinterpret_cast<uint32_t *>(smem + sizeof(Shared));  // X0 | X1 | V
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), nctas = (int)cl.num_blocks();
    const int nw = (int)a.nwords;
    const int per = (nw + nctas - 1) / nctas;
    const int w0 = min(nw, rank * per), w1 = min(nw, w0 + per);  // own words
    uint32_t *V = maps + 2 * nw;
    const int32_t p0 = w0 * 32, p1 = (int32_t)min(a.n, (int64_t)w1 * 32);
    // the root's position and degrees, in flight during the clearing
    const int32_t rp = __ldg(a.inv + in.root);
    const int32_t r_out = __ldg(a.odeg + rp), r_in = __ldg(a.ideg + rp);
    for (int w = threadIdx.x; w < nw; w += kThreads) {
        V[w] = __ldg(a.vinit + w);
        maps[w] = 0;
    }
    for (int32_t p = p0 + (int32_t)threadIdx.x; p < p1; p += kThreads) {
        a.level_pos[p] = -1;
        a.parent_pos[p] = kFull;
    }
    if (kLearned) s.mlp.load(a.mlp);
    if (threadIdx.x < 8) reinterpret_cast<unsigned *>(s.cnt)[threadIdx.x] = 0;
    if (threadIdx.x < 2) s.longest[threadIdx.x] = 0;
    __syncthreads();
    State t;
    const uint32_t rbit = 1u << (rp & 31), rold = V[rp >> 5];
    t.level = t.levels_td = t.levels_bu = 0;
    t.prev_dir = -1;
    t.nf = t.reached = 1;
    t.prev_nf = 0;
    t.mf = t.edges = r_out;
    t.nu = (unsigned)in.n_live - (r_in > 0 ? 1 : 0);
    t.mu = (unsigned)in.m_in - r_in;
    t.active = (unsigned)in.active0 - ((rold != kFull && (rold | rbit) == kFull) ? 1 : 0);
    __syncthreads();
    if (threadIdx.x == 0) {
        V[rp >> 5] = rold | rbit;
        maps[rp >> 5] = rbit;
        if (rp >= p0 && rp < p1) {
            a.level_pos[rp] = 0;
            a.parent_pos[rp] = (uint32_t)in.root;
        }
        if (rank == 0) a.ctl->err = 0;
        s.done = 0;
    }
    if (threadIdx.x < 32) next_level<kLearned>(s, t, a, in, t.mf);
    cl.sync();
    bool listed = false;  // the lists hold the frontier, the bitmaps are stale
    while (true) {
        const int L = s.level, dir = s.dir;
        const bool lists = s.lists;
        uint32_t *F = maps + (L & 1 ? nw : 0);
        uint32_t *N = maps + (L & 1 ? 0 : nw);
        if (listed && !lists) {
            lists_to_maps(a, s, cl, nctas, L, F, V, w0, w1);
            cl.sync();
            if (threadIdx.x < 32) {
                unsigned k = 0;
                if ((int)threadIdx.x < nctas) k = cl.map_shared_rank(&s, threadIdx.x)->cnt[L & 1].full;
                t.active = __reduce_add_sync(kFull, k);
            }
            cl.sync();  // read by all before it is reset
            if (threadIdx.x == 0) s.cnt[L & 1].full = 0;
            __syncthreads();
            listed = false;
        }
        if (lists) {
            if (!listed) {
                maps_to_lists(a, s, F, L & 1, w0, w1);
                // (the last level's visited bits are in before others claim)
                if (kLearned) cl.sync();
            } else if (s.even) even_lists(s, cl, rank, nctas, L & 1);
            listed = true;
            list_level<kLearned>(a, s, cl, L, V, per);
        } else if (dir == ALB_DIR_TOPDOWN) {
            for (int w = threadIdx.x; w < nw; w += kThreads) N[w] = 0;
            push_level(a, s, F, V, N, w0, w1, rank, nctas, s.nf <= kSplitRows);
            cl.sync();
            merge_words(a, s, cl, nctas, L, V, N, w0, w1);
        } else {
            if (a.nlong) pull_long(a, s, F, V, w0, w1);
            pull_words(a, s, cl, nctas, L, F, V, N, w0, w1);
        }
        cl.sync();
        if (threadIdx.x < 32) {
            Counts k = {0, 0, 0, 0};
            if ((int)threadIdx.x < nctas) k = cl.map_shared_rank(&s, threadIdx.x)->cnt[L & 1];
            const unsigned most = lists ? __reduce_max_sync(kFull, k.mo) : 0;
            if (lists) {
                unsigned longest = 0;
                if ((int)threadIdx.x < nctas)
                    longest = cl.map_shared_rank(&s, threadIdx.x)->longest[L & 1];
                longest = __reduce_max_sync(kFull, longest);
                const unsigned upto = warp_inclusive_scan(k.n);
                const unsigned tot = __shfl_sync(kFull, upto, 31);
                if ((int)threadIdx.x < nctas) s.before[threadIdx.x] = upto - k.n;
                if (threadIdx.x == 0) {
                    s.before[nctas] = tot;
                    s.even = most > kListEven && nctas > 1 &&
                             (tot / nctas + 1) * (unsigned long long)longest <= kListCap;
                }
            }
            t.prev_nf = t.nf;
            t.nf = __reduce_add_sync(kFull, k.n);
            t.mf = __reduce_add_sync(kFull, k.mo);
            t.mu -= __reduce_add_sync(kFull, k.mi);
            t.active -= __reduce_add_sync(kFull, k.full);
            t.nu -= t.nf;
            t.reached += t.nf;
            t.edges += t.mf;
            t.prev_dir = dir;
            if (dir == ALB_DIR_TOPDOWN) t.levels_td++;
            else t.levels_bu++;
            t.level++;
            if (threadIdx.x == 0) {
                // (the other parity's counts were read by everyone before the
                // last barrier)
                s.cnt[(L + 1) & 1] = Counts{0, 0, 0, 0};
                s.longest[(L + 1) & 1] = 0;
                s.done = t.nf == 0 || t.level >= in.level_cap;
            }
            next_level<kLearned>(s, t, a, in, lists ? most : max(t.mf, t.nf));
        } else if (!lists) {
            for (int w = threadIdx.x - 32; w < nw; w += kThreads - 32) V[w] |= N[w];
        }
        __syncthreads();
        if (s.done) break;
    }
    for (int32_t p = p0 + (int32_t)threadIdx.x; p < p1; p += kThreads) {
        const int32_t v = __ldg(a.perm + p);
        if (out_level) out_level[v] = __ldcg(a.level_pos + p);
        if (out_parent) out_parent[v] = (int32_t)__ldcg(a.parent_pos + p);
    }
    if (rank == 0 && threadIdx.x == 0) {
        result->level = t.level;
        result->done = 1;
        result->err = *(volatile int32_t *)&a.ctl->err;
        result->levels_td = t.levels_td;
        result->levels_bu = t.levels_bu;
        result->reached = t.reached;
        result->edges = t.edges;
    }
    cl.sync();  // no CTA leaves while another may read its counts
}

// CTAs for a graph of nw bitmap words: enough that every warp has a word.
int cluster_ctas(int64_t nw) {
    int k = 1;
    while (k < kMaxCtas && (int64_t)k * kWarps < nw) k <<= 1;
    return k;
}

// Dynamic shared memory: the CTA's state and the three bitmaps.
size_t map_bytes(int64_t nw) { return sizeof(Shared) + sizeof(uint32_t) * 3 * (size_t)nw; }

using Kernel = void (*)(BfsArgs, InitParams, int32_t *, int32_t *, BfsCtl *);

cudaError_t allow_cluster(Kernel f) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)map_bytes(kClusterMaxN / 32));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

cudaLaunchConfig_t config(int ctas, size_t smem, cudaStream_t st, cudaLaunchAttribute &at) {
    at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cfg;
}

// Whether the device runs a cluster of the largest shape (asked once for each).
bool cluster_ready(int device) {
    static std::mutex mu;
    static std::map<int, bool> known;
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find(device);
    if (it != known.end()) return it->second;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = config(kMaxCtas, map_bytes(kClusterMaxN / 32), nullptr, at);
    bool ok = true;
    for (Kernel f : {k_bfs_cluster<false>, k_bfs_cluster<true>}) {
        int n = 0;
        ok = ok && allow_cluster(f) == cudaSuccess &&
             cudaOccupancyMaxActiveClusters(&n, f, &cfg) == cudaSuccess && n >= 1;
    }
    if (!ok) cudaGetLastError();
    known[device] = ok;
    return ok;
}

}  // namespace

bool cluster_takes(const alb_graph *g, const alb_bfs_opts &o, const BfsArgs &a) {
    // Policies that push (or may) go to all SMs where there are many edges a
    // vertex: 16 SMs push 2 M edges of 4,000 vertices in 189 us, all of them in
    // 89, 33 M of 65,000 in 948 and 201 (learned 214 / 92, 99 / 86); around 100 a
    // vertex, R-MAT of 2^15, learned is 75 / 83 and top-down 153 / 109. The other
    // policies pull there: 38 / 60 and 93 / 83.
    if ((o.policy == ALB_POLICY_TOPDOWN || o.policy == ALB_POLICY_LEARNED) &&
        g->sell.m_out > 100 * g->n)
        return false;
    // (counters are 32 bits wide)
    return g->n <= kClusterMaxN && g->sell.m_in <= INT32_MAX && g->sell.m_out <= INT32_MAX &&
           o.loop != ALB_LOOP_HOST && !o.trace && o.policy != ALB_POLICY_BOTTOMUP_NOBYPASS &&
           a.withhold_level < 0 && !a.short_bulk && cluster_ready(g->device);
}

alb_status cluster_launch(const BfsArgs &a, const InitParams &in, int32_t *d_level,
                          int32_t *d_parent, BfsCtl *result, cudaStream_t st) {
    const Kernel f = in.policy == ALB_POLICY_LEARNED && a.mlp ? k_bfs_cluster<true>
                                                              : k_bfs_cluster<false>;
    ALB_CK(allow_cluster(f));
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = config(cluster_ctas(a.nwords), map_bytes(a.nwords), st, at);
    ALB_CK(cudaLaunchKernelEx(&cfg, f, a, in, d_level, d_parent, result));
    return ALB_OK;
}

}  // namespace alb
