// Single-root BFS as one cooperative kernel, one block of 1024 threads per SM:
// initial state, every level, counters. Outputs are written by a second kernel
// (k_scatter_tiles). It serves both device-driven loops of graphs too large
// for one cluster, or too dense for its pushes (bfs_cluster.cu); traced runs and
// the pull without bypass keep the kernels of bfs.cu, whose counters they report.
//
// Blocks meet at one arrival counter (1.3 us; records that every block stores
// and every block polls took 4.6, on lines of their own 2.2). What a phase
// counted is added up in the block and goes out as one atomic per counter and
// block; at list levels it rides on the arrival itself: the word that the
// blocks wait on holds the arrivals, the claimed vertices and their edges.
//
// A frontier lives in one of three forms: a bitmap (after a bottom-up level),
// a bitmap and a queue (after a top-down level), or one list per block in
// shared memory (small frontiers): the block that claims a vertex pushes it
// at the next level, with the row's bounds and id fetched together with the
// claim, so that a level is two round trips to memory and one barrier.
//
// Bottom-up levels come in two shapes: word by word while most rows of a word
// are unvisited (coalesced column loads, lane per row), and row by row when
// few are (the unvisited rows of 32 words dealt out to the lanes), where the
// word shape would wait out a chain of loads for one or two rows of each word.
#include <algorithm>
#include <cstring>

#include "bfs_grid.h"
#include "graph.h"
#include "selector.cuh"

namespace alb {
namespace {

constexpr int kThreads = 1024, kWarps = kThreads / 32;
constexpr int kMaxBlocks = 160;     // fields of a list level's word
constexpr int kCtl = kWarps - 1;    // the warp that waits at barriers and decides
constexpr int kListThreads = kThreads - 32;  // the others hold a list's edges
constexpr int kPer = 2;             // edges per thread and pass
// A block's edges at a list level: one pass, or three on graphs without long
// rows (grids), whose searches are list levels almost throughout. The grid of
// 2^24 has frontiers of up to 150,000 rows and 570,000 edges: 12 to 15 us a
// list level, 35 a level of queues (two passes were too few for 37 of its 503).
constexpr int kListPass = kPer * kListThreads, kListCapMax = 3 * kListPass;
// Its rows, which are what takes shared memory (and L1 from the other phases):
// a claim past them goes to the queue and the bitmap (overflow).
constexpr int kListRows = kListPass;
constexpr int kFewEdges = 16;       // longest row of such a graph
constexpr int kListRow = 255;       // the longest row that claims put on a list
constexpr int kRowShift = 19;       // list counters: rows above, edges below
constexpr unsigned kEdgeMask = (1u << kRowShift) - 1;
static_assert((int64_t)kListPass * kListRow <= kEdgeMask && kListCapMax * kFewEdges <= kEdgeMask &&
                  kListCapMax < 1 << (32 - kRowShift),
              "a list's counter");
constexpr int kBigShift = 38;  // big-row counter: rows above, chunks below
constexpr unsigned long long kBigMask = (1ull << kBigShift) - 1;
constexpr int64_t kStageMax = 192 * 1024;  // frontier bitmap staged in shared memory

// A level's frontier.
enum Form : int { kMap = 0, kQueue = 1, kList = 2 };

struct __align__(16) Counts {
    unsigned long long mo, mi;
    unsigned n, full;
};

// A list's rows: start of the push row less the edges before it in the list,
// those edges, the row's id and position. Four arrays of kListRows entries.
struct List {
    uint32_t *st;
    int32_t *off, *ou, *pos;
};

struct Shared {
    BfsCtl c;
    // of the call: longest push row, rows and entries as GridArgs has them
    int64_t max_out, m_out;
    int level_cap, learned, cap;  // cap: edges of a list
    int dir, form, lists, even, sparse, scan, ok, over, uneven;
    Counts warp[kWarps];
    // sums of the last counting barrier; nbig: the big-row counter
    unsigned long long n, mo, mi, full, nbig;
    unsigned nq[2];
    unsigned cn, cmo, cmi, wide;  // a list level's claims in this block; rows too long for it
    unsigned cwords;              // words of the visited bitmap that they filled (kExact)
    unsigned long long at;  // this block's place in a queue
    __align__(8) uint64_t bar;
    MlpCopy mlp;
};

// Dynamic shared memory: Shared, then one of these at a time: two lists by
// level parity, the warps' row numbers, or the staged frontier.
union Pool {
    uint32_t lists[2 * 4 * kListRows];
    uint16_t rows[kWarps][1024];  // bitmap bits of 32 words as row numbers
    uint32_t stage[1];
};
constexpr size_t kPoolAt = (sizeof(Shared) + 15) & ~(size_t)15;

// (declared where it is used, so that its accesses are known to be shared)
#define ALB_GRID_SHARED                                   \
    extern __shared__ __align__(16) unsigned char dyn[]; \
    Shared &s = *reinterpret_cast<Shared *>(dyn);        \
    Pool &pool = *reinterpret_cast<Pool *>(dyn + kPoolAt)

__device__ __forceinline__ List list_at(Pool &pool, int par) {
    constexpr int n = kListRows;
    uint32_t *b = pool.lists + (size_t)par * 4 * n;
    return List{b, (int32_t *)b + n, (int32_t *)b + 2 * n, (int32_t *)b + 3 * n};
}

// ------------------------------------------------------------- the barriers

// The counting barriers that one level can have, each with four sums of its
// own in the level's row of GridSlots::acc: a block may add to the next one's
// while another still reads back the last one's.
enum Sums : int { kSumLevel = 0, kSumLong = 4, kSumFits = 8, kSumActive = 12 };

constexpr unsigned long long kBarFailed = 1ull << 62;  // a wait gave up
// The arrival counter's word of a.bar, a line apart from the one that the
// traced persistent kernel counts on (and starts from 0 each time).
constexpr int kBarWord = 16;

__device__ __forceinline__ unsigned long long atom_add_acq_rel(unsigned long long *p,
                                                               unsigned long long v) {
    unsigned long long old;
    asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v)
                 : "memory");
    return old;
}

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ bool withheld(const BfsArgs &a, int L) {
    return a.withhold_level >= 0 && L == a.withhold_level && (int)blockIdx.x == a.withhold_block;
}

__device__ __forceinline__ unsigned long long sum64(unsigned long long v) { return warp_sum(v); }

// What the calling warp counted; the next counting barrier adds it up.
__device__ __forceinline__ void put_counts(Shared &s, unsigned n, unsigned long long mo,
                                           unsigned long long mi, unsigned full) {
    Counts k;
    k.n = __reduce_add_sync(kFull, n);
    k.full = __reduce_add_sync(kFull, full);
    k.mo = sum64(mo);
    k.mi = sum64(mi);
    if (lane_id() == 0) s.warp[threadIdx.x >> 5] = k;
}

// Grid barrier on the arrival counter, which is never reset: a block's
// barrier ends when the count reaches the next multiple of the block count.
// acc (null: none): the counts of every warp of every block are added up there
// and read back into s.n .. s.full. big (null: none): read into s.nbig.
__device__ bool barrier(const BfsArgs &a, Shared &s, int L, unsigned long long *acc = nullptr,
                        const unsigned long long *big = nullptr) {
    if (withheld(a, L)) return false;
    __syncthreads();
    if ((threadIdx.x >> 5) == kCtl) {
        const unsigned lane = lane_id();
        if (acc) {
            const Counts k = s.warp[lane];
            const unsigned n = __reduce_add_sync(kFull, k.n), full = __reduce_add_sync(kFull, k.full);
            const unsigned long long mo = sum64(k.mo), mi = sum64(k.mi);
            const unsigned long long v = lane == 0 ? n : lane == 1 ? full : lane == 2 ? mo : mi;
            if (lane < 4 && v) atomicAdd(acc + lane, v);
            __syncwarp();
        }
        const unsigned long long nb = gridDim.x;
        unsigned long long *bar = a.bar + kBarWord, v = 0;
        if (lane == 0) v = atom_add_acq_rel(bar, 1ull);
        v = __shfl_sync(kFull, v, 0);
        const unsigned long long target = (v / nb + 1) * nb;
        v++;
        const uint64_t t0 = globaltimer_ns();
        bool ok = true;
        while (__any_sync(kFull, v < target)) {  // (all lanes poll: see list_barrier)
            if (__any_sync(kFull, globaltimer_ns() - t0 > a.barrier_ns)) {
                if (lane == 0) {
                    atomicExch(&a.ctl->err, ALB_ERR_TIMEOUT);
                    atomicOr(bar, kBarFailed);
                }
                ok = false;
                break;
            }
            v = ld_acquire(bar);
        }
        if (lane == 0) s.ok = ok && !(v & kBarFailed);
        __syncwarp();
        if (acc && lane < 4)
            (lane == 0 ? s.n : lane == 1 ? s.full : lane == 2 ? s.mo : s.mi) = __ldcg(acc + lane);
        if (big && lane == 4) s.nbig = __ldcg(big);
    }
    __syncthreads();
    return s.ok;
}

// The list level's barrier word: 8 bits of arrivals, 8 of blocks whose next
// list does not fit, 8 of blocks with more than five eighths of that, 20 of
// claimed vertices, 20 of their edges, a block's counted up to 2^12 - 1: exact
// where neither flag is set.
constexpr int kArrive = 56, kOver = 48, kUneven = 40, kVerts = 20, kEdgeBits = 12;
static_assert(kMaxBlocks * kListCapMax < (1 << (kUneven - kVerts)) && kMaxBlocks < 256 &&
                  kMaxBlocks * ((1 << kEdgeBits) - 1) < (1 << kVerts) &&
                  5 * kListCapMax / 8 < (1 << kEdgeBits),
              "fields of the list word");

// One warp, after the block's claims: arrives and waits, and leaves the sums in
// s, exactly: acc holds the edges where the word does not, and filled words. All lanes poll: with
// one lane waiting the warp came out of it in two parts, and every shuffle of
// the decision that follows paid for bringing them together (12,900 cycles
// instead of 2,000).
template <bool kExact>
__device__ __forceinline__ bool list_barrier(const BfsArgs &a, const GridArgs &x, Shared &s, int L,
                                             unsigned long long *word, unsigned long long *acc) {
    if (withheld(a, L)) return false;
    const unsigned mo = s.cmo, mi = s.cmi, cn = s.cn;
    const bool over = s.wide || mo > (unsigned)s.cap || cn > (unsigned)kListRows;
    const unsigned long long mine = (1ull << kArrive) | ((unsigned long long)over << kOver) |
                                    ((unsigned long long)(8 * mo > 5 * (unsigned)s.cap) << kUneven) |
                                    ((unsigned long long)cn << kVerts) |
                                    min(mo, (1u << kEdgeBits) - 1);
    const unsigned lane = lane_id();
    __syncwarp();
    if (lane == 0 && mo) atomicAdd(acc, (unsigned long long)mo);
    if (lane == 0 && !x.sym && mi) atomicAdd(acc + 1, (unsigned long long)mi);
    if (kExact && lane == 0 && s.cwords) atomicAdd(acc + 2, (unsigned long long)s.cwords);
    if (lane == 0) s.cn = s.cmo = s.cmi = s.wide = 0;
    if (kExact && lane == 0) s.cwords = 0;
    unsigned long long v = 0;
    if (lane == 0) v = atom_add_acq_rel(word, mine) + mine;
    v = __shfl_sync(kFull, v, 0);
    const unsigned nb = gridDim.x;
    const uint64_t t0 = globaltimer_ns();
    bool ok = true;
    while (__any_sync(kFull, (v >> kArrive) != nb)) {
        if (__any_sync(kFull, globaltimer_ns() - t0 > a.barrier_ns)) {
            if (lane == 0) atomicExch(&a.ctl->err, ALB_ERR_TIMEOUT);
            ok = false;
            break;
        }
        v = ld_acquire(word);
    }
    const bool any_over = ((v >> kOver) & 255) != 0, any_uneven = ((v >> kUneven) & 255) != 0;
    unsigned long long emo = v & ((1u << kVerts) - 1);
    if (any_over || any_uneven) emo = __ldcg(acc);
    const unsigned long long emi = x.sym ? emo : __ldcg(acc + 1);
    const unsigned long long words = kExact ? __ldcg(acc + 2) : 0;
    if (lane == 0) {
        s.n = (v >> kVerts) & ((1u << (kUneven - kVerts)) - 1);
        s.uneven = any_uneven;
        s.over = any_over;
        s.mo = emo;
        s.mi = emi;
        s.full = words;
    }
    __syncwarp();
    return ok;
}

// --------------------------------------------------------------- list levels

// d_count: the row's edges as counted, at most kListRow where the list may
// turn out too large to be used.
// False: no room.
__device__ __forceinline__ bool append(const List &q, unsigned *nq, int32_t u, int64_t st,
                                       int32_t d_count, int32_t ou) {
    const unsigned at = atomicAdd(nq, (1u << kRowShift) | (unsigned)d_count);
    const unsigned i = at >> kRowShift, off = at & kEdgeMask;
    if (i >= (unsigned)kListRows) return false;
    q.st[i] = (uint32_t)st - off;
    q.off[i] = (int32_t)off;
    q.ou[i] = ou;
    q.pos[i] = u;
    return true;
}

// A push row's start, length and id: one 16-byte record (GridArgs::vrec), or
// from the three arrays.
struct RowRec {
    int64_t st;
    int32_t d, id;
};
__device__ __forceinline__ RowRec row_rec(const BfsArgs &a, const int4 *vrec, int32_t u) {
    RowRec r;
    if (vrec) {
        const int4 q = __ldg(vrec + u);
        r.st = (int64_t)(((uint64_t)(uint32_t)q.y << 32) | (uint32_t)q.x);
        r.d = q.z;
        r.id = q.w;
    } else {
        r.st = __ldg(a.prow + u);
        r.d = (int32_t)(__ldg(a.prow + u + 1) - r.st);
        r.id = __ldg(a.perm + u);
    }
    return r;
}

__device__ __forceinline__ void append_row(const BfsArgs &a, const int4 *vrec, const List &q,
                                           unsigned *nq, int32_t u, int32_t most) {
    ALB_CHECK_ID(u, a.n, 0, &a.ctl->err);
    const RowRec r = row_rec(a, vrec, u);
    // (no room: a queue's share that is then found not to fit)
    append(q, nq, u, r.st, min(r.d, most), r.id);
}

// This block's share of the queue Q (nf rows) onto its list.
__device__ void queue_to_list(const BfsArgs &a, const int4 *vrec, const List &q, unsigned *nq,
                              const int32_t *Q, int64_t nf, int32_t most) {
    if (threadIdx.x == 0) *nq = 0;
    __syncthreads();
    const int64_t b0 = nf * blockIdx.x / gridDim.x, b1 = nf * (blockIdx.x + 1) / gridDim.x;
    for (int64_t i = b0 + threadIdx.x; i < b1; i += kThreads)
        append_row(a, vrec, q, nq, __ldcg(Q + i), most);
    __syncthreads();
}

// The frontier bits of this block's words onto its list; both bitmaps cleared.
__device__ void map_to_list(const BfsArgs &a, const int4 *vrec, const List &q, int cap, unsigned *nq,
                            uint32_t *F, uint32_t *N) {
    if (threadIdx.x == 0) *nq = 0;
    __syncthreads();
    const int64_t w0 = a.nwords * blockIdx.x / gridDim.x, w1 = a.nwords * (blockIdx.x + 1) / gridDim.x;
    for (int64_t w = w0 + threadIdx.x; w < w1; w += kThreads) {
        uint32_t m = __ldcg(F + w);
        N[w] = 0;
        if (m) F[w] = 0;
        for (; m; m &= m - 1) append_row(a, vrec, q, nq, (int32_t)(w * 32 + __ffs(m) - 1), cap);
    }
    __syncthreads();
}

// A row of d > kBigRow edges onto the grid-wide list, in chunks (push_big).
__device__ __forceinline__ void put_big(const BfsArgs &a, unsigned long long *big_slot, int32_t u,
                                        int64_t d) {
    const unsigned long long nch = (unsigned long long)((d + kBigChunk - 1) / kBigChunk);
    const unsigned long long old = atomicAdd(big_slot, (1ull << kBigShift) | nch);
    const int64_t at = (int64_t)(old >> kBigShift);
    a.big[at] = u;
    a.big_base[at] = (int64_t)(old & kBigMask);
}

// The queue entry of row u where the big rows are listed as the queue is made:
// those are in it as ~u, which push_rows passes over.
__device__ __forceinline__ int32_t queued(const BfsArgs &a, unsigned long long *big_slot, int32_t u) {
    const int32_t d = __ldg(a.odeg + u);
    if (d <= kBigRow) return u;
    put_big(a, big_slot, u, d);
    return ~u;
}

// The list back to the frontier bitmap F and, where Q is given, to the queue
// (big_slot, if given: big rows listed).
__device__ void leave_list(const BfsArgs &a, Shared &s, const List &q, unsigned cnt, uint32_t *F,
                           int32_t *Q, unsigned long long *q_slot, unsigned long long *big_slot) {
    const int rows = min((int)(cnt >> kRowShift), kListRows);
    if (Q) {
        if (threadIdx.x == 0 && rows) s.at = atomicAdd(q_slot, (unsigned long long)rows);
        __syncthreads();
    }
    for (int i = threadIdx.x; i < rows; i += kThreads) {
        const int32_t u = q.pos[i];
        if (F) atomicOr(F + (u >> 5), 1u << (u & 31));
        if (Q && ALB_CHECK_POS(s.at + i, a.n, &a.ctl->err))
            Q[s.at + i] = big_slot ? queued(a, big_slot, u) : u;
    }
}

// A list level's edges of one thread: target, its row and the edge's source.
// None of it depends on what the level finds, so it is fetched while the block
// waits at the barrier before.
struct Edges {
    int32_t v[kPer];
    uint32_t ou[kPer];
    RowRec r[kPer];
};

// first: the pass's first edge. (The control warp holds none.)
__device__ __forceinline__ void fetch_edges(const BfsArgs &a, const GridArgs &x, const List &q,
                                            int cap, unsigned cnt, int first, Edges &E) {
    const int nq = (int)(cnt >> kRowShift), ne = (int)(cnt & kEdgeMask);
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int e = first + (int)threadIdx.x + k * kListThreads;
        E.v[k] = -1;
        if (e >= ne || ne > cap || nq > kListRows || threadIdx.x >= kListThreads) continue;
        int j = 0;  // the last row that starts at or before edge e
        static_assert(kListRows <= 2048, "the first step");
        for (int step = 1024; step > 0; step >>= 1)
            if (j + step < nq && q.off[j + step] <= e) j += step;
        E.v[k] = __ldg(a.pcol + (uint32_t)(q.st[j] + (uint32_t)e));
        ALB_CHECK_ID(E.v[k], a.n, -1, &a.ctl->err);
        E.ou[k] = (uint32_t)q.ou[j];
    }
#pragma unroll
    for (int k = 0; k < kPer; k++)
        if (E.v[k] >= 0) E.r[k] = row_rec(a, x.vrec, E.v[k]);
}

// A claim of level L without room in the block's next list (which is then
// taken for over, and left): its place in the next queue and bitmap at once.
__device__ __noinline__ void overflow(const BfsArgs &a, int32_t v, int L) {
    uint32_t *N = (L & 1) ? a.bm0 : a.bm1;
    int32_t *NQ = (L & 1) ? a.q0 : a.q1;
    const unsigned long long at = atomicAdd(&a.ctl->qn[(L + 1) % 3], 1ull);
    if (ALB_CHECK_POS(at, a.n, &a.ctl->err)) NQ[at] = v;
    atomicOr(N + (v >> 5), 1u << (v & 31));
}

// Targets are claimed by the compare-and-swap that moves their level from -1.
__device__ __forceinline__ void claim(const BfsArgs &a, const Edges &E, int L, int32_t (&was)[kPer]) {
#pragma unroll
    for (int k = 0; k < kPer; k++)
        was[k] = E.v[k] >= 0 ? atomicCAS(a.level_pos + E.v[k], -1, L + 1) : 0;
}

// kExact: the words of the visited bitmap that the claims fill are counted. How
// many have an unvisited row is a feature of the learned policy, whose
// directions under ALB_LOOP_GRAPH are those of the host-driven loop. Under
// ALB_LOOP_PERSISTENT they are counted when the lists are left, as that loop
// always did: the words that come back from the atomics, and the sum's way to
// every block, are 10 % of the time of the grid of 2^24.
template <bool kExact>
__device__ __forceinline__ void list_level(const BfsArgs &a, const GridArgs &x, Shared &s,
                                           const Edges &E, const int32_t (&was)[kPer],
                                           const List &nx, unsigned *nnx, int L) {
    unsigned n = 0, mo = 0, mi = 0;
    uint32_t vis[kPer];  // kExact: the claims' words before (full: no claim)
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        vis[k] = kFull;
        if (E.v[k] < 0 || (was[k] != -1 && was[k] != L + 1)) continue;
        // (no look at the parent first: a list's frontier has few edges, and
        // each access to a large graph's arrays is a miss)
        atomicMin(a.parent_pos + E.v[k], E.ou[k]);
        if (was[k] != -1) continue;
        if (kExact) vis[k] = atomicOr(a.vis + (E.v[k] >> 5), 1u << (E.v[k] & 31));
        else atomicOr(a.vis + (E.v[k] >> 5), 1u << (E.v[k] & 31));
        if (!append(nx, nnx, E.v[k], E.r[k].st, min(E.r[k].d, kListRow), E.r[k].id))
            overflow(a, E.v[k], L);
        if (E.r[k].d > kListRow) s.wide = 1;
        n++;
        mo += (unsigned)E.r[k].d;
        if (!x.sym) mi += (unsigned)__ldg(a.ideg + E.v[k]);
    }
    if (!__any_sync(kFull, n != 0)) return;
    n = __reduce_add_sync(kFull, n);
    mo = __reduce_add_sync(kFull, mo);
    if (!x.sym) mi = __reduce_add_sync(kFull, mi);
    unsigned words = 0;
    if (kExact) {
#pragma unroll
        for (int k = 0; k < kPer; k++)
            words += vis[k] != kFull && (vis[k] | (1u << (E.v[k] & 31))) == kFull;
        words = __reduce_add_sync(kFull, words);
    }
    if (lane_id() == 0) {
        if (kExact && words) atomicAdd(&s.cwords, words);
        atomicAdd(&s.cn, n);
        atomicAdd(&s.cmo, mo);
        if (mi) atomicAdd(&s.cmi, mi);
    }
}

// Bitmap words of this block that still have an unvisited row (while lists are
// used they are not watched but under kExact).
__device__ void count_active(const BfsArgs &a, Shared &s) {
    const int64_t w0 = a.nwords * blockIdx.x / gridDim.x, w1 = a.nwords * (blockIdx.x + 1) / gridDim.x;
    unsigned n = 0;
    for (int64_t w = w0 + threadIdx.x; w < w1; w += kThreads) n += __ldcg(a.vis + w) != kFull;
    put_counts(s, n, 0, 0, 0);
}

// ----------------------------------------------------------- top-down levels

// Four pushed edges per lane (v[k] < 0: none): see push_edges4 in bfs.cu. The
// visited words (which no push writes) and the next frontier's are read through
// L1, as fresh as the last barrier's acquire: a bit that another block has set
// since only costs one atomic more. Read from L2 each time, a small graph's few
// lines are what a push of many edges waits for: 33 M edges of 65,000 vertices
// 327 -> 189 us, 8 M 287 -> 122.
__device__ __forceinline__ void push4(const BfsArgs &a, uint32_t *N, const int32_t (&v)[4],
                                      const uint32_t (&ou)[4]) {
    bool live[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
        live[k] = v[k] >= 0 && !((a.vis[v[k] >> 5] >> (v[k] & 31)) & 1u);
    uint32_t cur[4], nw[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        cur[k] = live[k] ? __ldcg(a.parent_pos + v[k]) : 0u;
        nw[k] = live[k] ? N[v[k] >> 5] : ~0u;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (!live[k]) continue;
        const uint32_t bit = 1u << (v[k] & 31);
        if (ou[k] < cur[k]) atomicMin(a.parent_pos + v[k], ou[k]);
        if (!(nw[k] & bit)) atomicOr(N + (v[k] >> 5), bit);
    }
}

// The 128 flattened edges from eb on of a warp's rows: row j's edges start at
// ex[j] (ascending; a row without edges shares its start with the next).
struct WarpRows {
    int64_t ex[32], st[32];
    int32_t ou[32];
};

// Rows of the queue, a few per warp, their edges flattened over the lanes;
// rows longer than kBigRow go on the grid-wide list if they are not on it.
__device__ void push_rows(const BfsArgs &a, WarpRows *wr, const int32_t *Q, int64_t nf,
                          int64_t mf, uint32_t *N, unsigned long long *big_slot) {
    const int lane = lane_id(), wib = threadIdx.x >> 5;
    const int64_t nwarps = (int64_t)gridDim.x * kWarps;
    const int64_t gw = (int64_t)blockIdx.x * kWarps + wib;
    WarpRows &r = wr[wib];
    // rows per warp: all warps busy, and about one 128-edge step each
    const int64_t mean = max((int64_t)1, mf / max(nf, (int64_t)1));
    int G = 1;
    while (G < 32 && ((int64_t)G * nwarps < nf || 2 * G * mean <= 128)) G <<= 1;
    for (int64_t cb = gw * G; cb < nf; cb += nwarps * G) {
        const int64_t i = cb + lane;
        int64_t st = 0, d = 0;
        int32_t ou = 0;
        if (lane < G && i < nf) {
            int32_t u = __ldcg(Q + i);
            if (u >= 0) {
                ALB_CHECK_ID(u, a.n, 0, &a.ctl->err);
                st = __ldg(a.prow + u);
                d = __ldg(a.prow + u + 1) - st;
                ou = __ldg(a.perm + u);
            }
            if (d > kBigRow) {
                put_big(a, big_slot, u, d);
                d = 0;
            }
        }
        const int64_t inc = warp_inclusive_scan(d);
        const int64_t T = __shfl_sync(kFull, inc, 31);
        r.ex[lane] = inc - d;
        r.st[lane] = st;
        r.ou[lane] = ou;
        __syncwarp();
        for (int64_t e0 = lane; e0 < T; e0 += 128) {
            int32_t v[4];
            uint32_t ou4[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int64_t e = e0 + 32 * k;
                v[k] = -1;
                ou4[k] = 0;
                if (e < T) {
                    int j = 0;
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1)
                        if (r.ex[j + step] <= e) j += step;
                    v[k] = __ldg(a.pcol + r.st[j] + (e - r.ex[j]));
                    ALB_CHECK_ID(v[k], a.n, -1, &a.ctl->err);
                    ou4[k] = (uint32_t)r.ou[j];
                }
            }
            push4(a, N, v, ou4);
        }
        __syncwarp();
    }
}

// The big rows' kBigChunk-edge chunks, a contiguous run per warp.
__device__ void push_big(const BfsArgs &a, uint32_t *N, unsigned long long ctr) {
    const int64_t nbig = (int64_t)(ctr >> kBigShift), total = (int64_t)(ctr & kBigMask);
    const int lane = lane_id();
    const int64_t nwarps = (int64_t)gridDim.x * kWarps;
    const int64_t gw = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    const int64_t k0 = total * gw / nwarps, k1 = total * (gw + 1) / nwarps;
    if (k0 >= k1) return;
    int64_t lo = 0, hi = nbig - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (__ldcg(a.big_base + mid) <= k0) lo = mid;
        else hi = mid - 1;
    }
    int64_t base = 0, next = k0, st = 0, d = 0;
    uint32_t ou = 0;
    lo--;
    for (int64_t k = k0; k < k1; k++) {
        while (k >= next) {  // the run crosses into the next long row
            lo++;
            base = __ldcg(a.big_base + lo);
            next = lo + 1 < nbig ? __ldcg(a.big_base + lo + 1) : total;
            const int32_t u = __ldcg(a.big + lo);
            st = __ldg(a.prow + u);
            d = __ldg(a.prow + u + 1) - st;
            ou = (uint32_t)__ldg(a.perm + u);
        }
        const int64_t e = (k - base) * kBigChunk + lane;
        int32_t v[4];
        const uint32_t ou4[4] = {ou, ou, ou, ou};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[q] = e + 32 * q < d ? __ldg(a.pcol + st + e + 32 * q) : -1;
            if (v[q] >= 0) ALB_CHECK_ID(v[q], a.n, -1, &a.ctl->err);
        }
        push4(a, N, v, ou4);
    }
}

// The set bits of 32 words (lane l holds word l) as row numbers 0 .. 1023 in
// the warp's buffer; returns how many.
__device__ __forceinline__ int list_bits(uint16_t *buf, uint32_t m) {
    const int lane = lane_id();
    const int inc = warp_inclusive_scan(__popc(m));
    int at = inc - __popc(m);
    for (; m; m &= m - 1) buf[at++] = (uint16_t)(lane * 32 + __ffs(m) - 1);
    __syncwarp();
    return __shfl_sync(kFull, inc, 31);
}

// (sym, here and below: a row's two lengths are one number, loaded once: 1 to
// 3 % of a search.)
// After the pushes: the old frontier's bits are cleared over its queue, the
// new frontier N goes to the next queue with levels, visited bits and counters.
__device__ void finish_push(const BfsArgs &a, Shared &s, uint16_t (*rows)[1024], const int32_t *Q,
                            int64_t nf, uint32_t *F, const uint32_t *N, int32_t *NQ,
                            unsigned long long *nq_slot, int L, bool sym) {
    const int lane = lane_id(), wib = threadIdx.x >> 5;
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * kThreads;
    for (int64_t i = tid; i < nf; i += nth) {
        const int32_t u = __ldcg(Q + i);
        F[(u < 0 ? ~u : u) >> 5] = 0;
    }
    unsigned cn = 0, full = 0;
    unsigned long long mo = 0, mi = 0;
    for (int64_t w0 = tid & ~31ll; w0 < a.nwords; w0 += nth) {
        const int64_t w = w0 + lane;
        const uint32_t m = w < a.nwords ? __ldcg(N + w) : 0u;
        if (!__any_sync(kFull, m != 0)) continue;
        if (m) {
            const uint32_t old = __ldcg(a.vis + w);
            a.vis[w] = old | m;
            full += old != kFull && (old | m) == kFull;
        }
        const int tot = list_bits(rows[wib], m);
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(nq_slot, (unsigned long long)tot);
        base = __shfl_sync(kFull, base, 0);
        for (int i = lane; i < tot; i += 32) {
            const int32_t p = (int32_t)(w0 * 32) + rows[wib][i];
            if (ALB_CHECK_POS((int64_t)base + i, a.n, &a.ctl->err)) NQ[base + i] = p;
            a.level_pos[p] = L + 1;
            const int32_t od = __ldg(a.odeg + p), id = sym ? od : __ldg(a.ideg + p);
            cn++;
            mo += (unsigned long long)od;
            mi += (unsigned long long)id;
        }
        __syncwarp();
    }
    put_counts(s, cn, mo, mi, full);
}

// Frontier bitmap to queue (big rows listed), next bitmap cleared.
__device__ void map_to_queue(const BfsArgs &a, uint16_t (*rows)[1024], const uint32_t *F,
                             uint32_t *N, int32_t *Q, unsigned long long *q_slot,
                             unsigned long long *big_slot) {
    const int lane = lane_id(), wib = threadIdx.x >> 5;
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * kThreads;
    for (int64_t w0 = tid & ~31ll; w0 < a.nwords; w0 += nth) {
        const int64_t w = w0 + lane;
        uint32_t m = 0;
        if (w < a.nwords) {
            m = __ldcg(F + w);
            N[w] = 0;
        }
        if (!__any_sync(kFull, m != 0)) continue;
        const int tot = list_bits(rows[wib], m);
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(q_slot, (unsigned long long)tot);
        base = __shfl_sync(kFull, base, 0);
        for (int i = lane; i < tot; i += 32)
            if (ALB_CHECK_POS((int64_t)base + i, a.n, &a.ctl->err))
                Q[base + i] = queued(a, big_slot, (int32_t)(w0 * 32) + rows[wib][i]);
        __syncwarp();
    }
}

// ---------------------------------------------------------- bottom-up levels

// First frontier source among sources [st, en) of one long row (-1: none).
__device__ __forceinline__ int32_t scan_long(const BfsArgs &a, const uint32_t *F, int64_t st,
                                             int64_t en) {
    const int lane = lane_id();
    for (int64_t e0 = st; e0 < en; e0 += 128) {
        int32_t c[4];
        uint32_t f[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t e = e0 + 32 * u + lane;
            c[u] = e < en ? __ldg(a.lcol + e) : -1;
            if (c[u] >= 0) ALB_CHECK_ID(c[u], a.n, -1, &a.ctl->err);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) f[u] = c[u] >= 0 ? __ldcg(F + (c[u] >> 5)) : 0u;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const unsigned m = __ballot_sync(kFull, c[u] >= 0 && ((f[u] >> (c[u] & 31)) & 1u));
            if (m) return __shfl_sync(kFull, c[u], __ffs(m) - 1);
        }
    }
    return -1;
}

// Unvisited long rows, a warp each over the first kLongChunk sources; rows
// with more and no hit there go on the grid-wide list (pull_long_tail). A
// hit's parent goes to parent_pos, where the slice pass finds it. Counts (n)
// the unvisited ones.
__device__ void pull_long(const BfsArgs &a, Shared &s, const uint32_t *F,
                          unsigned long long *big_slot) {
    const int lane = lane_id();
    const int64_t nwarps = (int64_t)gridDim.x * kWarps;
    const int64_t gw = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    unsigned seen = 0;
    for (int64_t i0 = gw; i0 < a.nlong; i0 += 32 * nwarps) {
        const int64_t i = i0 + lane * nwarps;
        int32_t p_l = 0;
        bool todo_l = false;
        if (i < a.nlong) {
            p_l = __ldg(a.lrow + i);
            todo_l = !((__ldcg(a.vis + (p_l >> 5)) >> (p_l & 31)) & 1u);
        }
        unsigned todo = __ballot_sync(kFull, todo_l);
        seen += lane == 0 ? __popc(todo) : 0;
        for (; todo; todo &= todo - 1) {
            const int b = __ffs(todo) - 1;
            const int32_t p = __shfl_sync(kFull, p_l, b);
            const int64_t r = i0 + b * nwarps;
            const int64_t st = __ldg(a.lptr + r), en = __ldg(a.lptr + r + 1);
            const int64_t head = min(en, st + kLongChunk);
            const int32_t found = scan_long(a, F, st, head);
            if (lane != 0) continue;
            if (found >= 0) {
                a.parent_pos[p] = (uint32_t)__ldg(a.perm + found);
            } else if (head < en) {
                const unsigned long long nch =
                    (unsigned long long)((en - head + kLongChunk - 1) / kLongChunk);
                const unsigned long long old = atomicAdd(big_slot, (1ull << kBigShift) | nch);
                const int64_t at = (int64_t)(old >> kBigShift);
                a.big[at] = (int32_t)r;
                a.big_base[at] = (int64_t)(old & kBigMask);
            }
        }
    }
    put_counts(s, seen, 0, 0, 0);
}

__device__ void pull_long_tail(const BfsArgs &a, const uint32_t *F, unsigned long long ctr) {
    const int64_t nrows = (int64_t)(ctr >> kBigShift), total = (int64_t)(ctr & kBigMask);
    const int64_t nwarps = (int64_t)gridDim.x * kWarps;
    for (int64_t k = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5); k < total; k += nwarps) {
        int64_t lo = 0, hi = nrows - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if (__ldcg(a.big_base + mid) <= k) lo = mid;
            else hi = mid - 1;
        }
        const int32_t r = __ldcg(a.big + lo);
        const int64_t st = __ldg(a.lptr + r) + (1 + k - __ldcg(a.big_base + lo)) * kLongChunk;
        const int64_t en = min(__ldg(a.lptr + r + 1), st + kLongChunk);
        const int32_t found = scan_long(a, F, st, en);
        if (found >= 0 && lane_id() == 0)
            atomicMin(a.parent_pos + __ldg(a.lrow + r), (uint32_t)__ldg(a.perm + found));
    }
}

// The group's first source in the frontier (-1: none), f0 .. f3 its frontier words.
__device__ __forceinline__ int32_t first_hit(const int4 &c, uint32_t f0, uint32_t f1, uint32_t f2,
                                             uint32_t f3) {
    if ((f0 >> (c.x & 31)) & 1u) return c.x;
    if ((f1 >> (c.y & 31)) & 1u) return c.y;
    if ((f2 >> (c.z & 31)) & 1u) return c.z;
    if ((f3 >> (c.w & 31)) & 1u) return c.w;
    return -1;
}
template <bool kStaged>
__device__ __forceinline__ int32_t test_group(const uint32_t *F, const int4 &c) {
    auto word = [&](int32_t v) { return kStaged ? F[v >> 5] : __ldcg(F + (v >> 5)); };
    const uint32_t f0 = word(c.x), f1 = word(c.y), f2 = word(c.z), f3 = word(c.w);
    return first_hit(c, f0, f1, f2, f3);
}

// Word shape: a warp takes runs of words from the level's counter, lane l's
// visited word loaded a run ahead, and pulls two words at a time, lane per
// row. Runs shrink towards the level's end, from a quarter of what an even
// split gives a warp (32 words at most) to 4: with equal runs of 26 words half
// of the warps of R-MAT scale 24 had nothing left for the last fifth of the
// level. A uniform random graph of 2^24 1,025 -> 975 us in all, R-MAT of
// 2^23 255 -> 243, scale 24 from a leaf 379 -> 367 and from a hub 614 -> 610;
// equal runs of 8: 985, 248, 381, 643. Bound: the gathers of frontier bits, an
// address per clock and SM (2^22 vertices of mean degree 8: 31 M in 108 us).
// kScan (pull_scan): rows are mostly read to their ends, and a wide slice's step
// is a column load and two words' frontier tests one after the other; there both
// words' frontier words are requested before either is tested, one round trip a
// step instead of two. (Everywhere it costs registers that the kernel has not
// got: a hub's search of R-MAT scale 22 146 -> 156 us.)
template <bool kStaged, bool kScan>
__device__ __forceinline__ void pull_words(const BfsArgs &a, Shared &s, const uint32_t *F, uint32_t *N, int L,
                           unsigned long long *ctr, bool sym) {
    constexpr int kW = 2;
    const int lane = lane_id();
    const int32_t C = a.C, log2C = a.log2C;
    const int64_t warps = (int64_t)gridDim.x * kWarps;
    const int most = (int)min((int64_t)32, max((int64_t)kW, a.nwords / (warps * 4))), least = min(4, most);
    int64_t nxt = 0;
    int run = 0;  // words of the run at nxt
    const uint64_t pol = l2_evict_first();
    unsigned cn = 0, full = 0;
    unsigned long long mo = 0, mi = 0;
    // the next run, and its visited words
    auto grab = [&]() {
        run = max(least, (int)min((int64_t)most, (a.nwords - nxt) / (warps * 6)));
        unsigned long long v = 0;
        if (lane == 0) v = atomicAdd(ctr, (unsigned long long)run);
        nxt = (int64_t)__shfl_sync(kFull, v, 0);
        return lane < run && nxt + lane < a.nwords ? __ldcg(a.vis + nxt + lane) : kFull;
    };
    uint32_t vcur = grab();
    int64_t cur = nxt;
    int rcur = run;
    uint32_t vnxt = grab();
    while (cur < a.nwords) {
        const bool valid = lane < rcur && cur + lane < a.nwords;
        if (valid && vcur == kFull) N[cur + lane] = 0;
        unsigned todo = __ballot_sync(kFull, valid && vcur != kFull);
        const int64_t base_w = cur;
        const uint32_t vrun = vcur;
        cur = nxt;
        vcur = vnxt;
        rcur = run;
        if (cur < a.nwords) vnxt = grab();
        while (todo) {
            int qs[kW], nr = 0;
#pragma unroll
            for (int t = 0; t < kW; t++) {
                qs[t] = todo ? __ffs(todo) - 1 : qs[0];
                nr += todo != 0;
                todo &= todo - 1;
            }
            uint32_t vis[kW];
            int32_t p[kW], ng[kW], found[kW];
            bool act[kW], maybe_long[kW];
            const int4 *cp[kW];
            int4 c[kW];
            int64_t so[kW];
#pragma unroll
            for (int t = 0; t < kW; t++) {
                vis[t] = __shfl_sync(kFull, vrun, qs[t]);
                p[t] = (int32_t)((base_w + qs[t]) * 32) + lane;
                act[t] = t < nr && !((vis[t] >> lane) & 1u);
                const int32_t sl = (act[t] ? p[t] : 0) >> log2C;
                ng[t] = act[t] ? (__ldg(a.width + sl) + 3) >> 2 : 0;
                so[t] = act[t] ? __ldg(a.slice_off + sl) : 0;
                found[t] = -1;
            }
#pragma unroll
            for (int t = 0; t < kW; t++) {
                cp[t] = a.col4 + (so[t] >> 2) + (p[t] & (C - 1));
                c[t] = make_int4(p[t], p[t], p[t], p[t]);
                if (ng[t] > 0) c[t] = ld_stream(cp[t], pol);
            }
            // an unvisited row whose first entry is padding is a long row
#pragma unroll
            for (int t = 0; t < kW; t++) maybe_long[t] = act[t] && c[t].x == p[t];
            for (int32_t j = 0;; j++) {
                bool any = false;
#pragma unroll
                for (int t = 0; t < kW; t++) {
                    act[t] = act[t] && j < ng[t];
                    any = any || act[t];
                }
                if (!__any_sync(kFull, any)) break;
                int4 nx[kW];
#pragma unroll
                for (int t = 0; t < kW; t++) {
                    nx[t] = make_int4(p[t], p[t], p[t], p[t]);
                    if (act[t] && j + 1 < ng[t]) nx[t] = ld_stream(cp[t] + (int64_t)(j + 1) * C, pol);
                }
                uint32_t f[kW][4];
                if (kScan) {
#pragma unroll
                    for (int t = 0; t < kW; t++) {
                        if (!act[t]) continue;
                        ALB_CHECK_ID4(c[t], a.nwords * 32, p[t], &a.ctl->err);
                        f[t][0] = F[c[t].x >> 5], f[t][1] = F[c[t].y >> 5];
                        f[t][2] = F[c[t].z >> 5], f[t][3] = F[c[t].w >> 5];
                    }
                }
#pragma unroll
                for (int t = 0; t < kW; t++) {
                    if (!act[t]) continue;
                    // padding is the row itself, never in the frontier, and
                    // ends the row: the first hit is the smallest source
                    if (kScan) {
                        found[t] = first_hit(c[t], f[t][0], f[t][1], f[t][2], f[t][3]);
                    } else {
                        ALB_CHECK_ID4(c[t], a.nwords * 32, p[t], &a.ctl->err);
                        found[t] = test_group<kStaged>(F, c[t]);
                    }
                    act[t] = found[t] < 0 && c[t].w != p[t];
                    c[t] = nx[t];
                }
            }
#pragma unroll
            for (int t = 0; t < kW; t++) {
                if (t >= nr) break;
                bool reached = found[t] >= 0, by_long = false;
                if (maybe_long[t] && !reached && a.nlong)
                    by_long = reached = __ldcg(a.parent_pos + p[t]) != kFull;
                const unsigned nm = __ballot_sync(kFull, reached);
                if (lane == 0) {
                    const int64_t w = base_w + qs[t];
                    N[w] = nm;
                    if (nm) {
                        a.vis[w] = vis[t] | nm;
                        full += vis[t] != kFull && (vis[t] | nm) == kFull;
                    }
                }
                if (reached) {
                    a.level_pos[p[t]] = L + 1;
                    if (!by_long) a.parent_pos[p[t]] = (uint32_t)__ldg(a.perm + found[t]);
                    const int32_t od = __ldg(a.odeg + p[t]), id = sym ? od : __ldg(a.ideg + p[t]);
                    cn++;
                    mo += (unsigned long long)od;
                    mi += (unsigned long long)id;
                }
            }
        }
    }
    put_counts(s, cn, mo, mi, full);
}

// The word shape for a frontier that few rows have a source in, as a function of
// its own: the kernel around it keeps its registers.
__device__ __noinline__ void pull_scan(BfsArgs a, const uint32_t *F, uint32_t *N, int L,
                                       unsigned long long *ctr, bool sym) {
    ALB_GRID_SHARED;
    (void)pool;
    pull_words<false, true>(a, s, F, N, L, ctr, sym);
}

// Row shape: the unvisited rows of 32 words, dealt out to the lanes.
__device__ void pull_rows(const BfsArgs &a, Shared &s, uint16_t (*rows)[1024], const uint32_t *F,
                          uint32_t *N, int L, bool sym) {
    const int lane = lane_id(), wib = threadIdx.x >> 5;
    const int32_t C = a.C, log2C = a.log2C;
    unsigned cn = 0, full = 0;
    unsigned long long mo = 0, mi = 0;
    // fewer words a step where that keeps more warps busy
    const int64_t nwarps = (int64_t)gridDim.x * kWarps;
    const int span = (int)min((int64_t)32, max((int64_t)1, a.nwords / nwarps));
    for (int64_t w0 = ((int64_t)blockIdx.x * kWarps + wib) * span; w0 < a.nwords;
         w0 += nwarps * span) {
        const int64_t w = w0 + lane;
        const bool valid = lane < span && w < a.nwords;
        const uint32_t vis = valid ? __ldcg(a.vis + w) : kFull;
        uint32_t next = 0;  // lane l: the reached rows of word l
        const bool some = __any_sync(kFull, vis != kFull);
        const int tot = some ? list_bits(rows[wib], ~vis) : 0;
        for (int i0 = 0; i0 < tot; i0 += 32) {
            const int i = i0 + lane;
            int32_t p = 0, found = -1;
            bool reached = false;
            int r = 0;
            if (i < tot) {
                r = rows[wib][i];
                p = (int32_t)(w0 * 32) + r;
                const int32_t sl = p >> log2C;
                const int32_t ng = (__ldg(a.width + sl) + 3) >> 2;
                const int4 *cp = a.col4 + (__ldg(a.slice_off + sl) >> 2) + (p & (C - 1));
                int4 c = make_int4(p, p, p, p);
                if (ng > 0) c = __ldcs(cp);
                bool by_long = false;
                if (c.x == p) {  // a long row: the pass over them has run
                    by_long = a.nlong && __ldcg(a.parent_pos + p) != kFull;
                } else {
                    for (int32_t j = 0; j < ng; j++) {
                        if (j) c = __ldcs(cp + (int64_t)j * C);
                        ALB_CHECK_ID4(c, a.nwords * 32, p, &a.ctl->err);
                        found = test_group<false>(F, c);
                        if (found >= 0 || c.w == p) break;
                    }
                }
                reached = by_long || found >= 0;
                if (reached) {
                    a.level_pos[p] = L + 1;
                    if (!by_long) a.parent_pos[p] = (uint32_t)__ldg(a.perm + found);
                    const int32_t od = __ldg(a.odeg + p), id = sym ? od : __ldg(a.ideg + p);
                    cn++;
                    mo += (unsigned long long)od;
                    mi += (unsigned long long)id;
                }
            }
            // every reached row's bit to the lane that holds its word
            __syncwarp();
            for (unsigned m = __ballot_sync(kFull, reached); m; m &= m - 1) {
                const int rr = __shfl_sync(kFull, r, __ffs(m) - 1);
                if ((rr >> 5) == lane) next |= 1u << (rr & 31);
            }
        }
        if (valid) {
            N[w] = next;
            if (next) {
                a.vis[w] = vis | next;
                full += (vis | next) == kFull;
            }
        }
        __syncwarp();
    }
    put_counts(s, cn, mo, mi, full);
}

// Copies the frontier bitmap into shared memory: one bulk copy on an mbarrier
// (parity: how often it completed before). Waits end after a.bulk_ns.
__device__ bool stage_frontier(const BfsArgs &a, Shared &s, uint32_t *dst, const uint32_t *F,
                               unsigned parity) {
    const uint32_t bytes = (uint32_t)(((a.nwords * 4) + 15) & ~15ll);
    if (threadIdx.x == 0) {
        // the bitmap and the buffer were last accessed the ordinary way
        asm volatile("fence.proxy.async;" ::: "memory");
        mbar_expect_tx(&s.bar, bytes);
        bulk_g2s(dst, F, bytes, &s.bar);
    }
    const uint64_t t0 = globaltimer_ns();
    bool ok = true;
    while (!mbar_try_wait(&s.bar, parity)) {
        if (globaltimer_ns() - t0 > a.bulk_ns) {
            if (threadIdx.x == 0) atomicExch(&a.ctl->err, ALB_ERR_TIMEOUT);
            ok = false;
            // the copy may still be writing here: stay until it lands
            const uint64_t t1 = globaltimer_ns();
            while (!mbar_try_wait(&s.bar, parity) && globaltimer_ns() - t1 < 4 * a.bulk_ns)
                __nanosleep(1024);
            break;
        }
    }
    return __syncthreads_and(ok);
}

// ------------------------------------------------------------------ the loop

// The next level's direction and form from the traversal's state (one warp,
// all lanes alike).
__device__ __forceinline__ void next_level(Shared &s, const BfsCtl &c) {
    int dir;
    if (s.learned && s.mlp.loaded()) {
        float f[kMlpIn];
        level_features_warp(c, f);
        dir = s.mlp.select(f);
    } else {
        dir = rule_dir(c);
    }
    // lists: no block may hold more than kListRows rows or s.cap edges. From lists, the
    // last barrier said whether one does; from a queue or bitmap, the whole
    // frontier fits one block, or (queue) its equal shares should fit with
    // room to spare, which is checked once they are laid out -- as when lists
    // that grew apart are dealt out anew.
    const int64_t nb = gridDim.x;
    const bool listed = s.form == kList;
    const bool all_fit = c.mf <= s.cap && c.nf <= kListRows;
    const bool shares = s.max_out <= kListRow && 4 * c.mf <= 3 * s.cap * nb &&
                        4 * c.nf <= 3 * kListRows * nb;
    const bool td = dir == ALB_DIR_TOPDOWN && s.m_out <= UINT32_MAX && s.max_out < (1 << 20);
    const bool even = listed && shares && (s.over || (s.uneven && 2 * c.mf <= s.cap * nb));
    const bool lists = td && (listed ? !s.over || even : all_fit || (s.form == kQueue && shares));
    if (lane_id() == 0) {
        s.dir = dir;
        s.even = even;
        s.lists = lists;
        s.nq[(c.level + 1) & 1] = 0;
        // row shape: under half of the rows of the words that have any unvisited
        // (at 10 of 32 a uniform random graph of 2^24 takes 1,145 us, at 16 1,081;
        // at 24 one of 2^22 364 -> 420)
        s.sparse = c.nu < 16 * c.active_words;
        // few rows have a source in the frontier: under a 32nd of the unvisited
        // rows' entries point into it (bottom-up from a leaf of R-MAT of 2^22
        // 1,344 -> 960 us, of 2^21 890 -> 620)
        s.scan = 32 * c.mf < c.mu;
    }
}

// The level's end (one warp): counters rolled over, the next level decided.
__device__ __noinline__ void end_level(int next_form) {
    ALB_GRID_SHARED;
    (void)pool;
    BfsCtl c;
    c.policy = s.c.policy;
    c.alpha = s.c.alpha;
    c.beta = s.c.beta;
    c.n = s.c.n;
    c.nwords = s.c.nwords;
    c.feat_mean_deg = s.c.feat_mean_deg;
    c.feat_skew = s.c.feat_skew;
    c.prev_nf = s.c.nf;
    c.nf = (int64_t)s.n;
    c.mf = (int64_t)s.mo;
    c.nu = s.c.nu - (int64_t)s.n;
    c.mu = s.c.mu - (int64_t)s.mi;
    c.active_words = s.c.active_words - (int64_t)s.full;
    c.reached = s.c.reached + (int64_t)s.n;
    c.edges = s.c.edges + (int64_t)s.mo;
    c.prev_dir = s.dir;
    c.levels_td = s.c.levels_td + (s.dir == ALB_DIR_TOPDOWN);
    c.levels_bu = s.c.levels_bu + (s.dir != ALB_DIR_TOPDOWN);
    c.level = s.c.level + 1;
    c.done = s.n == 0 || c.level >= s.level_cap;
    __syncwarp();
    if (lane_id() == 0) {
        BfsCtl &o = s.c;
        o.prev_nf = c.prev_nf;
        o.nf = c.nf;
        o.mf = c.mf;
        o.nu = c.nu;
        o.mu = c.mu;
        o.active_words = c.active_words;
        o.reached = c.reached;
        o.edges = c.edges;
        o.prev_dir = c.prev_dir;
        o.levels_td = c.levels_td;
        o.levels_bu = c.levels_bu;
        o.level = c.level;
        o.done = c.done;
        s.form = next_form;
    }
    __syncwarp();
    next_level(s, c);
}

// The next level's counters (read last at level L - 2, by blocks that have all
// passed a barrier since) and the queue cursor after it.
__device__ __forceinline__ void clear_next(const BfsArgs &a, const GridArgs &x, int L) {
    if (blockIdx.x == 0 && threadIdx.x < 16) {
        const int k = (L + 1) % 3;
        x.slots->acc[k][threadIdx.x] = 0;
        if (threadIdx.x == 0) {
            x.slots->word[k][0] = 0;
            a.ctl->nbig[k] = a.ctl->work[k] = 0;
            a.ctl->qn[(L + 2) % 3] = 0;
        }
    }
}

// kScan: frontiers too large to stage may be pulled while they are small, as
// under the bottom-up policy (pull_scan; the call alone, where it is never made,
// costs the grid of 2^24 8 %).
template <bool kExact, bool kScan>
__global__ void __launch_bounds__(kThreads, 1) k_bfs_grid(BfsArgs a, InitParams in, GridArgs x) {
    ALB_GRID_SHARED;
    __shared__ WarpRows wr[kWarps];
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * kThreads;
    const int32_t rp = __ldg(a.inv + in.root);
    const int32_t r_out = __ldg(a.odeg + rp), r_in = __ldg(a.ideg + rp);
    const uint32_t rbit = 1u << (rp & 31), rold = __ldg(a.vinit + (rp >> 5));
    // initial state (the arrays are padded to whole 16 bytes or tails are
    // written one by one)
    for (int64_t i = tid; i < a.n / 4; i += nth) {
        reinterpret_cast<int4 *>(a.level_pos)[i] = make_int4(-1, -1, -1, -1);
        reinterpret_cast<int4 *>(a.parent_pos)[i] = make_int4(-1, -1, -1, -1);
    }
    for (int64_t p = (a.n & ~3ll) + tid; p < a.n; p += nth) {
        a.level_pos[p] = -1;
        a.parent_pos[p] = kFull;
    }
    for (int64_t w = tid; w < a.nwords; w += nth) {
        a.vis[w] = __ldg(a.vinit + w) | (w == (rp >> 5) ? rbit : 0u);
        a.bm0[w] = w == (rp >> 5) ? rbit : 0u;
        a.bm1[w] = 0;
    }
    const bool learned = in.policy == ALB_POLICY_LEARNED && a.mlp;
    if (learned) s.mlp.load(a.mlp);
    for (int i = threadIdx.x; i < (int)(sizeof(BfsCtl) / 4); i += kThreads)
        reinterpret_cast<uint32_t *>(&s.c)[i] = 0;
    if (threadIdx.x < kWarps) s.warp[threadIdx.x] = Counts{0, 0, 0, 0};
    __syncthreads();
    if (threadIdx.x == 0) {
        s.form = kQueue;
        s.max_out = x.max_out;
        s.m_out = x.m_out;
        s.level_cap = in.level_cap;
        s.learned = learned;
        s.cap = x.list_cap;
        s.cn = s.cmo = s.cmi = s.wide = s.cwords = 0;
        mbar_init(&s.bar, 1);
        BfsCtl &c = s.c;
        c.prev_dir = c.dir = -1;
        c.policy = in.policy;
        c.alpha = in.alpha;
        c.beta = in.beta;
        c.n = a.n;
        c.nwords = a.nwords;
        c.nf = c.reached = 1;
        c.mf = c.edges = r_out;
        c.nu = in.n_live - (r_in > 0 ? 1 : 0);
        c.mu = in.m_in - r_in;
        c.active_words = in.active0 - ((rold != kFull && (rold | rbit) == kFull) ? 1 : 0);
        c.feat_mean_deg = in.mean_deg;
        c.feat_skew = in.skew;
        if (blockIdx.x == 0) {
            a.q0[0] = rp;
            for (int k = 0; k < 3; k++) a.ctl->nbig[k] = a.ctl->work[k] = a.ctl->qn[k] = 0;
            for (int k = 0; k < (int)(sizeof(GridSlots) / 8); k++)
                reinterpret_cast<unsigned long long *>(x.slots)[k] = 0;
            a.ctl->err = 0;
        }
    }
    bool ok = barrier(a, s, -1);
    if (ok && tid == rp % nth) {  // (after the clearing, before level 0 ends)
        a.level_pos[rp] = 0;
        a.parent_pos[rp] = (uint32_t)in.root;
    }
    const bool ctl = (threadIdx.x >> 5) == kCtl;
    if (ctl) next_level(s, s.c);
    const int cap = x.list_cap;
    __syncthreads();
    unsigned staged = 0;             // bulk copies completed
    int64_t long_left = a.nlong;     // upper bound of the unvisited long rows
    while (ok) {
        const int L = s.c.level, dir = s.dir;
        int form = s.form;
        bool lists = s.lists;
        const bool even = s.even;
        const int64_t nf = s.c.nf, mf = s.c.mf;
        uint32_t *F = (L & 1) ? a.bm1 : a.bm0, *N = (L & 1) ? a.bm0 : a.bm1;
        int32_t *Q = (L & 1) ? a.q1 : a.q0, *NQ = (L & 1) ? a.q0 : a.q1;
        unsigned long long *big = &a.ctl->nbig[L % 3], *work = &a.ctl->work[L % 3],
                           *nqn = &a.ctl->qn[(L + 1) % 3];
        clear_next(a, x, L);
        unsigned long long *acc = x.slots->acc[L % 3];
        const int par = L & 1;
        int next_form;
        if (lists && form == kMap) {
            map_to_list(a, x.vrec, list_at(pool, par), cap, &s.nq[par], F, N);
        } else if (lists && (form == kQueue || even)) {
            const List q = list_at(pool, par);
            if (even) {  // back to a queue first
                leave_list(a, s, q, s.nq[par], F, Q, &a.ctl->qn[L % 3], nullptr);
                form = kQueue;
                if (!(ok = barrier(a, s, L))) break;
            }
            const bool all = mf <= cap && nf <= kListRows;
            queue_to_list(a, x.vrec, q, &s.nq[par], Q, nf, all ? cap : kListRow);
            const unsigned k = s.nq[par];
            if (!all) {  // does every block's share fit?
                const bool no = (k & kEdgeMask) > (unsigned)cap || (k >> kRowShift) > (unsigned)kListRows;
                put_counts(s, threadIdx.x == 0 && no, 0, 0, 0);
                if (!(ok = barrier(a, s, L, acc + kSumFits))) break;
                lists = s.n == 0;
            }
            // both bitmaps are empty while lists are used
            if (lists)
                for (unsigned i = threadIdx.x; i < (k >> kRowShift); i += kThreads)
                    F[q.pos[i] >> 5] = 0;
        }
        if (lists) {
            // list levels until another form is due; while the control warp
            // waits and decides, the others fetch the next level's edges
            Edges E;
            fetch_edges(a, x, list_at(pool, par), cap, s.nq[par], 0, E);
            for (int l = L;;) {
                const int p = l & 1;
                const List cur = list_at(pool, p), nx = list_at(pool, p ^ 1);
                const unsigned cnt = s.nq[p];
                for (int e = 0;;) {
                    int32_t was[kPer];
                    claim(a, E, l, was);
                    const Edges now = E;
                    e += kListPass;
                    const bool more = e < (int)(cnt & kEdgeMask);
                    if (more) fetch_edges(a, x, cur, cap, cnt, e, E);
                    list_level<kExact>(a, x, s, now, was, nx, &s.nq[p ^ 1], l);
                    if (!more) break;
                }
                __syncthreads();
                if (ctl) {
                    const bool k = list_barrier<kExact>(a, x, s, l, x.slots->word[l % 3],
                                                        x.slots->acc[l % 3]);
                    if (lane_id() == 0) s.ok = k;
                    __syncwarp();
                    if (k) end_level(kList);
                } else {
                    fetch_edges(a, x, nx, cap, s.nq[p ^ 1], 0, E);
                }
                __syncthreads();
                ok = s.ok;
                if (!ok || s.c.done || !s.lists || s.even) break;
                l++;
                clear_next(a, x, l);
            }
            if (!ok || s.c.done) break;
            continue;
        } else {
            if (form == kList) {
                leave_list(a, s, list_at(pool, par), s.nq[par], F, dir == ALB_DIR_TOPDOWN ? Q : nullptr,
                           &a.ctl->qn[L % 3], big);
                count_active(a, s);
                if (!(ok = barrier(a, s, L, acc + kSumActive, big))) break;
                if (threadIdx.x == 0) s.c.active_words = (int64_t)s.n;
            }
            if (dir == ALB_DIR_TOPDOWN) {
                if (form == kMap) {
                    map_to_queue(a, pool.rows, F, N, Q, &a.ctl->qn[L % 3], big);
                    if (!(ok = barrier(a, s, L, nullptr, big))) break;
                }
                // the big rows are known beforehand where the queue was made
                // in this level: then they are pushed beside the others, a
                // barrier and a phase of latency less (R-MAT of 10^6 vertices:
                // 119 -> 114 us in all). finish_push does not list them: most
                // of its queues are of levels that turn out bottom-up.
                const bool known = form != kQueue;
                push_rows(a, wr, Q, nf, mf, N, big);
                if (known && s.nbig) push_big(a, N, s.nbig);
                if (!(ok = barrier(a, s, L, nullptr, known ? nullptr : big))) break;
                if (!known && s.nbig) {
                    push_big(a, N, s.nbig);
                    if (!(ok = barrier(a, s, L))) break;
                }
                finish_push(a, s, pool.rows, Q, nf, F, N, NQ, nqn, L, x.sym);
                next_form = kQueue;
            } else {
                if (long_left) {
                    pull_long(a, s, F, big);
                    if (!(ok = barrier(a, s, L, acc + kSumLong, big))) break;
                    long_left = (int64_t)s.n;
                    if (s.nbig) {
                        pull_long_tail(a, F, s.nbig);
                        if (!(ok = barrier(a, s, L))) break;
                    }
                }
                if (s.sparse) {
                    pull_rows(a, s, pool.rows, F, N, L, x.sym);
                } else if (a.nwords * 4 <= kStageMax) {
                    if (!(ok = stage_frontier(a, s, pool.stage, F, staged++ & 1))) break;
                    pull_words<true, false>(a, s, pool.stage, N, L, work, x.sym);
                } else if (kScan && s.scan) {
                    pull_scan(a, F, N, L, work, x.sym);
                } else {
                    pull_words<false, false>(a, s, F, N, L, work, x.sym);
                }
                next_form = kMap;
            }
        }
        if (!(ok = barrier(a, s, L, acc + kSumLevel))) break;
        if (ctl) end_level(next_form);
        __syncthreads();
        if (s.c.done) break;
    }
    if (tid == 0) {
        x.result->level = s.c.level;
        x.result->done = ok;
        x.result->err = *(volatile int32_t *)&a.ctl->err;
        x.result->levels_td = s.c.levels_td;
        x.result->levels_bu = s.c.levels_bu;
        x.result->reached = s.c.reached;
        x.result->edges = s.c.edges;
    }
}

// One record per position: start and length of its push row, its id.
__global__ void k_row_recs(BfsArgs a, int4 *vrec) {
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < a.n; p += nth) {
        const int64_t st = __ldg(a.prow + p);
        vrec[p] = make_int4((int32_t)(uint32_t)st, (int32_t)(st >> 32), __ldg(a.odeg + p),
                            __ldg(a.perm + p));
    }
}

// Outputs in original ids. The order permutes only inside sigma windows, so a
// tile of whole windows is its own image: positions are read and ids written
// in order, 16 bytes a thread, and permuted in shared memory. (Scattered
// 4-byte stores inside the windows took 142 us at n = 2^24.)
__global__ void __launch_bounds__(kScatterThreads)
    k_scatter_tiles(int64_t n, int32_t tile, const int32_t *perm, const int32_t *level_pos,
                    const uint32_t *parent_pos, int32_t *level, int32_t *parent) {
    extern __shared__ int32_t st[];  // levels, then parents
    for (int64_t t0 = (int64_t)blockIdx.x * tile; t0 < n; t0 += (int64_t)gridDim.x * tile) {
        const int32_t m = (int32_t)min((int64_t)tile, n - t0);
        for (int32_t i = 4 * (int32_t)threadIdx.x; i < m; i += 4 * kScatterThreads) {
            if (i + 4 <= m) {
                const int4 v = __ldg(reinterpret_cast<const int4 *>(perm + t0 + i));
                const int4 l = __ldcs(reinterpret_cast<const int4 *>(level_pos + t0 + i));
                const int4 p = __ldcs(reinterpret_cast<const int4 *>(parent_pos + t0 + i));
                const int32_t b = (int32_t)t0;
                st[v.x - b] = l.x, st[v.y - b] = l.y, st[v.z - b] = l.z, st[v.w - b] = l.w;
                st[tile + v.x - b] = p.x, st[tile + v.y - b] = p.y;
                st[tile + v.z - b] = p.z, st[tile + v.w - b] = p.w;
            } else {
                for (int32_t k = i; k < m; k++) {
                    const int32_t v = perm[t0 + k] - (int32_t)t0;
                    st[v] = level_pos[t0 + k];
                    st[tile + v] = (int32_t)parent_pos[t0 + k];
                }
            }
        }
        __syncthreads();
        for (int half = 0; half < 2; half++) {
            int32_t *out = half ? parent : level;
            if (!out) continue;
            out += t0;
            const int32_t *src = st + half * tile;
            const bool wide = ((uintptr_t)out & 15) == 0;
            for (int32_t i = 4 * (int32_t)threadIdx.x; i < m; i += 4 * kScatterThreads) {
                if (wide && i + 4 <= m)
                    __stcs(reinterpret_cast<int4 *>(out + i), *reinterpret_cast<const int4 *>(src + i));
                else
                    for (int32_t k = i; k < min(i + 4, m); k++) out[k] = src[k];
            }
        }
        __syncthreads();
    }
}

constexpr int kTileMax = 16384;  // the largest sort window

size_t shared_bytes(int64_t nwords) {
    const int64_t stage = nwords * 4 <= kStageMax ? (nwords * 4 + 15) & ~15ll : 0;
    return kPoolAt + std::max(sizeof(Pool), (size_t)stage);
}

}  // namespace

bool grid_takes(const alb_graph *g, const alb_bfs_opts &o, const BfsArgs &a) {
    return o.loop != ALB_LOOP_HOST && !o.trace && o.policy != ALB_POLICY_BOTTOMUP_NOBYPASS &&
           !a.short_bulk && g->num_sms <= kMaxBlocks;
}

alb_status grid_launch(const alb_graph *g, const BfsArgs &a, const InitParams &in,
                       const GridArgs &args_in, cudaStream_t st) {
    GridArgs x = args_in;
    x.list_cap = x.max_out <= kFewEdges ? kListCapMax : kListPass;
    const size_t smem = shared_bytes(a.nwords);
    const bool scan = in.policy == ALB_POLICY_BOTTOMUP && a.nwords * 4 > kStageMax;
    void (*f)(BfsArgs, InitParams, GridArgs) = x.exact ? k_bfs_grid<true, false>
                                               : scan  ? k_bfs_grid<false, true>
                                                       : k_bfs_grid<false, false>;
    ALB_CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)shared_bytes(kStageMax / 4)));
    // the bitmaps' L2 window goes with the launch: the stream may be the
    // caller's, and have one of its own
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    at[1].id = cudaLaunchAttributeAccessPolicyWindow;
    at[1].val.accessPolicyWindow = g->bfs.win;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)g->num_sms);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = g->bfs.win.num_bytes > 0 ? 2 : 1;
    ALB_CK(cudaLaunchKernelEx(&cfg, f, a, in, x));
    return ALB_OK;
}

alb_status row_recs_launch(const alb_graph *g, const BfsArgs &a, int4 *vrec, cudaStream_t st) {
    launch_resident(k_row_recs, 256, g->num_sms, st, a, vrec);
    ALB_CK(cudaGetLastError());
    return ALB_OK;
}

alb_status scatter_launch(const alb_graph *g, const BfsArgs &a, int32_t *level, int32_t *parent,
                          cudaStream_t st) {
    const int32_t sigma = std::max(1, g->sell.sigma);
    const int32_t tile = sigma >= 1024 ? sigma : sigma * (1024 / sigma);
    // 16-byte accesses start at a multiple of four rows
    const bool fits = tile % 4 == 0;
    if (!fits) return ALB_ERR_UNSUPPORTED;
    const size_t smem = 2 * sizeof(int32_t) * (size_t)tile;
    // (always the largest tile's: the limit is the function's, and another
    // thread's search may be about to be launched)
    if (smem > 48 * 1024)
        ALB_CK(cudaFuncSetAttribute(k_scatter_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(2 * sizeof(int32_t) * kTileMax)));
    const int64_t tiles = (a.n + tile - 1) / tile;
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, (int64_t)g->num_sms * 32);
    k_scatter_tiles<<<grid, kScatterThreads, smem, st>>>(a.n, tile, a.perm, a.level_pos,
                                                         a.parent_pos, level, parent);
    ALB_CK(cudaGetLastError());
    return ALB_OK;
}

}  // namespace alb
