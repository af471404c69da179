// Persistent work-list BFS: many (graph, root) traversals of small and
// uneven graphs in one launch. No counterpart in the reference, which runs
// one graph per process (bfs/src/main.c).
//
// One CTA runs one traversal at a time and pops the next (graph, root) item
// from a global counter; items are ordered longest first (stored entries),
// so the tail of the launch holds the short ones. The three bitmaps of the
// traversal (frontier, next frontier, visited; one bit per sorted position)
// live in shared memory, so bottom-up frontier tests and top-down visited
// probes never leave the SM; the SELL-C-sigma and push-CSR arrays of each
// graph stay in HBM, built by alb_sell_build with that graph's own C, sigma
// and long-row threshold. Direction: Beamer alpha/beta per graph.
// Bound: the largest items' own time, a chain of memory round trips per level
// that a CTA can only spread over its warps: up to 1024 threads (at 64
// registers, one CTA per SM) whatever fewer were asked for, pushes
// dealt out evenly to threads (block_push), pulls two words per warp at a
// time. 48 R-MAT graphs of 2^10 to 2^16 vertices, 8 roots each: 222 us; 3.5 ms
// with 256 threads, a row per warp and a word per warp at a time.
// Output: level arrays (original ids), one per item, concatenated in the
// order items were added. Graphs whose bitmaps do not fit in one CTA's shared
// memory are not refused: their items run one by one on the device-driven
// single-root path (alb_bfs_device, the entry's alpha and beta) into the same
// output, before the launch. Those that fit but for the push's lists (540,000 to
// 617,000 vertices) do so where they are few, and else run in a launch of their
// own whose pushes walk the bitmap, a warp per row.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <new>
#include <numeric>
#include <vector>

#include "block_push.cuh"
#include "graph.h"

namespace alb {
namespace {

struct WlGraph {
    int64_t n, nwords;
    int32_t C, log2C;
    const int32_t *perm, *inv, *ideg, *odeg, *width;
    const int64_t *slice_off;
    const int4 *col4;
    const int64_t *prow;
    const int32_t *pcol;
    int64_t nlong;
    const int32_t *lrow;
    const int64_t *lptr;
    const int32_t *lcol;
    const uint32_t *vinit;
    int64_t m_in;
    float alpha, beta;
};

struct WlItem {
    int32_t graph, root;
    int64_t out;  // offset of this item's level array
};

constexpr int kPullWords = 2;  // words a warp pulls at a time
constexpr int kLeanShare = 7;  // see alb_worklist_run_device

struct WlState {
    int item, dir;
    unsigned next_word;
    unsigned n, mo, mi;  // what the level found
    int nlong;           // long rows left after their head
};
// kLean: for graphs whose bitmaps leave no room for the push's lists
template <bool kLean>
struct WlShared : WlState {
    PushLists rows;  // list: those long rows' numbers
};
template <>
struct WlShared<true> : WlState {};

__device__ __forceinline__ void wl_count(WlState &s, unsigned n, unsigned mo, unsigned mi) {
    n = __reduce_add_sync(kFull, n);
    mo = __reduce_add_sync(kFull, mo);
    mi = __reduce_add_sync(kFull, mi);
    if (lane_id() == 0 && n) {
        atomicAdd(&s.n, n);
        atomicAdd(&s.mo, mo);
        atomicAdd(&s.mi, mi);
    }
}

// Whether a source in [st, en) of the long-row list is in F (one warp).
__device__ __forceinline__ bool wl_scan(const WlGraph &g, const uint32_t *F, int64_t st,
                                        int64_t en) {
    for (int64_t e0 = st + lane_id(); ; e0 += 128) {
        bool hit = false;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int64_t e = e0 + 32 * u;
            const int32_t c = e < en ? __ldg(g.lcol + e) : -1;
            hit = hit || (c >= 0 && ((F[c >> 5] >> (c & 31)) & 1u));
        }
        if (__any_sync(kFull, hit)) return true;
        if (__all_sync(kFull, e0 + 128 >= en)) return false;
    }
}

// Unvisited long rows: a warp over the first kLongChunk sources of each, the
// CTA together over the rest of a row without a source in the frontier there
// (kLean: the warp over all of it).
template <int kT, bool kLean>
__device__ void wl_pull_long(const WlGraph &g, WlShared<kLean> &s, const uint32_t *F, const uint32_t *V,
                             uint32_t *N, int32_t *lv, int L) {
    const int lane = lane_id(), wib = threadIdx.x >> 5;
    if (threadIdx.x == 0) s.nlong = 0;
    __syncthreads();
    unsigned n = 0, mo = 0, mi = 0;
    auto reach = [&](int32_t p) {
        atomicOr(&N[p >> 5], 1u << (p & 31));
        lv[__ldg(g.perm + p)] = L + 1;
        n++;
        mo += (unsigned)__ldg(g.odeg + p);
        mi += (unsigned)__ldg(g.ideg + p);
    };
    for (int64_t i = wib; i < g.nlong; i += kT / 32) {
        const int32_t p = __ldg(g.lrow + i);
        if ((V[p >> 5] >> (p & 31)) & 1u) continue;
        const int64_t st = __ldg(g.lptr + i), en = __ldg(g.lptr + i + 1);
        const int64_t head = kLean ? en : min(en, st + kLongChunk);
        bool found = wl_scan(g, F, st, head);
        if constexpr (!kLean) {
            int q = 0;
            if (!found && head < en) {
                if (lane == 0) q = atomicAdd(&s.nlong, 1);
                q = __shfl_sync(kFull, q, 0);
                if (q < kPushRows) {
                    if (lane == 0) s.rows.list[q] = (int32_t)i;
                } else {  // (a full list: the warp scans the whole row)
                    found = wl_scan(g, F, head, en);
                }
            }
        }
        if (found && lane == 0) reach(p);
    }
    if constexpr (!kLean) {
        __syncthreads();
        const int left = min(s.nlong, kPushRows);
        for (int q = 0; q < left; q++) {
            const int32_t i = s.rows.list[q];
            const int64_t st = __ldg(g.lptr + i) + kLongChunk, en = __ldg(g.lptr + i + 1);
            bool found = false;
            for (int64_t e0 = st; e0 < en && !found; e0 += (kT / 32) * kLongChunk) {
                const int64_t b = e0 + wib * kLongChunk;
                found = __syncthreads_or(b < en && wl_scan(g, F, b, min(en, b + kLongChunk)));
            }
            if (found && threadIdx.x == 0) reach(__ldg(g.lrow + i));
        }
    }
    wl_count(s, n, mo, mi);
}

// Bottom-up pull, kPullWords words per warp at a time, lane per row.
__device__ __forceinline__ void wl_pull(const WlGraph &g, WlState &s, const uint32_t *F,
                                        const uint32_t *V, uint32_t *N, int32_t *lv, int L) {
    const int lane = lane_id(), nw = (int)g.nwords;
    unsigned n = 0, mo = 0, mi = 0;
    while (true) {
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(&s.next_word, (unsigned)kPullWords);
        const int wa = (int)__shfl_sync(kFull, at, 0);
        if (wa >= nw) break;
        int32_t p[kPullWords], ng[kPullWords];
        bool act[kPullWords], found[kPullWords];
        const int4 *cp[kPullWords];
        int4 c[kPullWords];
        int64_t so[kPullWords];
#pragma unroll
        for (int t = 0; t < kPullWords; t++) {
            const uint32_t vis = wa + t < nw ? V[wa + t] : kFull;
            p[t] = (wa + t) * 32 + lane;
            act[t] = !((vis >> lane) & 1u);
            found[t] = false;
            const int32_t sl = (act[t] ? p[t] : 0) >> g.log2C;
            ng[t] = act[t] ? (__ldg(g.width + sl) + 3) >> 2 : 0;
            so[t] = act[t] ? __ldg(g.slice_off + sl) : 0;
        }
#pragma unroll
        for (int t = 0; t < kPullWords; t++) {
            cp[t] = g.col4 + (so[t] >> 2) + (p[t] & (g.C - 1));
            c[t] = make_int4(p[t], p[t], p[t], p[t]);
            if (ng[t] > 0) c[t] = __ldg(cp[t]);
        }
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
                if (j + 1 < ng[t]) nx = __ldg(cp[t] + (int64_t)(j + 1) * g.C);
                // (padding is the row itself, never in the frontier)
                found[t] = ((F[c[t].x >> 5] >> (c[t].x & 31)) | (F[c[t].y >> 5] >> (c[t].y & 31)) |
                            (F[c[t].z >> 5] >> (c[t].z & 31)) | (F[c[t].w >> 5] >> (c[t].w & 31))) & 1u;
                act[t] = !found[t] && c[t].w != p[t];
                c[t] = nx;
            }
        }
#pragma unroll
        for (int t = 0; t < kPullWords; t++) {
            if (wa + t >= nw) break;
            const unsigned nm = __ballot_sync(kFull, found[t]);
            if (lane == 0) N[wa + t] = nm;
            if (found[t]) {
                lv[__ldg(g.perm + p[t])] = L + 1;
                n++;
                mo += (unsigned)__ldg(g.odeg + p[t]);
                mi += (unsigned)__ldg(g.ideg + p[t]);
            }
        }
    }
    wl_count(s, n, mo, mi);
}

// Top-down push without lists: a warp looks through 32 words at a time, lane per
// word, and takes their rows one by one, lane per edge.
template <class Push>
__device__ __forceinline__ void wl_push_lean(const WlGraph &g, const uint32_t *F, int nw, int warps,
                                             Push push) {
    const int lane = lane_id();
    for (int wb = (int)(threadIdx.x & ~31u); wb < nw; wb += 32 * warps) {
        const uint32_t m = wb + lane < nw ? F[wb + lane] : 0u;
        for (unsigned todo = __ballot_sync(kFull, m != 0); todo; todo &= todo - 1) {
            const int q = __ffs(todo) - 1;
            // the word's rows: their bounds by one lane each
            const uint32_t mq = __shfl_sync(kFull, m, q);
            int32_t st = 0, d = 0;
            if ((mq >> lane) & 1u) {
                const int32_t u = (wb + q) * 32 + lane;
                st = (int32_t)__ldg(g.prow + u);
                d = (int32_t)__ldg(g.prow + u + 1) - st;
            }
            for (unsigned rows = mq; rows; rows &= rows - 1) {
                const int r = __ffs(rows) - 1;
                const int32_t b = __shfl_sync(kFull, st, r), n = __shfl_sync(kFull, d, r);
                for (int32_t e = lane; e < n; e += 32) push(__ldg(g.pcol + b + e));
            }
        }
    }
}

// kT threads, 1024 / kT CTAs per SM.
template <int kT, bool kLean>
__global__ void __launch_bounds__(kT, 1024 / kT)
    k_worklist(const WlGraph *graphs, const WlItem *items, int32_t nitems, unsigned int *next_item,
               int32_t *out) {
    extern __shared__ __align__(16) unsigned char smem[];
    WlShared<kLean> &s = *reinterpret_cast<WlShared<kLean> *>(smem);
    uint32_t *maps = reinterpret_cast<uint32_t *>(smem + sizeof(WlShared<kLean>));
    const int lane = lane_id();
    while (true) {
        if (threadIdx.x == 0) s.item = (int)atomicAdd(next_item, 1u);
        __syncthreads();
        const int it = s.item;
        if (it >= nitems) break;
        const WlItem item = items[it];
        const WlGraph g = graphs[item.graph];
        const int nw = (int)g.nwords;
        uint32_t *F = maps, *N = maps + nw, *V = maps + 2 * nw;
        int32_t *lv = out + item.out;
        for (int w = threadIdx.x; w < nw; w += kT) {
            V[w] = g.vinit[w];
            F[w] = 0;
        }
        for (int64_t v = threadIdx.x; v < g.n; v += kT) lv[v] = -1;
        const int32_t rp = __ldg(g.inv + item.root);
        unsigned nf = 1, prev_nf = 0, mf = (unsigned)__ldg(g.odeg + rp),
                 mu = (unsigned)g.m_in - (unsigned)__ldg(g.ideg + rp);
        __syncthreads();
        if (threadIdx.x == 0) {
            V[rp >> 5] |= 1u << (rp & 31);
            F[rp >> 5] |= 1u << (rp & 31);
            lv[item.root] = 0;
        }
        int prev_dir = -1;
        __syncthreads();
        for (int L = 0; nf > 0 && L <= g.n; L++) {
            if (threadIdx.x == 0) {  // Beamer's rule (dev.cuh)
                BfsCtl c;
                c.prev_dir = prev_dir;
                c.nf = nf;
                c.prev_nf = prev_nf;
                c.mf = mf;
                c.mu = mu;
                c.n = g.n;
                c.alpha = g.alpha;
                c.beta = g.beta;
                s.dir = beamer_dir(c);
                s.next_word = s.n = s.mo = s.mi = 0;
            }
            __syncthreads();
            const int dir = s.dir;
            if (dir == ALB_DIR_BOTTOMUP) {
                wl_pull(g, s, F, V, N, lv, L);
                __syncthreads();
                if (g.nlong) {
                    wl_pull_long<kT, kLean>(g, s, F, V, N, lv, L);
                    __syncthreads();
                }
                for (int w = threadIdx.x; w < nw; w += kT) V[w] |= N[w];
            } else {
                for (int w = threadIdx.x; w < nw; w += kT) N[w] = 0;
                auto push = [&](int32_t v) {
                    const uint32_t bit = 1u << (v & 31);
                    if (!((V[v >> 5] | N[v >> 5]) & bit)) atomicOr(&N[v >> 5], bit);
                };
                if constexpr (kLean) {
                    __syncthreads();  // (all of N is cleared)
                    wl_push_lean(g, F, nw, kT / 32, push);
                } else {
                    // a frontier that fits the list is listed at once: a look at
                    // 64 words at a time costs 0.3 us where they are empty and 2
                    // where not, 60 us for 72 rows of 2^16
                    block_push<kT>(
                        s.rows, F, 0, nw, nf <= (unsigned)kPushRows ? nw : kPushWords, g.pcol,
                        [&](int32_t u, int32_t &st, int32_t &d, int32_t &ou) {
                            st = (int32_t)__ldg(g.prow + u);
                            d = (int32_t)__ldg(g.prow + u + 1) - st;
                            ou = 0;
                        },
                        [&](const int32_t (&v)[4], const uint32_t (&)[4]) {
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                if (v[k] >= 0) push(v[k]);
                        });
                }
                __syncthreads();
                // the new frontier: levels, visited bits, counters; a warp per
                // 32 words, lane per row
                unsigned n = 0, mo = 0, mi = 0;
                for (int wb = (int)(threadIdx.x & ~31u); wb < nw; wb += kT) {
                    const uint32_t m = wb + lane < nw ? N[wb + lane] : 0u;
                    if (m) V[wb + lane] |= m;
                    for (unsigned todo = __ballot_sync(kFull, m != 0); todo; todo &= todo - 1) {
                        const int q = __ffs(todo) - 1;
                        if (!((__shfl_sync(kFull, m, q) >> lane) & 1u)) continue;
                        const int32_t p = (wb + q) * 32 + lane;
                        lv[__ldg(g.perm + p)] = L + 1;
                        n++;
                        mo += (unsigned)__ldg(g.odeg + p);
                        mi += (unsigned)__ldg(g.ideg + p);
                    }
                }
                wl_count(s, n, mo, mi);
            }
            __syncthreads();
            uint32_t *t = F;  // N becomes the frontier
            F = N;
            N = t;
            prev_nf = nf;
            nf = s.n;
            mf = s.mo;
            mu -= s.mi;
            prev_dir = dir;
            __syncthreads();  // the sums have been read
        }
    }
}

}  // namespace
}  // namespace alb

struct alb_worklist {
    struct Entry {
        alb_graph *g;
        std::vector<int32_t> roots;
        float alpha, beta;
    };
    std::vector<Entry> entries;
    int64_t total_out = 0;
    // The launch's arguments: a page-locked image of the graphs, items and item
    // counter, and its device copy. Filled anew by every run, kept between them
    // (allocated and freed each time they cost 19 us); one run at a time.
    std::mutex mu;
    unsigned char *h_args = nullptr, *d_args = nullptr;
    size_t args_cap = 0;
    int device = 0;

    // (on the current device, dev)
    alb_status reserve(size_t bytes, int dev) {
        if (bytes <= args_cap && dev == device) return ALB_OK;
        release();
        ALB_CK(cudaMallocHost((void **)&h_args, bytes));
        const alb_status rc = alb::dmalloc((void **)&d_args, bytes, "worklist arguments");
        if (rc != ALB_OK) {
            release();
            return rc;
        }
        args_cap = bytes;
        device = dev;
        return ALB_OK;
    }
    void release() {
        if (!h_args) return;
        int prev = -1;
        cudaGetDevice(&prev);
        cudaSetDevice(device);
        cudaFreeHost(h_args);
        alb::dfree(d_args);
        cudaGetLastError();
        if (prev >= 0) cudaSetDevice(prev);
        h_args = d_args = nullptr;
        args_cap = 0;
    }
    ~alb_worklist() { release(); }
};

using namespace alb;

extern "C" {

alb_status alb_worklist_create(alb_worklist **out) {
    if (!out) return fail(ALB_ERR_INVALID, "alb_worklist_create: out is NULL");
    try {
        *out = new alb_worklist();
    } catch (const std::bad_alloc &) {
        return fail(ALB_ERR_OOM, "alb_worklist_create: host allocation failed");
    }
    return ALB_OK;
}

void alb_worklist_destroy(alb_worklist *w) { delete w; }

alb_status alb_worklist_add(alb_worklist *w, alb_graph *g, const int32_t *roots, int32_t nroots,
                            float alpha, float beta) {
    if (!w || !g || !roots || nroots < 1) return fail(ALB_ERR_INVALID, "alb_worklist_add: bad arguments");
    if (!g->sell.built) return fail(ALB_ERR_STATE, "alb_worklist_add: call alb_sell_build first");
    if (!(alpha > 0) || !(beta > 0)) return fail(ALB_ERR_INVALID, "alb_worklist_add: alpha, beta > 0");
    for (int i = 0; i < nroots; i++)
        if (roots[i] < 0 || roots[i] >= g->n)
            return fail(ALB_ERR_INVALID, "alb_worklist_add: root %d outside the graph", roots[i]);
    try {
        w->entries.push_back({g, std::vector<int32_t>(roots, roots + nroots), alpha, beta});
    } catch (const std::bad_alloc &) {
        return fail(ALB_ERR_OOM, "alb_worklist_add: host allocation failed");
    }
    w->total_out += g->n * (int64_t)nroots;
    return ALB_OK;
}

alb_status alb_worklist_size(const alb_worklist *w, int64_t *level_entries, int32_t *items) {
    if (!w) return fail(ALB_ERR_INVALID, "alb_worklist_size: worklist is NULL");
    int32_t k = 0;
    for (auto &e : w->entries) k += (int32_t)e.roots.size();
    if (level_entries) *level_entries = w->total_out;
    if (items) *items = k;
    return ALB_OK;
}

alb_status alb_worklist_run_device(alb_worklist *w, int32_t block, int32_t *d_levels,
                                   alb_stats *st) {
    if (!w || w->entries.empty() || !d_levels)
        return fail(ALB_ERR_INVALID, "alb_worklist_run: empty worklist or no output");
    if (!(block == 128 || block == 256 || block == 512 || block == 1024))
        return fail(ALB_ERR_UNSUPPORTED, "alb_worklist_run: block must be 128, 256, 512 or 1024");
    alb_graph *g0 = w->entries[0].g;
    ALB_CK(cudaSetDevice(g0->device));
    int max_smem = 0;
    ALB_CK(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, g0->device));
    // a graph fits the kernel when its three bitmaps and the rest of the
    // shared state fit in one CTA (and its edges in 32-bit counters)
    auto fits = [&](const Sell &s, size_t state) {
        return sizeof(uint32_t) * 3 * (size_t)s.nwords + std::max<size_t>(state, 1024) <=
                   (size_t)max_smem && s.m_in <= INT32_MAX && s.m_out <= INT32_MAX;
    };
    // Where there is no room for the push's lists, an item takes 13 to 25 times
    // as long in the kernel as on the single-root path, one CTA against all SMs,
    // but as many as there are SMs run side by side: the kernel takes them from
    // a seventh of that on (kLeanShare). Uniform random, 580,000 vertices of mean
    // degree 6, 16 items 2.37 ms in the kernel and 2.19 one by one, 32 2.45 and
    // 4.30, 152 2.66 and 20.3; 560,000 of degree 40 3.23 and 1.89, 3.16 and 3.78,
    // 2.99 and 17.9; a grid of 577,600 21.8 and 25.5, 21.8 and 50.4, 22.7 and 244.
    struct Part {
        std::vector<WlItem> items;
        std::vector<int64_t> cost;
        int64_t nwords_max = 0;
    } part[2];  // with the lists, without
    int64_t lean_items = 0;
    for (const auto &e : w->entries)
        if (e.g->sell.built && !fits(e.g->sell, sizeof(WlShared<false>) + 1024) &&
            fits(e.g->sell, sizeof(WlShared<true>)))
            lean_items += (int64_t)e.roots.size();
    const bool lean = kLeanShare * lean_items >= g0->num_sms;
    std::vector<WlGraph> hg;
    int64_t off = 0;
    float big_ms = 0.f;
    int64_t big_kernels = 0;
    for (size_t gi = 0; gi < w->entries.size(); gi++) {
        const auto &e = w->entries[gi];
        const Sell &s = e.g->sell;
        if (!s.built) return fail(ALB_ERR_STATE, "alb_worklist_run: a graph lost its SELL build");
        const bool lists = fits(s, sizeof(WlShared<false>) + 1024);
        if (!lists && !(lean && fits(s, sizeof(WlShared<true>)))) {
            // too large for one CTA's shared memory: the single-root path
            alb_bfs_opts o;
            alb_bfs_opts_default(&o);
            o.policy = ALB_POLICY_BEAMER;
            o.loop = ALB_LOOP_GRAPH;
            o.alpha = e.alpha;
            o.beta = e.beta;
            for (int32_t r : e.roots) {
                alb_stats bs;
                ALB_TRY(alb_bfs_device(e.g, r, &o, d_levels + off, nullptr, &bs));
                big_ms += bs.ms;
                big_kernels += bs.kernels;
                off += e.g->n;
            }
            continue;
        }
        WlGraph d;
        std::memset(&d, 0, sizeof(d));
        d.n = e.g->n;
        d.nwords = s.nwords;
        d.C = s.C;
        d.log2C = s.log2C;
        d.perm = s.perm;
        d.inv = s.inv;
        d.ideg = s.ideg;
        d.odeg = s.odeg;
        d.width = s.width;
        d.slice_off = s.slice_off;
        d.col4 = (const int4 *)s.col;
        d.prow = s.prow;
        d.pcol = s.pcol;
        d.nlong = s.nlong;
        d.lrow = s.lrow;
        d.lptr = s.lptr;
        d.lcol = s.lcol;
        d.vinit = s.vinit;
        d.m_in = s.m_in;
        d.alpha = e.alpha;
        d.beta = e.beta;
        hg.push_back(d);
        Part &p = part[lists ? 0 : 1];
        p.nwords_max = std::max(p.nwords_max, s.nwords);
        // the kernel's graph index is the position in hg
        for (int32_t r : e.roots) {
            p.items.push_back({(int32_t)hg.size() - 1, r, off});
            p.cost.push_back(e.g->nnz_in);
            off += e.g->n;
        }
    }
    if (hg.empty()) {  // every graph took the single-root path
        if (st) {
            std::memset(st, 0, sizeof(*st));
            st->ms = big_ms;
            st->kernels = big_kernels;
        }
        return ALB_OK;
    }
    // longest items first
    std::vector<WlItem> sorted;
    for (const Part &p : part) {
        std::vector<int32_t> order(p.items.size());
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(),
                         [&](int32_t a, int32_t b) { return p.cost[a] > p.cost[b]; });
        for (int32_t k : order) sorted.push_back(p.items[k]);
    }
    const size_t items_at = sizeof(WlGraph) * hg.size();
    const size_t ctr_at = items_at + sizeof(WlItem) * sorted.size();
    static_assert(sizeof(WlGraph) % 8 == 0 && sizeof(WlItem) % 8 == 0, "laid out one after the other");
    const size_t args = ctr_at + 8;  // a counter for each part
    std::lock_guard<std::mutex> lock(w->mu);
    alb_status rc = [&]() -> alb_status {
        ALB_TRY(w->reserve(args, g0->device));
        std::memcpy(w->h_args, hg.data(), items_at);
        std::memcpy(w->h_args + items_at, sorted.data(), ctr_at - items_at);
        std::memset(w->h_args + ctr_at, 0, 8);
        const WlGraph *dg = reinterpret_cast<const WlGraph *>(w->d_args);
        const WlItem *di = reinterpret_cast<const WlItem *>(w->d_args + items_at);
        unsigned int *dctr = reinterpret_cast<unsigned int *>(w->d_args + ctr_at);
        cudaStream_t stream = g0->stream;
        ALB_CK(cudaMemcpyAsync(w->d_args, w->h_args, args, cudaMemcpyHostToDevice, stream));
        ALB_CK(cudaEventRecord(g0->ev0, stream));
        int64_t launches = 0;
        for (int k = 0; k < 2; k++) {
            const int64_t count = (int64_t)part[k].items.size();
            if (count == 0) continue;
            const int64_t nw = part[k].nwords_max;
            // 1024 threads end the longest items soonest; where there are many
            // items for every SM, two CTAs of 512 get more of them done; graphs
            // of a word per warp of 256 threads and fewer than four have no use
            // for more
            const int threads = k == 1                      ? 1024
                                : nw <= 32 && block <= 256 ? 256
                                : block == 1024 || count <= 4 * (int64_t)g0->num_sms ? 1024
                                                                                     : 512;
            void (*f)(const WlGraph *, const WlItem *, int32_t, unsigned int *, int32_t *) =
                k == 1           ? k_worklist<1024, true>
                : threads == 256 ? k_worklist<256, false>
                : threads == 512 ? k_worklist<512, false>
                                 : k_worklist<1024, false>;
            const size_t smem = (k ? sizeof(WlShared<true>) : sizeof(WlShared<false>)) +
                                sizeof(uint32_t) * 3 * (size_t)nw;
            // (always the most: the limit is the function's, and another
            // thread's list may be about to be launched)
            ALB_CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
            int per_sm = 0;
            ALB_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, threads, smem));
            if (per_sm < 1)
                return fail(ALB_ERR_UNSUPPORTED, "alb_worklist_run: kernel does not fit");
            const unsigned grid =
                (unsigned)std::min<int64_t>((int64_t)per_sm * g0->num_sms, count);
            f<<<grid, threads, smem, stream>>>(dg, di, (int32_t)count, dctr + k, d_levels);
            ALB_CK(cudaGetLastError());
            di += count;
            launches++;
        }
        ALB_CK(cudaEventRecord(g0->ev1, stream));
        ALB_CK(cudaStreamSynchronize(stream));
        float ms = 0;
        ALB_CK(cudaEventElapsedTime(&ms, g0->ev0, g0->ev1));
        if (st) {
            std::memset(st, 0, sizeof(*st));
            st->ms = ms + big_ms;
            st->kernels = launches + big_kernels;
        }
        return ALB_OK;
    }();
    if (rc != ALB_OK) cudaStreamSynchronize(g0->stream);  // (the image may be on its way)
    return rc;
}

alb_status alb_worklist_run(alb_worklist *w, int32_t block, int32_t *levels, alb_stats *st) {
    if (!w || w->entries.empty() || !levels)
        return fail(ALB_ERR_INVALID, "alb_worklist_run: empty worklist or no output");
    alb_graph *g0 = w->entries[0].g;
    ALB_CK(cudaSetDevice(g0->device));
    int32_t *d = nullptr;
    ALB_TRY(dmalloc((void **)&d, sizeof(int32_t) * (size_t)w->total_out, "worklist levels"));
    alb_status rc = alb_worklist_run_device(w, block, d, st);
    if (rc == ALB_OK) {
        cudaError_t e = cudaMemcpy(levels, d, sizeof(int32_t) * (size_t)w->total_out,
                                   cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) rc = fail(ALB_ERR_CUDA, "alb_worklist_run: %s", cudaGetErrorString(e));
    }
    dfree(d);
    return rc;
}

}  // extern "C"
