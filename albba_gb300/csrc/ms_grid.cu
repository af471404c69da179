// Batched BFS as one cooperative kernel: one block of 1024 threads per SM runs
// every level, the steps of a level (ms.cuh) a grid barrier apart, and every
// block decides the next level by itself from the summed counters.
//
// What bounded the level loop as a CUDA graph was its launches: a level was 9
// to 10 kernels behind a switch and a while node, about 43 us on R-MAT scale
// 16 whatever the level held. Here a level takes one barrier (a pull) to five
// (a push with long rows and samples), some 1.5 us each, and steps without
// work are not run. 37 roots on R-MAT scale 16, a call with its output: 420 ->
// 153 us; 64 on scale 20 (learned policy) 728 -> 415; 64 on scale 24 (learned,
// random roots) 3,433 -> 3,175, of which the large pulls (870 to 970 and 240 to
// 400) are bound by their gathers and the output (870) by memory.
//
// The block keeps under 8 KB of shared memory: L1 holds the gathers' hubs.
// With 40 KB (the selector's weights and a frontier row table copied there)
// scale 24 took 5 % longer.
#include "ms_grid.h"

namespace alb {
namespace {

constexpr int kThreads = 1024, kWarps = kThreads / 32;
constexpr int kCtl = kWarps - 1;  // the warp that waits at barriers and decides
// Columns of a wide slice. The first bottom-up level of R-MAT scale 16 / 20
// takes 63 / 273 us with none, 57 / 182 at 128, 54 / 175 at 64.
constexpr int kSplit = 64;
constexpr unsigned long long kBarFailed = 1ull << 62;  // a wait gave up

using Level = MsSlots::Level;

struct Shared {
    MsCtl c;
    MsSums sum;               // the level's sums at the last counting barrier
    unsigned long long word[2];  // the counters that the last barrier read
    MsSums warp[kWarps];
    unsigned long long room[128];
    int ok;
    union {
        uint16_t buf[kWarps][kRowBuf];
        MsSampleRoom sample;
        uint64_t team[kWarps / kTeam * 32];
    };
};

__device__ __forceinline__ unsigned long long add_acq_rel(unsigned long long *p,
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

// Adds what the calling warp found in a step to its sums; the next counting
// barrier adds up the warps'.
__device__ __forceinline__ void put(Shared &s, const MsCounts &c) {
    const unsigned n = __reduce_add_sync(kFull, c.n), full = __reduce_add_sync(kFull, c.full),
                   done = __reduce_add_sync(kFull, c.done);
    const unsigned long long bytes = warp_sum(c.bytes);
    MsSums &w = s.warp[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    if (lane == 0) w.bytes += bytes;
    if (!__any_sync(kFull, c.bits != 0)) return;  // (then nothing else was found either)
    const unsigned long long bits = warp_sum((unsigned long long)c.bits), mo = warp_sum(c.mo),
                             mi = warp_sum(c.mi), edges = warp_sum(c.edges);
    if (lane != 0) return;
    w.n += n;
    w.bits += bits;
    w.full += full;
    w.done += done;
    w.mo += mo;
    w.mi += mi;
    w.edges += edges;
}

// Grid barrier on the arrival counter, which is never reset: a block's barrier
// ends when the count reaches the next multiple of the block count. acc (null:
// none): every warp's sums are added up there and read back into s.sum. word
// (null: none): two counters read into s.word.
__device__ bool barrier(const MsArgs &a, const MsGridArgs &x, Shared &s, int L,
                        MsSums *acc = nullptr, const unsigned long long *word = nullptr) {
    if (x.withhold_level >= 0 && L == x.withhold_level && (int)blockIdx.x == x.withhold_block)
        return false;
    __syncthreads();
    if ((threadIdx.x >> 5) == kCtl) {
        const int lane = threadIdx.x & 31;
        constexpr int kSums = (int)(sizeof(MsSums) / 8);
        unsigned long long *sums = reinterpret_cast<unsigned long long *>(acc);
        if (acc) {
            // lane l: sum l % 8 of warps l / 8, l / 8 + 4, ...
            static_assert(kSums == 8 && kWarps == 32, "four lanes a sum, eight warps a lane");
            unsigned long long v = 0;
#pragma unroll
            for (int w = 0; w < kWarps; w += 4) {
                unsigned long long *p =
                    reinterpret_cast<unsigned long long *>(&s.warp[w + (lane >> 3)]) + (lane & 7);
                v += *p;
                *p = 0;
            }
            v += __shfl_xor_sync(kFull, v, 8);
            v += __shfl_xor_sync(kFull, v, 16);
            if (lane < kSums && v) atomicAdd(sums + lane, v);
            __syncwarp();
        }
        const unsigned long long nb = gridDim.x;
        unsigned long long v = 0;
        if (lane == 0) v = add_acq_rel(&x.slots->bar, 1ull);
        v = __shfl_sync(kFull, v, 0);
        const unsigned long long target = (v / nb + 1) * nb;
        v++;
        const uint64_t t0 = globaltimer_ns();
        bool ok = true;
        // (all lanes poll: a warp that leaves a one-lane wait stays split)
        while (__any_sync(kFull, v < target)) {
            if (__any_sync(kFull, globaltimer_ns() - t0 > x.barrier_ns)) {
                if (lane == 0) {
                    atomicExch(&a.ctl->err, ALB_ERR_TIMEOUT);
                    atomicOr(&x.slots->bar, kBarFailed);
                }
                ok = false;
                break;
            }
            v = ld_acquire(&x.slots->bar);
        }
        if (lane == 0) s.ok = ok && !(v & kBarFailed);
        __syncwarp();
        if (acc && lane < kSums) reinterpret_cast<unsigned long long *>(&s.sum)[lane] = __ldcg(sums + lane);
        if (word && lane >= kSums && lane < kSums + 2)
            s.word[lane - kSums] = __ldcg(word + lane - kSums);
    }
    __syncthreads();
    return s.ok;
}

// The level's end (one warp): the sums go into the block's control block and
// the next level is decided, by the same rules in every block.
__device__ __noinline__ void end_level(const MsArgs &a, Shared &s) {
    const int lane = threadIdx.x & 31;
    MsCtl &c = s.c;
    unsigned long long e0 = 0, e1 = 0;
    if (c.dir == ALB_DIR_TOPDOWN) {  // (also read where the next level turns out top-down)
        e0 = __ldcg(&a.smp->deg[lane]);
        e1 = __ldcg(&a.smp->deg[lane + 32]);
    }
    if (lane == 0) ms_rollover(c, c.dir, s.sum);
    __syncwarp();
    BfsCtl fc;
    ms_feature_ctl(c, fc);
    int next;
    if (c.policy == ALB_POLICY_LEARNED && a.mlp && a.mlp[kMlpParams] != 0.0f) {
        float f[kMlpIn];
        level_features_warp(fc, f);
        next = mlp_select_warp(a.mlp, f);
    } else {
        next = rule_dir(fc);
    }
    unsigned long long tm = 0;
    if (next != ALB_DIR_TOPDOWN && c.dir == ALB_DIR_TOPDOWN && !c.done && c.push_budget > 0)
        tm = ms_pushed_roots(e0, e1, (unsigned long long)c.push_budget, c.used, s.room);
    __syncwarp();
    if (lane == 0) {
        c.tmask = tm;
        c.pushed_roots += __popcll(tm);
        ms_set_next(a, c, next);
    }
    __syncwarp();
}

// The initial state of this block's words, and of the roots among them.
__device__ void init_state(const MsArgs &a, const MsInit &in, Shared &s) {
    const int64_t w0 = a.nwords * blockIdx.x / gridDim.x, w1 = a.nwords * (blockIdx.x + 1) / gridDim.x;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (int64_t w = w0 + wib; w < w1; w += kWarps) {
        const uint32_t dead = __ldg(a.vinit + w);
        a.V[w * 32 + lane] = ((dead >> lane) & 1u) ? kAll : in.unused;
        a.S[w * 32 + lane] = 0;
        if (lane == 0) {
            a.D[w] = dead;
            a.A[w] = 0;
        }
    }
    __syncthreads();
    if (wib != 0) return;
    MsCounts c;
    int32_t mine[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int i = lane + 32 * h;
        mine[h] = -1;
        if (i >= in.nroots) continue;
        const int32_t p = __ldg(a.inv + in.roots[i]);
        if ((p >> 5) < w0 || (p >> 5) >= w1) continue;
        mine[h] = p;
        const unsigned od = (unsigned)__ldg(a.odeg + p);
        atomicOr((unsigned long long *)a.V + p, 1ull << i);
        if (atomicOr((unsigned long long *)a.S + p, 1ull << i) == 0) {
            c.n++;
            c.mo += od;
            atomicOr(a.A + (p >> 5), 1u << (p & 31));
        }
        // bit i belongs to root i alone, so every root counts once (it may be
        // set in V already when p has no sources: V starts full there)
        c.bits++;
        c.edges += od;
    }
    __syncwarp();
    // positions whose every root bit is now set
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int32_t p = mine[h];
        if (p < 0 || __ldcg((const unsigned long long *)a.V + p) != kAll) continue;
        const uint32_t bit = 1u << (p & 31), old = atomicOr(a.D + (p >> 5), bit);
        if (old & bit) continue;
        c.done++;
        c.mi += __ldg(a.ideg + p);
        c.full += (old | bit) == kFull;
    }
    put(s, c);
}

template <bool kBypass, bool kEarly>
__device__ __forceinline__ void pull(const MsArgs &a, const MsStep &x, const MsCtl &c,
                                     int split, unsigned long long *work, MsCounts &cnt) {
    if (c.filt)
        ms_pull<kBypass, kEarly, true>(a, x, c.grab, split, work, cnt);
    // the first bottom-up level after a top-down one takes two column groups
    // at a time: rows scan longest there before every root is accounted for;
    // later rows stop sooner and the second is mostly fetched for nothing
    else if (kEarly && c.prev_dir == ALB_DIR_TOPDOWN)
        ms_pull<kBypass, kEarly, false, kEarly>(a, x, c.grab, split, work, cnt);
    else
        ms_pull<kBypass, kEarly, false>(a, x, c.grab, split, work, cnt);
}

// A top-down level up to its counts. False: a wait gave up.
__device__ __forceinline__ bool level_down(const MsArgs &a, const MsGridArgs &x, Shared &s,
                                           const MsStep &p, Level &l, Level &next) {
    const int wib = threadIdx.x >> 5;
    int32_t *Q = (p.L & 1) ? a.q1 : a.q0;
    MsCounts cnt;
    // a queue made here has its big rows listed: they are pushed beside the
    // others (R-MAT scale 16: level 0 24 -> 18 us)
    const bool known = !s.c.q_valid;
    if (known) ms_compact(a, p, Q, &l.qn, &l.nbig);
    ms_zero_next(a, p);
    if (!barrier(a, x, s, p.L, nullptr, &l.nbig)) return false;
    if (blockIdx.x == 0 && threadIdx.x < 64) a.smp->deg[threadIdx.x] = 0;
    ms_push_rows<false>(a, p, Q, (int64_t)s.word[1], &l.nbig, cnt);
    if (known && s.word[0]) ms_push_big<false>(a, p, s.word[0], cnt);
    if (!barrier(a, x, s, p.L, nullptr, known ? nullptr : &l.nbig)) return false;
    if (!known && s.word[0]) {
        ms_push_big<false>(a, p, s.word[0], cnt);
        if (!barrier(a, x, s, p.L)) return false;
    }
    ms_finish(a, p, s.buf[wib], (p.L & 1) ? a.q0 : a.q1, &next.qn, cnt);
    put(s, cnt);
    if (!barrier(a, x, s, p.L, &l.acc)) return false;
    if (!ms_samples(a, s.c.push_budget, ALB_DIR_TOPDOWN, (int64_t)s.sum.n)) return true;
    ms_sample(a, p, s.sample, &l.acc.bytes);
    return barrier(a, x, s, p.L);
}

template <bool kEarly>
__device__ __forceinline__ bool long_rows(const MsArgs &a, const MsGridArgs &x, Shared &s,
                                          const MsStep &p, Level &l) {
    const int filt = s.c.filt;
    MsCounts cnt;
    ms_long_head<kEarly>(a, p, filt, &l.nbig, cnt);
    put(s, cnt);
    if (!barrier(a, x, s, p.L, &l.acc, &l.nbig)) return false;
    const unsigned long long ctr = s.word[0];
    if (!ctr) return true;
    MsCounts tail;
    ms_long_tail<kEarly>(a, p, filt, ctr, tail);
    if (!barrier(a, x, s, p.L)) return false;
    ms_long_fin(a, p, ctr, tail);
    put(s, tail);
    return barrier(a, x, s, p.L, &l.acc);
}

// A bottom-up level up to its counts. False: a wait gave up.
__device__ __forceinline__ bool level_up(const MsArgs &a, const MsGridArgs &x, Shared &s,
                                         const MsStep &p, Level &l) {
    int32_t *Q = (p.L & 1) ? a.q0 : a.q1;  // (the next level's: idle here)
    const bool early = s.c.dir == ALB_DIR_BOTTOMUP;
    if (p.tm) {
        MsCounts cnt;
        ms_tq(a, p, Q, &l.pqn, &l.pbig, cnt);
        put(s, cnt);
    }
    {
        MsCounts cnt;
        if (early) {
            // wide words by teams where runs are short, that is where a level is
            // not many times a wide word's time: at the first bottom-up level
            // after a top-down one, and where there is no word for every warp
            // at all of them (else most rows stop after a few columns later:
            // R-MAT scale 20's second one 54 -> 71 us)
            const bool teams = a.C >= 32 && s.c.grab < 32 &&
                               (s.c.prev_dir == ALB_DIR_TOPDOWN || a.nwords <= p.nwarps);
            const int split = teams ? kSplit : INT32_MAX;
            if (teams) ms_pull_wide(a, p, split, s.team, cnt);
            pull<true, true>(a, p, s.c, split, &l.work, cnt);
        } else {
            pull<false, false>(a, p, s.c, INT32_MAX, &l.work, cnt);
        }
        put(s, cnt);
    }
    if (!barrier(a, x, s, p.L, &l.acc, &l.pbig)) return false;
    const unsigned long long big = s.word[0];
    const int64_t pq = (int64_t)s.word[1];
    if (a.nlong && !(early ? long_rows<true>(a, x, s, p, l) : long_rows<false>(a, x, s, p, l)))
        return false;
    if (!pq) return true;
    MsCounts cnt;
    ms_push_rows<true>(a, p, Q, pq, &l.pbig, cnt);
    if (big) ms_push_big<true>(a, p, big, cnt);
    put(s, cnt);
    return barrier(a, x, s, p.L, &l.acc);
}

__global__ void __launch_bounds__(kThreads, 1)
k_ms_grid(const __grid_constant__ MsArgs a, const __grid_constant__ MsInit in,
          const __grid_constant__ MsGridArgs x) {
    __shared__ Shared s;
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    for (int i = threadIdx.x; i < (int)(sizeof(s.warp) / 8); i += kThreads)
        reinterpret_cast<unsigned long long *>(s.warp)[i] = 0;
    if (first) a.ctl->err = 0;
    bool ok = true;
    if (!x.resume) {
        if (blockIdx.x == 0) {  // (read by nobody before the barrier)
            for (int i = threadIdx.x; i < (int)(sizeof(Level) * 3 / 8); i += kThreads)
                reinterpret_cast<unsigned long long *>(x.slots->level)[i] = 0;
            if (threadIdx.x < 64) a.smp->deg[threadIdx.x] = 0;
        }
        __syncthreads();
        init_state(a, in, s);
        ok = barrier(a, x, s, -1, &x.slots->level[3].acc);
        if (threadIdx.x == kCtl * 32) {
            const MsSums &k = s.sum;
            ms_start(a, in, (int64_t)k.n, (int64_t)k.mo, (int64_t)k.bits, (int64_t)k.edges,
                     (int64_t)k.done, (int64_t)k.mi, (int64_t)k.full, s.c);
        }
    } else {
        for (int i = threadIdx.x; i < (int)(sizeof(MsCtl) / 8); i += kThreads)
            reinterpret_cast<unsigned long long *>(&s.c)[i] =
                __ldcg(reinterpret_cast<const unsigned long long *>(a.ctl) + i);
        if (threadIdx.x == 0) s.c.err = 0;
    }
    __syncthreads();
    while (ok && !s.c.done) {
        const int L = s.c.level;
        Level &l = x.slots->level[L % 3], &next = x.slots->level[(L + 1) % 3];
        const MsStep p = ms_step(a, L, L - s.c.base, s.c.tmask, true);
        long long *rec = first && s.c.gtrace_on && L < kGTraceCap ? a.gtrace + (int64_t)L * kGTraceW : nullptr;
        if (rec) rec[0] = (long long)globaltimer_ns();
        // the next level's counters: read last at level L - 2, and every block
        // has passed a barrier since
        if (first) next = Level{};
        ok = s.c.dir == ALB_DIR_TOPDOWN ? level_down(a, x, s, p, l, next) : level_up(a, x, s, p, l);
        if (!ok) break;
        if (first && L == 0) x.slots->level[3] = Level{};
        if (rec) {
            const MsCtl &c = s.c;
            rec[1] = (long long)globaltimer_ns();
            rec[2] = c.dir == ALB_DIR_TOPDOWN
                         ? (long long)(20 * c.nf + 16 * c.mf + 16 * (int64_t)s.sum.n)
                         : (long long)s.sum.bytes + 8 * a.npad + 8 * a.nwords;
            rec[3] = c.dir;
            rec[4] = c.nf;
            rec[5] = c.mf;
            rec[6] = c.nu;
            rec[7] = c.mu;
        }
        __syncthreads();
        if ((threadIdx.x >> 5) == kCtl) end_level(a, s);
        __syncthreads();
        if (s.c.need_flush) break;
    }
    if (blockIdx.x != 0) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        const int32_t err = *(volatile int32_t *)&a.ctl->err;
        if (err) s.c.err = err;
        if (!ok) s.c.done = s.c.need_flush = 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (int)(sizeof(MsCtl) / 8); i += kThreads) {
        const unsigned long long v = reinterpret_cast<const unsigned long long *>(&s.c)[i];
        reinterpret_cast<unsigned long long *>(a.ctl)[i] = v;
        reinterpret_cast<unsigned long long *>(x.result)[i] = v;
    }
}

}  // namespace

alb_status ms_grid_launch(const alb_graph *g, const MsArgs &a, const MsInit &in,
                          const MsGridArgs &x, cudaStream_t st) {
    MsArgs aa = a;
    MsInit ii = in;
    MsGridArgs xx = x;
    void *args[] = {&aa, &ii, &xx};
    ALB_CK(cudaFuncSetAttribute(k_ms_grid, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxL1));
    ALB_CK(cudaLaunchCooperativeKernel((void *)k_ms_grid, dim3((unsigned)g->num_sms), dim3(kThreads),
                                       args, 0, st));
    return ALB_OK;
}

}  // namespace alb
