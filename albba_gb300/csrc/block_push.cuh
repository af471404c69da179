// Top-down push of one block over the set bits of a bitmap in its shared
// memory: the rows of kPushWords words at a time are listed with the number of
// edges before each, and the list's edges are dealt out evenly to the block's
// threads, whatever the rows' lengths (a row per warp leaves a hub's edges to
// one warp; a binary search per edge is bound by shared-memory reads).
#pragma once

#include "dev.cuh"

namespace alb {

constexpr int kPushWords = 64, kPushRows = kPushWords * 32;

struct PushLists {
    int nlist;
    int32_t list[kPushRows], list_st[kPushRows], list_off[kPushRows + 1];
    int32_t warp_rows[32], warp_edges[32];
};

// Bits of F's words [from, to), span words at a time (as many bits as
// kPushRows at most in each). row(u, st, d, ou): first edge, edge count and
// source id of position u (d = 0: not pushed). push(v, ou): four edges per
// lane (v[k] < 0: none). kT: threads of the block, all of which call.
template <int kT, class Row, class Push>
__device__ __forceinline__ void block_push(PushLists &s, const uint32_t *F, int from, int to,
                                           int span, const int32_t *pcol, Row row, Push push) {
    constexpr int kW = kT / 32, kRowsPer = kPushRows / kT;
    const int lane = lane_id(), wib = threadIdx.x >> 5;
    for (int b = from; b < to; b += span) {
        if (threadIdx.x == 0) s.nlist = 0;
        __syncthreads();
        for (int w = b + (int)threadIdx.x; w < min(to, b + span); w += kT) {
            uint32_t m = F[w];
            int at = m ? atomicAdd(&s.nlist, __popc(m)) : 0;
            for (; m; m &= m - 1) s.list[at++] = w * 32 + __ffs(m) - 1;
        }
        __syncthreads();
        const int rows = s.nlist;
        if (rows == 0) continue;
        // rows kRowsPer i .. of thread i; those without edges are dropped
        int32_t st[kRowsPer], d[kRowsPer], ou[kRowsPer], nd = 0, nr = 0;
#pragma unroll
        for (int k = 0; k < kRowsPer; k++) {
            const int i = kRowsPer * (int)threadIdx.x + k;
            d[k] = 0;
            if (i >= rows) continue;
            row(s.list[i], st[k], d[k], ou[k]);
            nd += d[k];
            nr += d[k] > 0;
        }
        int32_t at = warp_inclusive_scan(nr), off = warp_inclusive_scan(nd);
        if (lane == 31) {
            s.warp_rows[wib] = at;
            s.warp_edges[wib] = off;
        }
        __syncthreads();
        const int32_t r_inc = warp_inclusive_scan(lane < kW ? s.warp_rows[lane] : 0),
                      e_inc = warp_inclusive_scan(lane < kW ? s.warp_edges[lane] : 0);
        const int32_t R = __shfl_sync(kFull, r_inc, 31), E = __shfl_sync(kFull, e_inc, 31);
        const int32_t r_b = __shfl_sync(kFull, r_inc, (wib + 31) & 31),
                      e_b = __shfl_sync(kFull, e_inc, (wib + 31) & 31);
        at += (wib ? r_b : 0) - nr;
        off += (wib ? e_b : 0) - nd;
#pragma unroll
        for (int k = 0; k < kRowsPer; k++) {
            if (!d[k]) continue;
            s.list[at] = ou[k];
            s.list_st[at] = st[k] - off;  // edge e of the list is pcol[st + e]
            s.list_off[at] = off;
            off += d[k];
            at++;
        }
        __syncthreads();
        // each warp takes a run of edges, 32 at a time (four times over before
        // the pushes): the rows that start among them make a bit mask, and a
        // lane's row is the mask's bits up to it further on
        const int32_t run = ((E + kW - 1) / kW + 31) & ~31;
        const int32_t e_end = min(E, run * (wib + 1));
        int j = 0;
        if (run * wib < E)
            for (int step = kPushRows / 2; step > 0; step >>= 1)
                if (j + step < R && s.list_off[j + step] <= run * wib) j += step;
        for (int32_t eb = run * wib; eb < e_end; eb += 128) {
            int32_t v[4];
            uint32_t ou4[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int32_t e0 = eb + 32 * k, e = e0 + lane;
                const int32_t q = j + 1 + lane, rel = q < R ? s.list_off[q] - e0 : 32;
                const unsigned starts = __reduce_or_sync(kFull, rel < 32 ? 1u << rel : 0u);
                const int r = j + __popc(starts & (lanemask_lt() | (1u << lane)));
                v[k] = -1;
                ou4[k] = 0;
                if (e < e_end) {
                    v[k] = __ldg(pcol + s.list_st[r] + e);
                    ou4[k] = (uint32_t)s.list[r];
                }
                j += __popc(starts);
            }
            push(v, ou4);
        }
        __syncthreads();
    }
}

}  // namespace alb
