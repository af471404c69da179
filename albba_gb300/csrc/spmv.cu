// fp64 SELL-C-sigma SpMV, y = A x.
//
// Reference: kernel_SELLCS_DFC (bfs/src/bfs_par_kernels.c:8-53) over the
// matrix built by convert_csr_to_sellcs_dfc (bfs/src/sparse_matrix.c:
// 523-623): rows sorted by length inside sigma windows, C = 256 lanes per
// slice, one column op per entry index, and per lane a fused multiply-add
// (_vel_vfmadd_vvvvl) of value * x[column] into an accumulator that starts at
// 0; y[row] is that accumulator. Entry k of a row is handled by column op k,
// so every row sums its entries in CSR order with one rounding per entry --
// the result is fixed by the CSR alone, whatever C, sigma or the lanes are.
//
// GB300 layout: the same sigma-window order (the library's device sort), C =
// 32 rows per slice so that one warp owns a slice and lane r its row r, and
// the 4-interleaved layout of the BFS's SELL: group g of slice s holds entries
// 4g..4g+3 of every row, lane r's four column ids at col[off + 128 g + 4 r]
// (one int4 per lane, 512 contiguous bytes per warp) and its four values at
// the same index of val (two double2 per lane, 1 KB per warp). Entries are
// kept exactly as given (diagonal and repeated entries included); padding is
// never read: a lane stops at its row's length, so the fma chain is the
// reference's, bit for bit.
//
// Rows longer than kSpLong entries keep an empty SELL row: in a slice such a
// row's lane waits on one group of x gathers at a time and holds its warp for
// milliseconds. They are kept in a list of their own, longest first. The
// chain of fused multiply-adds is what makes y bit-identical, and a dependent
// fp64 fma costs about 115 cycles on GB300 (for one active lane as for 32), so
// the list is summed in two ways: most lane per row (k_spmv_long: 32 chains side
// by side), and where a few are much longer those CTA per row with the chain's
// steps found 256 at a time as integers (k_spmv_hub, chain.cuh; hub_rows says
// which), so that the longest row's chain no longer sets the launch's length.
// Each runs on a stream of its own beside the slices. R-MAT scale 22, edge factor
// 16, signed values: 9.45 ms with every long row lane per row, 1.9 to 2.2 ms now;
// with positive values 0.85 ms. The longest row alone takes 6.6 ns an entry, and
// about twice that beside the others on its SM.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <utility>
#include <vector>

#include "chain.cuh"
#include "graph.h"
#include "ingest.h"
#include "scan.cuh"

struct alb_sellmat {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr, side2 = nullptr;  // hubs, long rows: beside the slices
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, fork = nullptr, join = nullptr, join2 = nullptr;
    int64_t n = 0, nnz = 0, nslices = 0, stored = 0;
    int32_t sigma = 0;
    int32_t num_sms = 0;
    int32_t wslices = 1;           // slices per sort window where windows are whole slices, else 1
    int32_t *perm = nullptr;       // position -> row
    int32_t *deg = nullptr;        // row length by position
    int64_t *slice_off = nullptr;  // first entry of each slice (multiple of 128)
    int32_t *col = nullptr;        // 4-interleaved column ids
    double *val = nullptr;         // values, same layout
    double *dx = nullptr, *dy = nullptr;  // staging for host vectors
    int64_t nlong = 0;             // rows longer than kSpLong
    int64_t nhub = 0;              // the first of them, CTA per row (hub_rows)
    int32_t *lrow = nullptr;       // their row ids, longest first
    int64_t *lptr = nullptr;       // first entries in lcol / lval: of each hub (a multiple of
                                   // 8), then of each slice of 32 other long rows (of 128)
    int32_t *llen = nullptr;       // their lengths
    int32_t *lcol = nullptr;       // their entries: hubs row by row, the others interleaved
    double *lval = nullptr;
};

namespace alb {
namespace {

constexpr int kSpC = 32;
constexpr int32_t kSpLong = 256;  // longer rows leave the slices

unsigned blocks_for(int64_t work, int block) {
    int64_t g = (work + block - 1) / block;
    return (unsigned)(g < 1 ? 1 : g);
}

__global__ void k_lengths(int64_t n, const int64_t *rp, int32_t *len) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r < n) len[r] = (int32_t)(rp[r + 1] - rp[r]);
}

__global__ void k_sp_positions(int64_t n, const int32_t *perm, const int32_t *len, int32_t *deg) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p < n) deg[p] = len[perm[p]];
}

// Slice sizes: 32 rows x the longest row rounded up to 4.
__global__ void k_sp_sizes(int64_t n, int64_t nslices, const int32_t *deg, int64_t *ssize) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= nslices) return;
    int32_t w = 0;
    for (int r = 0; r < kSpC; r++) {
        const int64_t p = s * kSpC + r;
        if (p < n && deg[p] <= kSpLong) w = max(w, deg[p]);
    }
    ssize[s] = (int64_t)kSpC * ((w + 3) & ~3);
}

// One thread per position: copies its row's entries (CSR order) into the
// interleaved slots; the slice's remaining groups of the row are padded with
// column 0 and value 0 (never read).
__global__ void k_sp_fill(int64_t n, int64_t npad, const int32_t *perm, const int32_t *deg,
                          const int64_t *slice_off, const int64_t *rp, const int32_t *col,
                          const double *val, int32_t *scol, double *sval) {
    const int64_t str = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npad; p += str) {
        const int64_t s = p / kSpC;
        const int64_t base = slice_off[s] + 4 * (p % kSpC);
        const int32_t ng = (int32_t)((slice_off[s + 1] - slice_off[s]) / (4 * kSpC));
        const int32_t d = p < n && deg[p] <= kSpLong ? deg[p] : 0;
        const int64_t b = p < n ? rp[perm[p]] : 0;
        for (int32_t g = 0; g < ng; g++) {
            int32_t c4[4];
            double v4[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int32_t e = 4 * g + k;
                c4[k] = e < d ? col[b + e] : 0;
                v4[k] = e < d ? val[b + e] : 0.0;
            }
            const int64_t at = base + (int64_t)g * 4 * kSpC;
            *reinterpret_cast<int4 *>(scol + at) = make_int4(c4[0], c4[1], c4[2], c4[3]);
            reinterpret_cast<double2 *>(sval + at)[0] = make_double2(v4[0], v4[1]);
            reinterpret_cast<double2 *>(sval + at)[1] = make_double2(v4[2], v4[3]);
        }
    }
}

// Warp per slice, lane per row. While a group's four fmas run (a dependent
// fma takes about 115 cycles), the next group's x gathers and the columns and
// values after them are in flight.
// Slices are taken rank by rank: the first (longest rows) of every sort
// window, then every window's second, and so on. In index order a grid stride
// that is a multiple of the slices per window hands one warp the longest
// slice of window after window: at R-MAT scale 22 that warp set the kernel's
// 1.66 ms. Small blocks: a matrix of a few hundred slices then spreads over
// the SMs, whose fp64 pipe takes 16 cycles per warp and fma.
constexpr int kSpBlock = 128;

__global__ void __launch_bounds__(kSpBlock)
    k_spmv(int64_t n, int64_t nslices, int32_t wslices, const int32_t *perm, const int32_t *deg,
           const int64_t *slice_off, const int32_t *col, const double *val, const double *x,
           double *y) {
    const int lane = threadIdx.x & 31;
    const uint32_t w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const uint64_t pol = l2_evict_first();
    const uint32_t nwin = (uint32_t)((nslices + wslices - 1) / wslices);
    const uint32_t total = nwin * (uint32_t)wslices;  // below 2^26 + sigma / 32
    for (uint32_t i = w0; i < total; i += nw) {
        const uint32_t rank = i / nwin;
        const int64_t s = (int64_t)(i - rank * nwin) * wslices + rank;
        if (s >= nslices) continue;  // the last window may be short
        const int64_t p = s * kSpC + lane;
        const int32_t dr = p < n ? __ldg(deg + p) : 0;
        const bool mine = p < n && dr <= kSpLong;  // long rows: k_spmv_long
        const int32_t d = mine ? dr : 0;
        const int32_t ng = (d + 3) >> 2;
        const int64_t base = __ldg(slice_off + s) + 4 * lane;
        const int4 *cp = reinterpret_cast<const int4 *>(col + base);
        const double2 *vp = reinterpret_cast<const double2 *>(val + base);
        double acc = 0.0;
        int4 c = make_int4(0, 0, 0, 0);
        double2 va = make_double2(0.0, 0.0), vb = va;
        double xv[4];
        // a group's gathers, c being its columns (padding is not followed)
        auto gather = [&](const int4 &q, int32_t left, double (&v)[4]) {
            v[0] = left > 0 ? __ldg(x + q.x) : 0.0;
            v[1] = left > 1 ? __ldg(x + q.y) : 0.0;
            v[2] = left > 2 ? __ldg(x + q.z) : 0.0;
            v[3] = left > 3 ? __ldg(x + q.w) : 0.0;
        };
        if (ng > 0) {
            c = ld_stream(cp, pol);
            va = __ldcs(vp);
            vb = __ldcs(vp + 1);
        }
        gather(c, d, xv);
        if (ng > 1) c = ld_stream(cp + kSpC, pol);
        for (int32_t g = 0; g < ng; g++) {
            const int32_t left = d - 4 * g;
            double2 van = va, vbn = vb;
            double xn[4];
            gather(c, left - 4, xn);
            if (g + 1 < ng) {
                van = __ldcs(vp + (int64_t)(g + 1) * 2 * kSpC);
                vbn = __ldcs(vp + (int64_t)(g + 1) * 2 * kSpC + 1);
            }
            if (g + 2 < ng) c = ld_stream(cp + (int64_t)(g + 2) * kSpC, pol);
            acc = fma(va.x, xv[0], acc);
            if (left > 1) acc = fma(va.y, xv[1], acc);
            if (left > 2) acc = fma(vb.x, xv[2], acc);
            if (left > 3) acc = fma(vb.y, xv[3], acc);
            va = van;
            vb = vbn;
#pragma unroll
            for (int k = 0; k < 4; k++) xv[k] = xn[k];
        }
        if (mine) y[__ldg(perm + p)] = acc;
    }
}

// Lane per long row, 32 rows of similar length per warp (longest first),
// interleaved as in a slice. Bound: the longest row's chain, 52 to 75 ns per
// entry. Every load has to land within the chain time of the groups before
// it: columns are requested 2 kLd groups of four entries ahead, values and x
// gathers kLd groups (kLd x 4 fmas) ahead, all in registers. Eight groups (2
// us) where the matrix has no hub rows; four beside hubs, whose CTAs (and the
// slices') then find more registers free. At 4 / 8: 900 rows of 4,000 entries
// 271 / 241 us, 3,000 of 30,000 2,314 / 1,974; R-MAT scale 22, which has hubs,
// 1,910 / 1,961. Rings in shared memory (cp.async) left the SM's L1 too small
// to hold the gathers in flight: 1.5 ms at R-MAT scale 22 instead of 0.7, and 6
// ms with the slices' gathers beside it.
constexpr int kSpLongBlock = 32;  // one warp per CTA
constexpr int kLb = 8;            // hub rows are padded to this many entries

template <int kLd>
__global__ void __launch_bounds__(kSpLongBlock)
    k_spmv_long(int64_t nrows, const int32_t *lrow, const int64_t *moff, const int32_t *llen,
                const int32_t *lcol, const double *lval, const double *x, double *y) {
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * kSpC + lane;
    const int32_t len = i < nrows ? llen[i] : 0;
    const int32_t ng = (len + 3) >> 2;
    const int64_t base = moff[blockIdx.x] + 4 * lane;
    const int4 *cp = reinterpret_cast<const int4 *>(lcol + base);
    const double2 *vp = reinterpret_cast<const double2 *>(lval + base);
    int4 c[kLd];
    double2 va[kLd], vb[kLd];
    double xv[kLd][4];
    // group g: its columns into c[j]; its values and gathers (padding points
    // at x[0] and is not used)
    auto cols = [&](int j, int32_t g) {
        if (g < ng) c[j] = __ldcs(cp + (int64_t)g * kSpC);
    };
    auto fetch = [&](int j, int32_t g) {
        if (g >= ng) return;
        va[j] = __ldcs(vp + (int64_t)g * 2 * kSpC);
        vb[j] = __ldcs(vp + (int64_t)g * 2 * kSpC + 1);
        xv[j][0] = __ldg(x + c[j].x);
        xv[j][1] = __ldg(x + c[j].y);
        xv[j][2] = __ldg(x + c[j].z);
        xv[j][3] = __ldg(x + c[j].w);
    };
#pragma unroll
    for (int j = 0; j < kLd; j++) cols(j, j);
#pragma unroll
    for (int j = 0; j < kLd; j++) {
        fetch(j, j);
        cols(j, kLd + j);
    }
    double acc = 0.0;
    for (int32_t g0 = 0; g0 < ng; g0 += kLd) {
#pragma unroll
        for (int j = 0; j < kLd; j++) {
            const int32_t g = g0 + j, left = len - 4 * g;
            if (left > 0) acc = fma(va[j].x, xv[j][0], acc);
            if (left > 1) acc = fma(va[j].y, xv[j][1], acc);
            if (left > 2) acc = fma(vb[j].x, xv[j][2], acc);
            if (left > 3) acc = fma(vb[j].y, xv[j][3], acc);
            fetch(j, g + kLd);
            cols(j, g + 2 * kLd);
        }
    }
    if (i < nrows) y[lrow[i]] = acc;
}

// CTA per hub row, 256 entries a tile, the chain's steps as integer prefix
// sums (chain.cuh). Warp 0 walks the chain. Warps 1 to 3 load: each takes
// every third tile, keeps its columns six tiles and its values and x gathers
// three tiles ahead in registers, and hands values, x and products over in
// shared memory. Warps 4 to 6 scan the next tile for the exponent the
// sum has now and its two neighbours. One block barrier a tile. Bound: warp
// 0's latency on the longest row -- a look through a tile's prefixes, and for
// each entry where the sum leaves its binade (a random walk of N signed terms
// does so about 8 sqrt(N) times) one fma and another look; the sum mostly
// moves between neighbouring binades, so the scans for them are at hand, and
// warp 0 scans for any other exponent itself (the last two are kept). After a
// step that leaves the sum small against its term, or a run of fewer than
// kRunSeq entries, kRunSeq are done by fma: a look costs as much as six, and
// there the next would find little (150 rows of 1,000 signed terms 87 -> 78 us,
// R-MAT scale 22 2,307 -> 2,205).
constexpr int kTile = 256, kPer = kTile / 32;  // lane l: entries 8l .. 8l + 7
constexpr int kHubFeed = 3, kHubScan = 3;      // warps that load, that scan
constexpr int kHubThreads = 32 * (1 + kHubFeed + kHubScan);
constexpr int kRunSeq = 8;
constexpr int kNoGuess = -2;  // near no exponent

struct HubTile {
    double v[kPer][32], x[kPer][32];
    int64_t h[kPer][32];  // the exact products (ChainTerm)
    int16_t e[kPer][32];
};

// Tiles first, first + kHubFeed, ... of a row, one feeding warp.
struct HubFeed {
    const int32_t *lcol;
    const double *lval, *x;
    int64_t at, end;  // this lane's first entry of the tile held; the row's end
    int32_t c[kPer];  // columns of the tile after the held one
    double v[kPer], xv[kPer];

    __device__ __forceinline__ void cols(int64_t e) {
        if (e >= end) return;  // rows are padded to kPer: a lane's block is whole or absent
        const int4 *q = reinterpret_cast<const int4 *>(lcol + e);
        const int4 a = __ldcs(q), b = __ldcs(q + 1);
        c[0] = a.x, c[1] = a.y, c[2] = a.z, c[3] = a.w;
        c[4] = b.x, c[5] = b.y, c[6] = b.z, c[7] = b.w;
    }
    __device__ __forceinline__ void fetch() {
        if (at >= end) return;
        const double2 *q = reinterpret_cast<const double2 *>(lval + at);
#pragma unroll
        for (int h = 0; h < kPer / 2; h++) {
            const double2 w = __ldcs(q + h);
            v[2 * h] = w.x, v[2 * h + 1] = w.y;
        }
#pragma unroll
        for (int k = 0; k < kPer; k++) xv[k] = __ldg(x + c[k]);
    }
    __device__ __forceinline__ void start(int64_t e) {
        at = e;
#pragma unroll
        for (int k = 0; k < kPer; k++) c[k] = 0, v[k] = xv[k] = 0.0;
        cols(at);
        fetch();
        cols(at + kHubFeed * kTile);
    }
    // the held tile goes to shared memory, the next one is requested
    __device__ __forceinline__ void hand(HubTile &t) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            t.v[k][lane] = v[k];
            t.x[k][lane] = xv[k];
            const bool in = at + k < end;  // an entry past the end adds nothing
            const ChainTerm p = chain_term(in ? (uint64_t)__double_as_longlong(v[k]) : 0,
                                           in ? (uint64_t)__double_as_longlong(xv[k]) : 0);
            t.h[k][lane] = p.h;
            t.e[k][lane] = (int16_t)p.e;
        }
        at += kHubFeed * kTile;
        fetch();
        cols(at + kHubFeed * kTile);
    }
};

// Prefix sums of k over a tile, up to and with each entry, for one exponent.
struct HubSums {
    int64_t P[kPer][32];
    uint8_t stop[32];  // each lane's entries that end a run: too large, or a tie
};

// One warp scans a tile for exponent E.
__device__ __forceinline__ void hub_scan(const HubTile &T, int E, HubSums &out) {
    const int lane = threadIdx.x & 31;
    unsigned stop = 0;
    int64_t q[kPer];
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        bool st;
        q[k] = chain_round(T.h[k][lane], T.e[k][lane], E, st);
        stop |= st ? 1u << k : 0u;
    }
#pragma unroll
    for (int k = 1; k < kPer; k++) q[k] += q[k - 1];
    const int64_t ex = warp_inclusive_scan(q[kPer - 1]) - q[kPer - 1];
#pragma unroll
    for (int k = 0; k < kPer; k++) out.P[k][lane] = q[k] + ex;
    out.stop[lane] = (uint8_t)stop;
}

__global__ void __launch_bounds__(kHubThreads)
    k_spmv_hub(const int32_t *lrow, const int64_t *lptr, const int32_t *llen, const int32_t *lcol,
               const double *lval, const double *x, double *y) {
    __shared__ HubTile s_t[3];
    // by tile parity, exponents guess - 1 .. guess + 1; then warp 0's own two
    __shared__ HubSums s_h[2 * kHubScan + 2];
    // by tile parity: exponent of the sum after the tile; the tile's guess
    __shared__ int s_E[2], s_guess[2];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t len = llen[blockIdx.x];
    const int64_t beg = lptr[blockIdx.x];
    const int64_t ntile = (len + kTile - 1) / kTile;
    HubFeed feed;
    if (wib > 0 && wib <= kHubFeed) {
        feed.lcol = lcol;
        feed.lval = lval;
        feed.x = x;
        feed.end = beg + len;
        feed.start(beg + (wib - 1) * kTile + kPer * lane);
        if (wib <= 2) feed.hand(s_t[wib - 1]);
    }
    if (threadIdx.x == 0) s_E[0] = s_E[1] = s_guess[0] = s_guess[1] = kNoGuess;
    double acc = 0.0;
    for (int64_t t = 0; t < ntile; t++) {
        __syncthreads();  // tiles t and t + 1 and tile t's scans are in place
        if (wib > kHubFeed) {
            const int E = s_E[(t + 1) & 1];  // of the sum after tile t - 1
            // (a zero or subnormal sum has no scans, not even of exponent 1)
            const bool scans = t + 1 < ntile && E > 0;
            if (scans)
                hub_scan(s_t[(t + 1) % 3], E + wib - kHubFeed - 2,
                         s_h[((t + 1) & 1) * kHubScan + wib - kHubFeed - 1]);
            if (wib == kHubFeed + 1 && lane == 0) s_guess[(t + 1) & 1] = scans ? E : kNoGuess;
            continue;
        }
        if (wib > 0) {
            if ((t + 2) % kHubFeed == wib - 1 && t + 2 < ntile) feed.hand(s_t[(t + 2) % 3]);
            continue;
        }
        const HubTile &T = s_t[t % 3];
        const int guess = s_guess[t & 1];
        const int cnt = (int)min((int64_t)kTile, len - t * kTile);
        const unsigned here = cnt - kPer * lane >= kPer ? 0xFFu
                              : cnt <= kPer * lane      ? 0u
                                                        : (1u << (cnt - kPer * lane)) - 1u;
        const int ahead = (int)(t & 1) * kHubScan + 1 - guess;  // + E: the prepared scan
        int E0 = -1, E1 = -1, last = 0;  // exponents of warp 0's own two; the one used last
        int ep = -4096;                  // biased exponent of the last product done by fma
        int s = 0;                       // entries done
        while (s < cnt) {
            const uint64_t ab = (uint64_t)__double_as_longlong(acc);
            const int E = (int)(ab >> 52) & 0x7FF;
            int run = kRunSeq, got = 0;  // got: entries that the look found
            const bool ready = (unsigned)(E - guess + 1) < 3u;
            // (a scan for an exponent that was not prepared pays only where
            // the sum stands clear of its terms)
            if (chain_runs(E) && (ready || E == E0 || E == E1 || E >= ep + 4)) {
                int h = ahead + E;
                if (!ready) {
                    if (E != E0 && E != E1) {
                        last = E0 < 0 ? 0 : E1 < 0 ? 1 : 1 - last;
                        __syncwarp();
                        hub_scan(T, E, s_h[2 * kHubScan + last]);
                        __syncwarp();
                        if (last) E1 = E;
                        else E0 = E;
                    }
                    last = E == E0 ? 0 : 1;
                    h = 2 * kHubScan + last;
                }
                const HubSums &H = s_h[h];
                // A = base + P (acc > 0) or base - P (acc < 0), less 2^52 + 1 so
                // that an entry's result is inside when its bits 52 and up are 0
                const int64_t sg = (int64_t)ab >> 63;
                const int64_t P0 = s > 0 ? H.P[(s - 1) & 7][(s - 1) >> 3] : 0;
                const int64_t A0 = (int64_t)(ab & ((uint64_t)kChainOne - 1));
                const int64_t base = A0 - 1 - sg - ((P0 ^ sg) - sg);
                unsigned out = H.stop[lane];
#pragma unroll
                for (int k = 0; k < kPer; k++) {
                    const int64_t w = (H.P[k][lane] ^ sg) + base;
                    out |= (uint32_t)((uint64_t)w >> 32) >= 0x00100000u ? 1u << k : 0u;
                }
                const int b0 = s - kPer * lane;  // this lane's entries done
                out &= here & (b0 <= 0 ? 0xFFu : b0 >= kPer ? 0u : 0xFFu << b0);
                // the first entry that ends the run (cnt: none)
                const int f = (int)__reduce_min_sync(
                    kFull, out ? (unsigned)(kPer * lane + __ffs(out) - 1) : (unsigned)cnt);
                got = f - s;
                if (f > s) {  // entries s .. f - 1 (A == 2^53 carries into the exponent)
                    const int64_t w = (H.P[(f - 1) & 7][(f - 1) >> 3] ^ sg) + base + 1;
                    acc = __longlong_as_double(
                        (long long)((ab & ~((uint64_t)kChainOne - 1)) + (uint64_t)w));
                    s = f;
                }
                if (s >= cnt) break;
                run = 1;
            }
            // the entry that ended the run; kRunSeq in all after a short one or
            // where the sum is left small against its term (exponents compared
            // as integers: the fp64 pipe is the chain's)
            ep = T.e[s & 7][s >> 3] - 1023;
            acc = fma(T.v[s & 7][s >> 3], T.x[s & 7][s >> 3], acc);
            s++;
            if (run == 1 && got >= kRunSeq && ((__double2hiint(acc) >> 20) & 0x7FF) >= ep + 2)
                continue;
            const int e = min(cnt, s + kRunSeq - 1);
            double pv[kRunSeq - 1], px[kRunSeq - 1];
#pragma unroll
            for (int r = 0; r < kRunSeq - 1; r++) {
                const int i = min(s + r, kTile - 1);
                pv[r] = T.v[i & 7][i >> 3];
                px[r] = T.x[i & 7][i >> 3];
            }
#pragma unroll
            for (int r = 0; r < kRunSeq - 1; r++)
                if (s + r < e) acc = fma(pv[r], px[r], acc);
            s = e;
        }
        if (lane == 0) s_E[t & 1] = (__double2hiint(acc) >> 20) & 0x7FF;
    }
    if (threadIdx.x == 0) y[lrow[blockIdx.x]] = acc;
}

__global__ void k_sp_long_flags(int64_t n, const int32_t *len, int32_t *flag) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r < n) flag[r] = len[r] > kSpLong ? 1 : 0;
}

__global__ void k_sp_long_scatter(int64_t n, const int32_t *flag, const int64_t *idx,
                                  int32_t *lrow) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r < n && flag[r]) lrow[idx[r]] = (int32_t)r;
}

// Block per slice of 32 long rows (longest first), lane per row, the block's
// warps over the groups of four entries.
__global__ void k_sp_long_fill(int64_t nrows, const int32_t *lrow, const int64_t *moff,
                               const int32_t *llen, const int64_t *rp, const int32_t *col,
                               const double *val, int32_t *lcol, double *lval) {
    const int64_t i = (int64_t)blockIdx.x * kSpC + (threadIdx.x & 31);
    if (i >= nrows) return;
    const int64_t src = rp[lrow[i]], dst = moff[blockIdx.x] + 4 * (threadIdx.x & 31);
    const int32_t len = llen[i];
    for (int32_t g = threadIdx.x >> 5; 4 * g < len; g += blockDim.x >> 5) {
        for (int k = 0; k < 4 && 4 * g + k < len; k++) {
            lcol[dst + (int64_t)g * 4 * kSpC + k] = col[src + 4 * g + k];
            lval[dst + (int64_t)g * 4 * kSpC + k] = val[src + 4 * g + k];
        }
    }
}

// One warp per hub row: its entries copied in CSR order.
__global__ void k_sp_hub_fill(int64_t nlong, const int32_t *lrow, const int64_t *lptr,
                              const int32_t *llen, const int64_t *rp, const int32_t *col,
                              const double *val, int32_t *lcol, double *lval) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = w0; i < nlong; i += nw) {
        const int64_t src = rp[lrow[i]], dst = lptr[i], len = llen[i];
        for (int64_t k = lane; k < len; k += 32) {
            lcol[dst + k] = col[src + k];
            lval[dst + k] = val[src + k];
        }
    }
}

// How many of the long rows (len: their lengths, longest first) have a CTA
// each. Lane per row does 32 rows at once but takes kLaneNs per entry of its
// longest. A hub row's CTA takes 3 ns per entry and, for signed terms, 0.35 us
// at each of the entries that leave the binade: about kHubNs per entry, and no
// more than kHubRootNs times the root of the length, all in all. wave: CTAs that
// run at once (two an SM, by their registers). Where there are more, each takes
// kShareNs per entry and kShareRootNs per root of the time of all SMs together.
// Signed terms are what is reckoned with: x is not known yet.
//
// The line between the two is drawn low, where the longest lane-per-row chain
// ends well before the longest hub's, unless more rows than a wave are above it;
// then at the lowest length whose reckoned time is within a tenth of the best.
// Rows of up to kMixedMost entries are left to the lanes where their values have
// both signs, which mostly means that the terms have (mixed(i): row i's values
// have): 30 rows of 600 take 37 us so and 51 as hubs, of 1,000 59 and 80 (17 and 19
// with positive terms). us, signed / positive terms: 100,000 rows of 1,000 entries take 418 lane
// per row and 15,199 / 3,926 as hubs, 900 of 4,000 241 and 517 / 80, 600 of 30,000
// 1,950 and 1,516 / 300, 150 of 1,000 59 and 81 / 20; R-MAT scale 22 (longest row
// 163,186) 2.29 / 0.85 ms with the line at 12 sqrt(N), 2.22 / 0.81 at 25 and 4.10 /
// 1.25 at 6, scale 16 (10,000) 0.34 / 0.07, 0.34 / 0.12 and 0.34 / 0.06.
constexpr double kLaneNs = 58, kHubNs = 80, kHubRootNs = 4400, kShareNs = 0.032, kShareRootNs = 4.8;
constexpr int32_t kMixedMost = 1000;

template <class Mixed>
int64_t hub_rows(const std::vector<int32_t> &len, int64_t wave, Mixed mixed) {
    auto above = [&](double t) -> int64_t {  // rows longer than t
        return std::lower_bound(len.begin(), len.end(), (int32_t)t, std::greater<int32_t>()) -
               len.begin();
    };
    const double longest = len[0], low = std::max((double)kSpLong, 12.0 * std::sqrt(longest));
    if (above(low) <= wave) {
        for (int64_t i = above(kMixedMost); i < above(low); i++)
            if (mixed(i)) return above(std::max(low, (double)kMixedMost));
        return above(low);
    }
    auto alone = [](double n) { return std::min(kHubNs * n, kHubRootNs * std::sqrt(n)); };
    std::vector<double> all(1, 0.0);  // all[k]: what the first k rows take of all SMs
    for (int64_t i = 0; i < above(low); i++)
        all.push_back(all.back() + kShareNs * len[i] + kShareRootNs * std::sqrt((double)len[i]));
    std::vector<std::pair<int64_t, double>> line;  // rows above it, time
    for (double t = low;; t *= 1.25) {
        const int64_t k = above(t);
        double ns = k < (int64_t)len.size() ? kLaneNs * len[(size_t)k] : 0.0;
        if (k > 0) ns = std::max(ns, alone(longest));
        if (k > wave) ns = std::max(ns, all[(size_t)k] + alone(len[(size_t)k - 1]) / 2);
        line.emplace_back(k, ns);
        if (k == 0) break;
    }
    double best = line[0].second;
    for (const auto &l : line) best = std::min(best, l.second);
    for (const auto &l : line)
        if (l.second <= 1.1 * best) return l.first;
    return 0;
}

alb_status build(alb_sellmat *m, const int64_t *rowptr, const int32_t *col, const double *val) {
    const int64_t n = m->n, nnz = m->nnz;
    cudaStream_t st = m->stream;
    int64_t *d_rp = nullptr, *ssize = nullptr;
    int32_t *d_col = nullptr, *len = nullptr;
    double *d_val = nullptr;
    auto tmp_free = [&]() {
        dfree(d_rp);
        dfree(d_col);
        dfree(d_val);
        dfree(len);
        dfree(ssize);
    };
    alb_status rc = [&]() -> alb_status {
        ALB_TRY(dmalloc((void **)&d_rp, sizeof(int64_t) * (size_t)(n + 1), "SpMV row offsets"));
        ALB_TRY(dmalloc((void **)&d_col, sizeof(int32_t) * (size_t)(nnz > 0 ? nnz : 1), "SpMV columns"));
        ALB_TRY(dmalloc((void **)&d_val, sizeof(double) * (size_t)(nnz > 0 ? nnz : 1), "SpMV values"));
        ALB_CK(cudaMemcpyAsync(d_rp, rowptr, sizeof(int64_t) * (size_t)(n + 1),
                               cudaMemcpyHostToDevice, st));
        if (nnz > 0) {
            ALB_CK(cudaMemcpyAsync(d_col, col, sizeof(int32_t) * (size_t)nnz, cudaMemcpyHostToDevice, st));
            ALB_CK(cudaMemcpyAsync(d_val, val, sizeof(double) * (size_t)nnz, cudaMemcpyHostToDevice, st));
        }
        bool sorted = true;
        ALB_TRY(csr_check(n, d_rp, d_col, nnz, st, &sorted));
        m->nslices = (n + kSpC - 1) / kSpC;
        // up to two slices for each quarter of an SM there is nothing to
        // balance, and index order is the faster one (n = 20,011: 11.9
        // against 13.9 us; at 131,072: 14.2 against 12.2)
        m->wslices = m->nslices > 8 * (int64_t)m->num_sms && m->sigma % kSpC == 0
                         ? m->sigma / kSpC : 1;
        const int64_t npad = m->nslices * kSpC;
        ALB_TRY(dmalloc((void **)&len, sizeof(int32_t) * (size_t)n, "SpMV lengths"));
        ALB_TRY(dmalloc((void **)&m->perm, sizeof(int32_t) * (size_t)n, "SpMV order"));
        ALB_TRY(dmalloc((void **)&m->deg, sizeof(int32_t) * (size_t)n, "SpMV degrees"));
        ALB_TRY(dmalloc((void **)&ssize, sizeof(int64_t) * (size_t)(m->nslices + 1), "SpMV sizes"));
        ALB_TRY(dmalloc((void **)&m->slice_off, sizeof(int64_t) * (size_t)(m->nslices + 1),
                        "SpMV slice offsets"));
        k_lengths<<<blocks_for(n, 256), 256, 0, st>>>(n, d_rp, len);
        ALB_CK(cudaGetLastError());
        ALB_TRY(window_order(n, m->sigma, len, m->perm, st));
        k_sp_positions<<<blocks_for(n, 256), 256, 0, st>>>(n, m->perm, len, m->deg);
        k_sp_sizes<<<blocks_for(m->nslices, 256), 256, 0, st>>>(n, m->nslices, m->deg, ssize);
        ALB_CK(cudaGetLastError());
        ALB_TRY(exclusive_scan(ssize, m->slice_off, m->nslices, st));
        ALB_CK(cudaMemcpyAsync(&m->stored, m->slice_off + m->nslices, sizeof(int64_t),
                               cudaMemcpyDeviceToHost, st));
        ALB_CK(cudaStreamSynchronize(st));
        ALB_TRY(dmalloc((void **)&m->col, sizeof(int32_t) * (size_t)(m->stored > 0 ? m->stored : 4),
                        "SpMV SELL columns"));
        ALB_TRY(dmalloc((void **)&m->val, sizeof(double) * (size_t)(m->stored > 0 ? m->stored : 4),
                        "SpMV SELL values"));
        k_sp_fill<<<blocks_for(npad, 256), 256, 0, st>>>(n, npad, m->perm, m->deg, m->slice_off,
                                                          d_rp, d_col, d_val, m->col, m->val);
        ALB_CK(cudaGetLastError());
        // long rows: list (longest first, ordered on the host: a few
        // thousand ids), offsets, entries
        int64_t *idx = nullptr;
        ALB_TRY(dmalloc((void **)&idx, sizeof(int64_t) * (size_t)(n + 1), "SpMV long index"));
        struct Free {
            int64_t *p;
            ~Free() { dfree(p); }
        } free_idx{idx};
        int32_t *flags = nullptr;
        ALB_TRY(dmalloc((void **)&flags, sizeof(int32_t) * (size_t)n, "SpMV long flags"));
        struct Free32 {
            int32_t *p;
            ~Free32() { dfree(p); }
        } free_flags{flags};
        k_sp_long_flags<<<blocks_for(n, 256), 256, 0, st>>>(n, len, flags);
        ALB_CK(cudaGetLastError());
        ALB_TRY(exclusive_scan(flags, idx, n, st));
        ALB_CK(cudaMemcpyAsync(&m->nlong, idx + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        ALB_CK(cudaStreamSynchronize(st));
        if (m->nlong > 0) {
            const int64_t nl = m->nlong;
            ALB_TRY(dmalloc((void **)&m->lrow, sizeof(int32_t) * (size_t)nl, "SpMV long rows"));
            ALB_TRY(dmalloc((void **)&m->lptr, sizeof(int64_t) * (size_t)(nl + 1), "SpMV long offsets"));
            k_sp_long_scatter<<<blocks_for(n, 256), 256, 0, st>>>(n, flags, idx, m->lrow);
            ALB_CK(cudaGetLastError());
            std::vector<int32_t> hrow((size_t)nl);
            ALB_CK(cudaMemcpyAsync(hrow.data(), m->lrow, sizeof(int32_t) * (size_t)nl,
                                   cudaMemcpyDeviceToHost, st));
            ALB_CK(cudaStreamSynchronize(st));
            std::vector<int64_t> hlen((size_t)nl);
            for (int64_t i = 0; i < nl; i++) hlen[(size_t)i] = rowptr[hrow[(size_t)i] + 1] - rowptr[hrow[(size_t)i]];
            std::vector<int64_t> order((size_t)nl);
            for (int64_t i = 0; i < nl; i++) order[(size_t)i] = i;
            std::stable_sort(order.begin(), order.end(),
                             [&](int64_t x, int64_t y) { return hlen[(size_t)x] > hlen[(size_t)y]; });
            std::vector<int32_t> srow((size_t)nl), slen((size_t)nl);
            std::vector<int64_t> sptr((size_t)nl + 1, 0);
            for (int64_t i = 0; i < nl; i++) {
                srow[(size_t)i] = hrow[(size_t)order[(size_t)i]];
                slen[(size_t)i] = (int32_t)hlen[(size_t)order[(size_t)i]];
            }
            auto mixed = [&](int64_t i) {
                const double *b = val + rowptr[srow[(size_t)i]], *e = b + slen[(size_t)i];
                return std::any_of(b, e, [](double v) { return v > 0; }) &&
                       std::any_of(b, e, [](double v) { return v < 0; });
            };
            const int per = resident_blocks((const void *)k_spmv_hub, kHubThreads);
            m->nhub = hub_rows(slen, (int64_t)m->num_sms * std::max(1, per), mixed);
            // hubs: rows one after the other, each padded to kLb entries; the
            // others: slices of 32 rows, as wide as the first (longest) one
            for (int64_t i = 0; i < m->nhub; i++)
                sptr[(size_t)i + 1] = sptr[(size_t)i] + ((slen[(size_t)i] + kLb - 1) / kLb) * kLb;
            int64_t nent = (sptr[(size_t)m->nhub] + 127) & ~127ll;
            const int64_t nmid = (nl - m->nhub + kSpC - 1) / kSpC;
            for (int64_t q = 0; q < nmid; q++) {
                sptr[(size_t)(m->nhub + q)] = nent;
                nent += (int64_t)kSpC * (((int64_t)slen[(size_t)(m->nhub + q * kSpC)] + kLb - 1) / kLb) * kLb;
            }
            ALB_TRY(dmalloc((void **)&m->llen, sizeof(int32_t) * (size_t)nl, "SpMV long lengths"));
            ALB_CK(cudaMemcpyAsync(m->lrow, srow.data(), sizeof(int32_t) * (size_t)nl,
                                   cudaMemcpyHostToDevice, st));
            ALB_CK(cudaMemcpyAsync(m->llen, slen.data(), sizeof(int32_t) * (size_t)nl,
                                   cudaMemcpyHostToDevice, st));
            ALB_CK(cudaMemcpyAsync(m->lptr, sptr.data(), sizeof(int64_t) * (size_t)(nl + 1),
                                   cudaMemcpyHostToDevice, st));
            // padded entries are never summed; zeroed so that the layout is
            // fixed by the CSR alone
            ALB_TRY(dmalloc((void **)&m->lcol, sizeof(int32_t) * (size_t)nent, "SpMV long columns"));
            ALB_TRY(dmalloc((void **)&m->lval, sizeof(double) * (size_t)nent, "SpMV long values"));
            ALB_CK(cudaMemsetAsync(m->lcol, 0, sizeof(int32_t) * (size_t)nent, st));
            ALB_CK(cudaMemsetAsync(m->lval, 0, sizeof(double) * (size_t)nent, st));
            if (m->nhub > 0)
                k_sp_hub_fill<<<blocks_for(m->nhub * 32, 256), 256, 0, st>>>(
                    m->nhub, m->lrow, m->lptr, m->llen, d_rp, d_col, d_val, m->lcol, m->lval);
            if (nmid > 0)
                k_sp_long_fill<<<(unsigned)nmid, 256, 0, st>>>(
                    nl - m->nhub, m->lrow + m->nhub, m->lptr + m->nhub, m->llen + m->nhub, d_rp,
                    d_col, d_val, m->lcol, m->lval);
            ALB_CK(cudaGetLastError());
            // the host vectors must outlive the copies
            ALB_CK(cudaStreamSynchronize(st));
        }
        ALB_CK(cudaStreamSynchronize(st));
        return ALB_OK;
    }();
    tmp_free();
    return rc;
}

void destroy(alb_sellmat *m) {
    if (!m) return;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    dfree(m->perm);
    dfree(m->deg);
    dfree(m->slice_off);
    dfree(m->col);
    dfree(m->val);
    dfree(m->dx);
    dfree(m->dy);
    dfree(m->lrow);
    dfree(m->lptr);
    dfree(m->lcol);
    dfree(m->lval);
    dfree(m->llen);
    if (m->side) cudaStreamSynchronize(m->side);
    if (m->side2) cudaStreamSynchronize(m->side2);
    if (m->ev0) cudaEventDestroy(m->ev0);
    if (m->ev1) cudaEventDestroy(m->ev1);
    if (m->fork) cudaEventDestroy(m->fork);
    if (m->join) cudaEventDestroy(m->join);
    if (m->join2) cudaEventDestroy(m->join2);
    if (m->stream) cudaStreamDestroy(m->stream);
    if (m->side) cudaStreamDestroy(m->side);
    if (m->side2) cudaStreamDestroy(m->side2);
    cudaGetLastError();
    if (prev >= 0) cudaSetDevice(prev);
    delete m;
}

alb_status launch(alb_sellmat *m, const double *d_x, double *d_y, float *us) {
    const int per = resident_blocks((const void *)k_spmv, kSpBlock);
    const int64_t want = (m->nslices + kSpBlock / 32 - 1) / (kSpBlock / 32);  // one slice a warp
    const int64_t cap = (int64_t)(per > 0 ? per : 2) * m->num_sms;
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min(want, cap));
    if (us) ALB_CK(cudaEventRecord(m->ev0, m->stream));
    // the long rows first: their chains are the longest of the launch
    const bool hubs = m->nhub > 0, rest = m->nlong > m->nhub;
    if (hubs || rest) ALB_CK(cudaEventRecord(m->fork, m->stream));
    if (hubs) {
        ALB_CK(cudaStreamWaitEvent(m->side, m->fork, 0));
        k_spmv_hub<<<(unsigned)m->nhub, kHubThreads, 0, m->side>>>(
            m->lrow, m->lptr, m->llen, m->lcol, m->lval, d_x, d_y);
        ALB_CK(cudaGetLastError());
        ALB_CK(cudaEventRecord(m->join, m->side));
    }
    if (rest) {
        ALB_CK(cudaStreamWaitEvent(m->side2, m->fork, 0));
        const auto f = hubs ? k_spmv_long<4> : k_spmv_long<8>;
        f<<<blocks_for(m->nlong - m->nhub, kSpC), kSpLongBlock, 0, m->side2>>>(
            m->nlong - m->nhub, m->lrow + m->nhub, m->lptr + m->nhub, m->llen + m->nhub, m->lcol,
            m->lval, d_x, d_y);
        ALB_CK(cudaGetLastError());
        ALB_CK(cudaEventRecord(m->join2, m->side2));
    }
    k_spmv<<<grid, kSpBlock, 0, m->stream>>>(m->n, m->nslices, m->wslices, m->perm, m->deg,
                                             m->slice_off, m->col, m->val, d_x, d_y);
    ALB_CK(cudaGetLastError());
    if (hubs) ALB_CK(cudaStreamWaitEvent(m->stream, m->join, 0));
    if (rest) ALB_CK(cudaStreamWaitEvent(m->stream, m->join2, 0));
    if (us) {
        ALB_CK(cudaEventRecord(m->ev1, m->stream));
        ALB_CK(cudaEventSynchronize(m->ev1));
        float ms = 0;
        ALB_CK(cudaEventElapsedTime(&ms, m->ev0, m->ev1));
        *us = ms * 1000.0f;
    }
    return ALB_OK;
}

}  // namespace
}  // namespace alb

using namespace alb;

extern "C" {

alb_status alb_sellmat_create(int64_t n, const int64_t *rowptr, const int32_t *col,
                              const double *values, int32_t sigma, alb_sellmat **out) {
    if (!out) return fail(ALB_ERR_INVALID, "alb_sellmat_create: out is NULL");
    *out = nullptr;
    if (n <= 0 || n > INT32_MAX || !rowptr || rowptr[0] != 0 || rowptr[n] < 0 ||
        (rowptr[n] > 0 && (!col || !values)))
        return fail(ALB_ERR_INVALID, "alb_sellmat_create: bad arguments");
    if (sigma < 1 || sigma > 16384)
        return fail(ALB_ERR_UNSUPPORTED, "alb_sellmat_create: sigma %d outside 1..16384", sigma);
    alb_sellmat *m = new alb_sellmat();
    m->n = n;
    m->nnz = rowptr[n];
    m->sigma = sigma;
    cudaError_t e = cudaGetDevice(&m->device);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&m->num_sms, cudaDevAttrMultiProcessorCount, m->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&m->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&m->ev1);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&m->fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&m->join, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->side2, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&m->join2, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        cudaGetLastError();
        destroy(m);
        return fail(ALB_ERR_CUDA, "alb_sellmat_create: %s", cudaGetErrorString(e));
    }
    alb_status rc = build(m, rowptr, col, values);
    if (rc != ALB_OK) {
        destroy(m);
        return rc;
    }
    *out = m;
    return ALB_OK;
}

void alb_sellmat_destroy(alb_sellmat *m) { destroy(m); }

alb_status alb_sellmat_info(const alb_sellmat *m, int64_t *n, int64_t *nnz, int64_t *stored) {
    if (!m) return fail(ALB_ERR_INVALID, "alb_sellmat_info: matrix is NULL");
    if (n) *n = m->n;
    if (nnz) *nnz = m->nnz;
    if (stored) *stored = m->stored;
    return ALB_OK;
}

alb_status alb_sellmat_spmv(alb_sellmat *m, const double *d_x, double *d_y, float *kernel_us) {
    if (!m || !d_x || !d_y) return fail(ALB_ERR_INVALID, "alb_sellmat_spmv: bad arguments");
    ALB_CK(cudaSetDevice(m->device));
    ALB_TRY(launch(m, d_x, d_y, kernel_us));
    ALB_CK(cudaStreamSynchronize(m->stream));
    return ALB_OK;
}

alb_status alb_sellmat_spmv_host(alb_sellmat *m, const double *x, double *y) {
    if (!m || !x || !y) return fail(ALB_ERR_INVALID, "alb_sellmat_spmv_host: bad arguments");
    ALB_CK(cudaSetDevice(m->device));
    if (!m->dx) ALB_TRY(dmalloc((void **)&m->dx, sizeof(double) * (size_t)m->n, "SpMV x"));
    if (!m->dy) ALB_TRY(dmalloc((void **)&m->dy, sizeof(double) * (size_t)m->n, "SpMV y"));
    ALB_CK(cudaMemcpyAsync(m->dx, x, sizeof(double) * (size_t)m->n, cudaMemcpyHostToDevice,
                           m->stream));
    ALB_TRY(launch(m, m->dx, m->dy, nullptr));
    ALB_CK(cudaMemcpyAsync(y, m->dy, sizeof(double) * (size_t)m->n, cudaMemcpyDeviceToHost,
                           m->stream));
    ALB_CK(cudaStreamSynchronize(m->stream));
    return ALB_OK;
}

}  // extern "C"
