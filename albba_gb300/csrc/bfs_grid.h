// Single-root BFS as one cooperative kernel (bfs_grid.cu).
#pragma once

#include "dev.cuh"
#include "graph.h"

namespace alb {

constexpr int kScatterThreads = 256;

// Counters of the running levels, by level modulo 3, cleared by the kernel.
struct GridSlots {
    unsigned long long acc[3][16];   // sums; a row of its own for each level
    unsigned long long word[3][16];  // list levels' arrival words, a line each
};

struct GridArgs {
    GridSlots *slots;
    const int4 *vrec;  // push rows' records, where list levels matter (row_recs_launch)
    int64_t max_out;  // longest push row (0: not known)
    int64_t m_out;
    int32_t sym;      // push and pull rows are the same
    int32_t exact;    // learned directions as the host-driven loop's (list_level)
    BfsCtl *result;   // page-locked: level, done, err, levels_*, reached, edges
    int32_t list_cap;  // set by grid_launch
};

// Whether the call runs as the cooperative kernel (traces, host-driven levels
// and the pull without bypass do not).
bool grid_takes(const alb_graph *g, const alb_bfs_opts &o, const BfsArgs &a);
alb_status grid_launch(const alb_graph *g, const BfsArgs &a, const InitParams &in,
                       const GridArgs &x, cudaStream_t st);

// Graphs whose longest row has at most this many entries (grids, uniform random
// graphs: long searches with small frontiers) get a 16-byte record per
// position, so that a claim costs one access where it cost three. On the grid
// of 2^24 vertices (503 levels) every such access misses L2 and the TLB.
constexpr int32_t kRecMaxDeg = 64;
alb_status row_recs_launch(const alb_graph *g, const BfsArgs &a, int4 *vrec, cudaStream_t st);

// Levels and parents by position into original ids (either may be null).
// ALB_ERR_UNSUPPORTED: the sort windows do not make tiles of whole 16 bytes.
alb_status scatter_launch(const alb_graph *g, const BfsArgs &a, int32_t *level, int32_t *parent,
                          cudaStream_t st);

}  // namespace alb
