// Single-root BFS of a small graph as one launch (bfs_cluster.cu).
#pragma once

#include "dev.cuh"
#include "graph.h"

namespace alb {

// Largest graph (vertices) the cluster kernel takes. Against the cooperative
// kernel on all SMs (bfs_grid.cu), us a call, Beamer / learned: R-MAT edge
// factor 16, n = 65,536: 65 / 87 against 77 / 91, at 131,072: 87 / 135 against
// 82 / 100; grid of 65,536: 968 / 1,447 against 1,186 / 1,793, of 131,044:
// 1,392 / 1,617 against 1,256 / 1,240; uniform random, mean degree 8, 32,768:
// 62 / 109 against 82 / 84, 65,536: 93 / 149 against 85 / 94.
constexpr int64_t kClusterMaxN = 1 << 16;

// Whether the call runs as one cluster launch. Calls that ask for what only
// the other loops have keep them: per-level traces, host-driven levels, the
// pull without bypass, the test hooks of the device-side waits.
bool cluster_takes(const alb_graph *g, const alb_bfs_opts &o, const BfsArgs &a);

// The whole traversal into d_level / d_parent (original ids, either may be
// null); result (page-locked host memory) receives level, done, err,
// levels_td, levels_bu, reached and edges.
alb_status cluster_launch(const BfsArgs &a, const InitParams &in, int32_t *d_level,
                          int32_t *d_parent, BfsCtl *result, cudaStream_t st);

}  // namespace alb
