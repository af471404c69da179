// Single-root BFS of a small graph as one launch (bfs_cluster.cu).
#pragma once

#include "dev.cuh"
#include "graph.h"

namespace alb {

// Largest graph (vertices) the cluster kernel takes: where the default policy's
// searches of R-MAT and uniform random graphs meet those of the cooperative
// kernel on all SMs (bfs_grid.cu). us a call, cluster against cooperative,
// Beamer; learned: R-MAT edge factor 16, n = 1,024: 37 / 63; 62 / 68, 65,536:
// 71 / 82; 107 / 97, 131,072: 103 / 85; 110 / 87. Uniform random, mean degree 8,
// 32,768: 66 / 86; 115 / 94, 65,536: 90 / 92; 142 / 101, 131,072: 123 / 86; 189 /
// 118. Grids of 65,536: 861 / 1,097; 1,300 / 1,585, of 131,044: 1,258 / 1,404; 1,393
// / 1,563. The learned policy pushes more, and so crosses at fewer vertices;
// where there are many edges a vertex it is sent away (cluster_takes).
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
