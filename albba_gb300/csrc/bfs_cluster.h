// Single-root BFS of a small graph as one launch (bfs_cluster.cu).
#pragma once

#include "dev.cuh"
#include "graph.h"

namespace alb {

// Largest graph (vertices) the cluster kernel takes: three bitmaps of it fit
// in one CTA's shared memory beside the kernel's 75 KB. In place of the
// persistent kernel it is taken up to half of that: at 262,144 vertices, 16 SMs
// lose to 152 where the learned policy pushes dense frontiers (R-MAT 194
// against 148 us, uniform random 272 against 216), at 131,072 they win (125
// against 137, 189 against 211). The CUDA-graph loop loses at either size.
constexpr int64_t kClusterMaxN = 1 << 18;
constexpr int64_t kClusterMaxPersistent = 1 << 17;

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
