// Batched BFS as one cooperative kernel (ms_grid.cu).
#pragma once

#include "graph.h"
#include "ms.cuh"

namespace alb {

// Counters of the running levels, by level modulo 3 (acc[3]: the roots), and
// the grid barrier's arrivals. All zero before the first launch; the kernel
// leaves them fit for the next one unless it gave up.
struct MsSlots {
    unsigned long long bar, pad[15];
    struct Level {
        MsSums acc;
        // long-row and long-frontier-row counter, queue length; the pushed
        // roots' long-row counter and queue length; word counter
        unsigned long long nbig, qn, pbig, pqn, work, pad[3];
    } level[4];
};

struct MsGridArgs {
    MsSlots *slots;
    MsCtl *result;  // page-locked
    int32_t resume;  // go on from the control block after a flush
    uint64_t barrier_ns;
    int32_t withhold_level, withhold_block;
};

alb_status ms_grid_launch(const alb_graph *g, const MsArgs &a, const MsInit &in,
                          const MsGridArgs &x, cudaStream_t st);

}  // namespace alb
