// Host-side plans of the PCG kernels: the resident PCG (krylov.cu: which rows a CTA keeps and gathers and how
// its blocks are sliced) and the batched PCG (batch.cu: its sliced copy of the system).
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <vector>

// What a PCG launch leaves for the host, in memory that the host clears before the launch (pcg_result_clear): the
// record is CTA 0's, gaveUp any CTA's.  A CTA that gave up waiting for the others leaves its rows of x unwritten, also
// when CTA 0 has seen the end of the solve.
struct PcgResult {
    int iterations;
    int status;   // -1: not written
    int gaveUp;
    double rr;    // final squared residual norm
    double bb;    // squared RHS norm
};
inline void pcg_result_clear(PcgResult& r) {
    r.status = -1;
    r.gaveUp = 0;
}
inline bool pcg_result_timed_out(const PcgResult& r) { return r.status == -1 || r.gaveUp != 0; }

struct PcgShape {
    int grid = 1, lpr = 32;  // CTAs and lanes per block row
    int copies = 1;          // slot sets of a reduction
    bool cluster = false;    // the grid is one cluster
};

struct PcgResidentPlan {
    PcgShape shape;
    size_t smem = 0;                 // dynamic shared memory of the largest CTA (0: does not fit)
    std::vector<int32_t> haloPtr;    // [CTAs + 1]
    std::vector<int32_t> haloIdx;    // rows outside a CTA's range that its rows couple to
    std::vector<int32_t> groupPtr;   // [CTAs][groups + 1] first step of each group of rows
    std::vector<uint16_t> lcol;      // [blocks] place of a block's column among the CTA's rows and halo
};

void ef_pcg_resident_plan(int vDouble, int nSM, int nNodes, const int32_t* rowPtr, const int32_t* colIdx,
                          PcgResidentPlan& plan);

// The batched PCG's tile shape (an index into kBatchTiles) before any tuning: 512 threads with 4 lanes per row, or 128 for batches of small problems, whose rows leave
// most of 512 threads idle at every barrier.  us of a solve with 128 and 512 threads: 2,000 problems of 8 nodes 133 and
// 343, 1,000 of 27 537 and 1,055, 500 of 64 796 and 1,159, 100 of 64 348 and 315, 152 of 125 888 and 686, 152 of 343
// 4,707 and 2,423
inline int ef_batch_default_tile(int64_t nProb, int64_t nNodes) { return nNodes <= 64 * nProb ? 1 : 6; }

// The batched PCG's sliced copy for one number of lanes per block row: device arrays
struct BatchPlanDev {
    int nGroups = 0;                       // groups of 32 / lanes rows, none across two problems
    const int32_t *nodePtr = nullptr;      // [problems + 1]
    const int32_t *order = nullptr;        // [problems] by decreasing size
    const int32_t *groupBase = nullptr;    // [problems] a problem's first entry of groupPtr
    const int32_t *groupPtr = nullptr;     // per problem [groups + 1] first step of each group
    const int32_t *groupRow = nullptr;     // [groups] first row
    const int32_t *groupEnd = nullptr;     // [groups] the problem's end row
    const int32_t *groupStep = nullptr;    // [groups][2] first and last step
    double* vals = nullptr;                // [steps][9][32] (null: no copy)
    int32_t* col = nullptr;                // [steps][32]
};
