// Host-side plan of the resident PCG kernel (krylov.cu): which rows a CTA keeps, gathers and how its blocks
// are sliced.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <vector>

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
