// C ABI of batches of independent problems in one context: problem ranges, tile shapes and their
// autotuner, the one-launch batched PCG and per-problem norms.

#include "ctx.h"

static const int kBatchLanes[3] = {1, 4, 8};

// the sliced layouts of the batched PCG for 1, 4 and 8 lanes per block row; their values and columns share one
// buffer, which every solve fills for its tile's lanes
static ef_status batch_plans(ef_ctx* c, int nProb, const int32_t* nodePtr) {
    for (void* p : c->batchMem) cudaFree(p);
    c->batchMem.clear();
    int64_t most = 1;
    auto keep = [&](const std::vector<int32_t>& v, const int32_t** out) -> ef_status {
        int32_t* d = nullptr;
        EF_CHECK(upload(&d, v));
        c->batchMem.push_back(d);
        *out = d;
        return EF_OK;
    };
    for (int i = 0; i < 3; ++i) {
        const int lpr = kBatchLanes[i], rpw = 32 / lpr;
        std::vector<int32_t> base(nProb), ptr, row, end, step;
        int64_t steps = 0;
        for (int p = 0; p < nProb; ++p) {
            base[p] = (int32_t)ptr.size();
            for (int32_t m0 = nodePtr[p]; m0 < nodePtr[p + 1]; m0 += rpw) {
                int w = 0;
                for (int32_t m = m0; m < std::min(nodePtr[p + 1], m0 + rpw); ++m)
                    w = std::max(w, (c->hRowPtr0[m + 1] - c->hRowPtr0[m] + lpr - 1) / lpr);
                ptr.push_back((int32_t)steps);
                row.push_back(m0);
                end.push_back(nodePtr[p + 1]);
                step.push_back((int32_t)steps);
                steps += w;
                step.push_back((int32_t)steps);
            }
            ptr.push_back((int32_t)steps);
        }
        if (steps >= ((int64_t)1 << 31)) {
            ef_set_error("ef_batch_setup: too many blocks");
            return EF_ERR_ARG;
        }
        BatchPlanDev& pl = c->batchPlan[i];
        pl = BatchPlanDev();
        pl.nGroups = (int)row.size();
        pl.nodePtr = c->dBatchNodePtr;
        pl.order = c->dBatchOrder;
        EF_CHECK(keep(base, &pl.groupBase));
        EF_CHECK(keep(ptr, &pl.groupPtr));
        EF_CHECK(keep(row, &pl.groupRow));
        EF_CHECK(keep(end, &pl.groupEnd));
        EF_CHECK(keep(step, &pl.groupStep));
        most = std::max(most, steps);
    }
    ef_status st = EF_OK;
    // the copy takes as much as the system itself and its padding; where there is no room for it (or with EF_BATCH_SLICED=0),
    // the kernels read the block rows
    const char* e = getenv("EF_BATCH_SLICED");
    double* vals = e && atoi(e) == 0 ? nullptr : dalloc<double>((size_t)288 * most, &st);
    int32_t* col = vals ? dalloc<int32_t>((size_t)32 * most, &st) : nullptr;
    if (!col) {
        cudaFree(vals);
        (void)cudaGetLastError();
        vals = nullptr;
        st = EF_OK;
    } else {
        c->batchMem.push_back(vals);
        c->batchMem.push_back(col);
    }
    c->dBatchTicket = dalloc<int>(1, &st);
    if (!c->dBatchTicket) return st;
    c->batchMem.push_back(c->dBatchTicket);
    for (BatchPlanDev& pl : c->batchPlan) {
        pl.vals = vals;
        pl.col = col;
    }
    std::vector<int> sizes(nProb);
    for (int p = 0; p < nProb; ++p) sizes[p] = nodePtr[p + 1] - nodePtr[p];
    c->batchCluster = ef_batch_cluster_size(c->nSM, sizes);
    if (!c->batchTileSet) c->batchTile = ef_batch_default_tile(nProb, c->nNodes);
    return EF_OK;
}

ef_status ef_batch_setup(ef_ctx* c, int nProb, const int32_t* nodePtr) {
    EF_REQUIRE_FINALIZED(c);
    if (nProb <= 0 || !nodePtr || nodePtr[0] != 0 || nodePtr[nProb] != (int32_t)c->nNodes) {
        ef_set_error("ef_batch_setup: node ranges must cover [0, nNodes)");
        return EF_ERR_ARG;
    }
    for (int p = 0; p < nProb; ++p)
        if (nodePtr[p + 1] < nodePtr[p]) {
            ef_set_error("ef_batch_setup: node ranges must be increasing");
            return EF_ERR_ARG;
        }
    if (!c->keFp64) {
        ef_set_error("ef_batch_setup: the batched solve runs on the FP64 system (EF_OPT_KE_FP64)");
        return EF_ERR_ARG;
    }
    // every block must couple nodes of one problem (block-diagonal system)
    std::vector<int32_t> prob(c->nNodes);
    for (int p = 0; p < nProb; ++p)
        for (int32_t m = nodePtr[p]; m < nodePtr[p + 1]; ++m) prob[m] = p;
    for (int64_t m = 0; m < c->nNodes; ++m)
        for (int32_t k = c->hRowPtr0[m]; k < c->hRowPtr0[m + 1]; ++k)
            if (prob[c->hColIdx0[k]] != prob[m]) {
                ef_set_error("ef_batch_setup: a block couples two problems");
                return EF_ERR_ARG;
            }
    std::vector<int32_t> order(nProb);
    for (int p = 0; p < nProb; ++p) order[p] = p;
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
        return nodePtr[a + 1] - nodePtr[a] > nodePtr[b + 1] - nodePtr[b];
    });
    if (c->dBatchNodePtr) cudaFree(c->dBatchNodePtr);
    if (c->dBatchOrder) cudaFree(c->dBatchOrder);
    ef_status st = EF_OK;
    c->dBatchNodePtr = dalloc<int32_t>(nProb + 1, &st);
    c->dBatchOrder = dalloc<int32_t>(nProb, &st);
    if (st != EF_OK) return st;
    EF_CUDA(cudaMemcpy(c->dBatchNodePtr, nodePtr, sizeof(int32_t) * (nProb + 1), cudaMemcpyHostToDevice));
    EF_CUDA(cudaMemcpy(c->dBatchOrder, order.data(), sizeof(int32_t) * nProb, cudaMemcpyHostToDevice));
    c->batchN = 0;
    EF_CHECK(batch_plans(c, nProb, nodePtr));
    c->batchN = nProb;
    return EF_OK;
}

ef_status ef_batch_set_tile(ef_ctx* c, int tile) {
    EF_REQUIRE_FINALIZED(c);
    if (tile < 0 || tile >= ef_batch_num_tiles()) {
        ef_set_error("ef_batch_set_tile: unknown tile shape");
        return EF_ERR_ARG;
    }
    c->batchTile = tile;
    c->batchTileSet = true;
    return EF_OK;
}

int ef_batch_tile_count(void) { return ef_batch_num_tiles(); }

ef_status ef_batch_tile_info(int tile, int* threadsPerCta, int* lanesPerRow) {
    if (tile < 0 || tile >= ef_batch_num_tiles() || !threadsPerCta || !lanesPerRow) return EF_ERR_ARG;
    ef_batch_tile_shape(tile, threadsPerCta, lanesPerRow);
    return EF_OK;
}

static ef_status batch_solve(ef_ctx* c, int tile, double rtol, int maxIter, const double* b, double* x, int* iters,
                             double* relres, cudaStream_t s) {
    const int64_t n = c->nDof;
    double* xd = c->w64[0];
    double* r64 = c->w64[2];
    // Dirichlet DOFs take b; the free part solves K_ff x_f = b_f - K_fd x_d per problem
    EF_CHECK(ef_launch_masked_copy(n, b, c->dMask, 1, 1.0, xd, 1, s));
    EF_CHECK(residual64(c, xd, b, r64, nullptr, s));
    double* w[6];
    for (int i = 0; i < 6; ++i) w[i] = (double*)c->w64k[1 + i];
    int tpb = 0, lpr = 0;
    ef_batch_tile_shape(tile, &tpb, &lpr);
    EF_CHECK(ef_launch_batched_pcg(tile, c->batchPlan[lpr == 1 ? 0 : (lpr == 4 ? 1 : 2)], c->batchCluster, c->nSM, c->batchN,
                                   c->dRowPtr, c->dColIdx, (const double*)c->dBsrVals, (const double*)c->dBinv, c->dMask,
                                   r64, w[0], w[1], w[5], w[2], w[3], w[4], maxIter, rtol * rtol, iters, relres,
                                   c->dBatchTicket, s));
    return ef_launch_add(n, xd, w[0], x, s);
}

ef_status ef_batch_solve(ef_ctx* c, double rtol, int maxIter, const double* b, double* x, int* iters, double* relres,
                         void* stream) {
    EF_REQUIRE_FINALIZED(c);
    if (c->batchN == 0) {
        ef_set_error("ef_batch_solve: call ef_batch_setup first");
        return EF_ERR_STATE;
    }
    if (!b || !x || !iters || !relres || !(rtol > 0.0) || maxIter < 0) return EF_ERR_ARG;
    return batch_solve(c, c->batchTile, rtol, maxIter, b, x, iters, relres, (cudaStream_t)stream);
}

ef_status ef_batch_autotune(ef_ctx* c, double rtol, int maxIter, const double* b, double* x, int* iters,
                            double* relres, void* stream, int* tileOut, float* msOut) {
    EF_REQUIRE_FINALIZED(c);
    if (c->batchN == 0) {
        ef_set_error("ef_batch_autotune: call ef_batch_setup first");
        return EF_ERR_STATE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    float best = 1e30f;
    int bestT = c->batchTile;
    for (int t = 0; t < ef_batch_num_tiles(); ++t) {
        EF_CHECK(batch_solve(c, t, rtol, maxIter, b, x, iters, relres, s));  // warm-up
        EF_CUDA(cudaEventRecord(c->ev[0], s));
        EF_CHECK(batch_solve(c, t, rtol, maxIter, b, x, iters, relres, s));
        EF_CUDA(cudaEventRecord(c->ev[1], s));
        EF_CUDA(cudaEventSynchronize(c->ev[1]));
        float ms = 0.f;
        EF_CUDA(cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]));
        if (msOut) msOut[t] = ms;
        if (ms < best) {
            best = ms;
            bestT = t;
        }
    }
    c->batchTile = bestT;
    c->batchTileSet = true;
    if (tileOut) *tileOut = bestT;
    return EF_OK;
}

ef_status ef_batch_norms(ef_ctx* c, const double* R, const double* F, const double* ddU, double* out, void* stream) {
    EF_REQUIRE_FINALIZED(c);
    if (c->batchN == 0) {
        ef_set_error("ef_batch_norms: call ef_batch_setup first");
        return EF_ERR_STATE;
    }
    if (!R || !F || !out) return EF_ERR_ARG;
    return ef_launch_batch_norms(c->batchN, c->dBatchNodePtr, R, F, ddU, out, (cudaStream_t)stream);
}

