// C ABI of the assembled system: the reference-layout VIJ values and scalar CSR, the Dirichlet
// set, the 3x3-block assembly, its FP64 product and residual, the block-Jacobi PCG runner, the
// convergence reductions and the device Newton check.

#include "ctx.h"

ef_status ef_export_vij(ef_ctx* c, double* Kvij, void* stream) {
    EF_REQUIRE_FINALIZED(c);
    if (!Kvij) return EF_ERR_ARG;
    const size_t ks = c->keFp64 ? sizeof(double) : sizeof(float);
    int64_t vijOff = 0;
    for (const auto& g : c->groups) {
        const void* K = (const char*)c->Kblk + (size_t)g.keOffset * 9 * ks;
        EF_CHECK(ef_launch_vij_export(g.nEl, g.nNodes, g.nPair, K, c->keFp64, Kvij + vijOff, (cudaStream_t)stream));
        vijOff += (int64_t)g.nEl * g.nDofEl * g.nDofEl;
    }
    return EF_OK;
}

ef_status ef_csr_pattern(ef_ctx* c, int32_t* indptr, int32_t* indices) {
    EF_REQUIRE_FINALIZED(c);
    if (!c->scalar) {
        ef_set_error("ef_csr_pattern: context finalized with EF_OPT_NO_SCALAR_CSR");
        return EF_ERR_STATE;
    }
    if (indptr) EF_CUDA(cudaMemcpy(indptr, c->hIndptr.data(), sizeof(int32_t) * (c->nDof + 1), cudaMemcpyDefault));
    if (indices) EF_CUDA(cudaMemcpy(indices, c->hIndices.data(), sizeof(int32_t) * c->nnz, cudaMemcpyDefault));
    return EF_OK;
}

ef_status ef_update_csr(ef_ctx* c, const double* Kvij, double* csrData, void* stream) {
    EF_REQUIRE_FINALIZED(c);
    if (!c->scalar || !csrData) {
        ef_set_error("ef_update_csr: no scalar CSR map or null output");
        return EF_ERR_STATE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (!Kvij) {  // the context's own element blocks, without the VIJ vector between
        CsrGroups G = {};
        for (const auto& g : c->groups) {
            G.vijEnd[G.n] = (int)((G.n ? G.vijEnd[G.n - 1] : 0) + (int64_t)g.nEl * g.nDofEl * g.nDofEl);
            G.nd[G.n] = g.nDofEl;
            G.keOffset[G.n++] = g.keOffset;
        }
        return ef_launch_csr_from_blocks(c->nnz, c->dCsrSeg, c->dCsrPerm, G, c->Kblk, c->keFp64, csrData, s);
    }
    return ef_launch_csr_scatter(c->nVIJ, c->nnz, c->dCsrSeg, c->dCsrPerm, Kvij, csrData, s);
}

ef_status ef_csr_dirichlet_rows(ef_ctx* c, double* csrData, const int64_t* rows, int64_t nRows, void* stream) {
    EF_REQUIRE_FINALIZED(c);
    if (!c->scalar || !csrData || (nRows > 0 && !rows)) return EF_ERR_ARG;
    if (nRows == 0) return EF_OK;
    for (int64_t i = 0; i < nRows; ++i)
        if (rows[i] < 0 || rows[i] >= c->nDof) {
            ef_set_error("ef_csr_dirichlet_rows: row out of range");
            return EF_ERR_ARG;
        }
    // the rows go through buffers of the context (no allocation and no synchronisation per call): a pinned copy, so
    // that the caller's array is free again, and a device one; both wait for the launch that last used them.  Under
    // stream capture that wait could not be kept (the event would belong to the capture, and a replay would read
    // whatever rows the pinned copy holds by then), so the call is refused there
    cudaStream_t s = (cudaStream_t)stream;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    EF_CUDA(cudaStreamIsCapturing(s, &capture));
    if (capture != cudaStreamCaptureStatusNone) {
        ef_set_error("ef_csr_dirichlet_rows: not under stream capture");
        return EF_ERR_STATE;
    }
    if (!c->csrRowsDone) EF_CUDA(cudaEventCreateWithFlags(&c->csrRowsDone, cudaEventDisableTiming));
    EF_CUDA(cudaEventSynchronize(c->csrRowsDone));
    if (c->csrRowsCap < nRows) {
        if (c->dCsrRows) cudaFree(c->dCsrRows);
        if (c->hCsrRows) cudaFreeHost(c->hCsrRows);
        c->dCsrRows = c->hCsrRows = nullptr;
        c->csrRowsCap = 0;
        ef_status st = EF_OK;
        c->dCsrRows = dalloc<int64_t>(nRows, &st);
        if (!c->dCsrRows) return st;
        EF_CUDA(cudaHostAlloc((void**)&c->hCsrRows, sizeof(int64_t) * nRows, cudaHostAllocDefault));
        c->csrRowsCap = nRows;
    }
    memcpy(c->hCsrRows, rows, sizeof(int64_t) * nRows);
    EF_CUDA(cudaMemcpyAsync(c->dCsrRows, c->hCsrRows, sizeof(int64_t) * nRows, cudaMemcpyHostToDevice, s));
    const ef_status st = ef_launch_csr_dirichlet_rows(nRows, c->dCsrRows, c->dIndptr, c->dIndices, csrData, s);
    EF_CUDA(cudaEventRecord(c->csrRowsDone, s));  // (the copy is under way in any case)
    return st;
}

ef_status ef_set_dirichlet(ef_ctx* c, const int64_t* dofs, int64_t n) {
    EF_REQUIRE_FINALIZED(c);
    std::vector<uint8_t> m(c->nDof, 0);
    for (int64_t i = 0; i < n; ++i) {
        if (dofs[i] < 0 || dofs[i] >= c->nDof) {
            ef_set_error("ef_set_dirichlet: DOF out of range");
            return EF_ERR_ARG;
        }
        m[dofs[i]] = 1;
    }
    {
        ef_status st = EF_OK;
        if (c->dDirIdx) cudaFree(c->dDirIdx);
        if (c->dDirMask) cudaFree(c->dDirMask);
        c->dDirIdx = nullptr;
        c->dDirMask = nullptr;
        c->nDir = n;
        if (n > 0) {
            c->dDirIdx = dalloc<int64_t>((size_t)n, &st);
            if (!c->dDirIdx) return st;
            EF_CUDA(cudaMemcpy(c->dDirIdx, dofs, sizeof(int64_t) * n, cudaMemcpyHostToDevice));
        }
        c->dDirMask = dalloc<uint8_t>((size_t)c->nDof, &st);
        if (!c->dDirMask) return st;
        EF_CUDA(cudaMemcpy(c->dDirMask, m.data(), c->nDof, cudaMemcpyHostToDevice));
    }
    for (int32_t sN : c->hTieS)
        for (int k = 0; k < 3; ++k) m[3 * (int64_t)sN + k] = 1;
    c->anyDirichlet = n > 0 || !c->hTieS.empty();
    EF_CUDA(cudaMemcpy(c->dMask, m.data(), c->nDof, cudaMemcpyHostToDevice));
    c->hMask = std::move(m);
    c->amgStale = true;
    c->amgMaskChanged = true;
    c->amgPowerDue = true;
    c->nnEdgeStale = true;
    c->nnVersion++;
    return EF_OK;
}

ef_status ef_assemble_bsr(ef_ctx* c, void* stream) {
    EF_REQUIRE_FINALIZED(c);
    cudaStream_t s = (cudaStream_t)stream;
    c->sellStale = true;
    EF_CHECK(ef_launch_bsr_scatter(c->nBlocks, c->dBsrSeg, c->dBsrSrc, c->dBsrW, c->Kblk, c->keFp64, c->dBsrVals, s));
    EF_CHECK(ef_launch_bj_setup(c->nNodes, c->dDiagPos, c->dNodeDof, c->dMask, c->dBsrVals, c->keFp64, c->dBinv,
                                c->dFlags, s));
    c->amgStale = true;
    c->nnEdgeStale = true;
    c->nnVersion++;
    return EF_OK;
}

ef_status ef_bsr_matvec(ef_ctx* c, const double* x, double* y, void* stream) {
    EF_REQUIRE_FINALIZED(c);
    return ef_launch_bsr_residual((int)c->nNodes, c->dRowPtr, c->dColIdx, c->dBsrVals, c->keFp64, x, nullptr,
                                  c->anyDirichlet ? c->dMask : nullptr, y, c->nSM, (cudaStream_t)stream);
}

// r = b - K x on free rows (0 on Dirichlet rows): with the exact FP64 tangent (matrix-free element
// apply) when the system is stored in FP32, else with the stored system; rr (host, may be null): r.r, then
// with a synchronisation of the stream
ef_status residual64(ef_ctx* c, const double* x, const double* b, double* r, double* rr, cudaStream_t s) {
    if (!c->exact) {
        EF_CHECK(ef_launch_bsr_residual((int)c->nNodes, c->dRowPtr, c->dColIdx, c->dBsrVals, c->keFp64, x, b, c->dMask, r,
                                        c->nSM, s));
        return rr ? dot_host(c, r, r, rr, s) : EF_OK;
    }
    if (c->dTieS) {  // the element apply needs the tied DOFs filled from their masters
        EF_CUDA(cudaMemcpyAsync(c->dTieTmp, x, sizeof(double) * c->nDof, cudaMemcpyDeviceToDevice, s));
        EF_CHECK(ef_launch_tie_fill((int64_t)c->hTieS.size(), c->dTieS, c->dTieA, c->dTieB, c->dTieTmp, s));
        x = c->dTieTmp;
    }
    for (size_t gi = 0; gi < c->groups.size(); ++gi) {
        const Group& g = c->groups[gi];
        if (g.tl)
            EF_CHECK(ef_launch_total_lagrange_apply(g, x, c->dTang[gi], c->dYe + g.peOffset, s));
        else
            EF_CHECK(ef_launch_small_strain_apply(g, x, c->dTang[gi], c->dYe + g.peOffset, s));
    }
    EF_CHECK(ef_launch_condense_residual(c->nNodes, c->dNodeDof, c->dCondPtr, c->dCondSrc, c->dCondW, c->dYe, b, c->dMask,
                                         r, c->dPart, c->nPart, c->dTicket, rr ? c->hResDev->red : nullptr, s));
    if (!rr) return EF_OK;
    EF_CUDA(cudaStreamSynchronize(s));
    *rr = c->hRes->red[0];
    return EF_OK;
}

ef_status dot_host(ef_ctx* c, const double* a, const double* b, double* out, cudaStream_t s) {
    EF_CHECK(ef_launch_dot(c->nDof, a, b, c->dPart, c->nPart, c->dTicket, c->hResDev->red, s));
    EF_CUDA(cudaStreamSynchronize(s));
    *out = c->hRes->red[0];
    return EF_OK;
}

// A plan that finds no memory, on the host or the device, is none: the streaming kernel needs nothing beyond the
// context's vectors (EF_PCG_RESIDENT=0 takes it always).
static void pcg_plan(ef_ctx* c, int vDouble) {
    if (c->pcgPlanned) return;
    c->pcgPlanned = true;
    c->pcgSmem = 0;
    const char* e = getenv("EF_PCG_RESIDENT");
    if (e && atoi(e) == 0) return;
    PcgResidentPlan p;
    try {
        ef_pcg_resident_plan(vDouble, c->nSM, (int)c->nNodes, c->hRowPtr0.data(), c->hColIdx0.data(), p);
    } catch (const std::exception&) {
        return;
    }
    if (p.smem == 0) return;
    if (upload(&c->dPcgHaloPtr, p.haloPtr) == EF_OK && upload(&c->dPcgHaloIdx, p.haloIdx) == EF_OK &&
        upload(&c->dPcgGroupPtr, p.groupPtr) == EF_OK && upload(&c->dPcgLcol, p.lcol) == EF_OK) {
        c->pcgSmem = p.smem;
        c->pcgShape = p.shape;
        return;
    }
    (void)cudaGetLastError();
    cudaFree(c->dPcgHaloPtr);
    cudaFree(c->dPcgHaloIdx);
    cudaFree(c->dPcgGroupPtr);
    cudaFree(c->dPcgLcol);
    c->dPcgHaloPtr = c->dPcgHaloIdx = c->dPcgGroupPtr = nullptr;
    c->dPcgLcol = nullptr;
}

// one PCG launch on the free DOFs: solves K d = rhs (rhs zero on Dirichlet DOFs); vDouble: the
// precision of the system
ef_status run_pcg(ef_ctx* c, int vDouble, const void* rhs, void* sol, int maxIter, double rtol,
                         PcgResult* out, ef_solve_info* prof, cudaStream_t s) {
    void** w = vDouble ? c->w64k : c->w32;
    pcg_plan(c, vDouble);
    pcg_result_clear(c->hRes->pcg);
    if (prof) EF_CUDA(cudaEventRecord(c->ev[0], s));
    if (c->pcgSmem > 0)
        EF_CHECK(ef_launch_pcg_resident(vDouble, c->pcgShape, (int)c->nNodes, c->dRowPtr, c->dPcgLcol, c->dPcgHaloPtr,
                                        c->dPcgHaloIdx, c->dPcgGroupPtr, c->pcgSmem, c->dBsrVals, c->dBinv, c->dMask,
                                        rhs, sol, w[3], c->dPcgSlots, &c->hResDev->pcg, maxIter, rtol * rtol, c->dFlags, s));
    else
        EF_CHECK(ef_launch_pcg(vDouble, c->nSM, (int)c->nNodes, c->dRowPtr, c->dColIdx, c->dBsrVals, c->dBinv, c->dMask,
                               rhs, sol, w[2], w[3], w[4], w[5], w[6], c->dPcgSlots, ef_pcg_slot_sets(),
                               &c->hResDev->pcg, maxIter, rtol * rtol, c->dFlags, s));
    if (prof) EF_CUDA(cudaEventRecord(c->ev[1], s));
    EF_CUDA(cudaStreamSynchronize(s));
    *out = c->hRes->pcg;
    if (prof) {
        float ms = 0.f;
        EF_CUDA(cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]));
        prof->kernelMs += ms;
        prof->kernelLaunches += 1;
    }
    if (pcg_result_timed_out(*out)) {
        ef_set_error("PCG: grid barrier timed out");
        return EF_ERR_DEVICE;
    }
    return EF_OK;
}



ef_status ef_newton_residual(ef_ctx* c, int mode, const double* P, const double* PExt, const double* dirValues,
                             const double* F, const double* ddU, int iteration, double prevResidual, int nGrew,
                             const ef_newton_opts* o, double* R, ef_newton_check* out, void* stream) {
    EF_REQUIRE_FINALIZED(c);
    if (!P || !R || (mode != 0 && mode != 1) || (mode == 1 && (!F || !o || !out)) ||
        (mode == 0 && c->nDir > 0 && !dirValues)) {
        ef_set_error("ef_newton_residual: bad arguments");
        return EF_ERR_ARG;
    }
    if (!c->dDirMask) {
        ef_set_error("ef_newton_residual: call ef_set_dirichlet first");
        return EF_ERR_STATE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (mode == 0) return ef_launch_newton_first(c->nDof, P, PExt, c->nDir, c->dDirIdx, dirValues, R, s);
    const NewtonTest q = {o->fluxTol, o->fluxTolAlt, o->corrTol, o->fluxFloor, o->nAccFluxes, prevResidual, iteration,
                          nGrew};
    EF_CHECK(ef_launch_newton_check(c->nDof, P, PExt, c->dDirMask, F, ddU, R, c->dPart, c->nPart, c->dTicket, q,
                                    c->hResDev->red, s));
    EF_CUDA(cudaStreamSynchronize(s));
    const double* r = c->hRes->red;
    out->converged = r[0] != 0.0;
    out->nGrew = (int)r[1];
    out->fluxResidual = r[2];
    out->fieldCorrection = r[3];
    out->spatialAveragedFlux = r[4];
    return EF_OK;
}

ef_status ef_norms(ef_ctx* c, const double* R, const double* F, const double* ddU, double* out, void* stream) {
    EF_REQUIRE_FINALIZED(c);
    if (!out) return EF_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    EF_CHECK(ef_launch_norms(c->nDof, R, F, ddU, c->dPart, c->nPart, c->dTicket, c->hResDev->red, s));
    EF_CUDA(cudaStreamSynchronize(s));
    memcpy(out, c->hRes->red, 3 * sizeof(double));
    return EF_OK;
}

