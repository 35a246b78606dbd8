// Krylov kernels on the 3x3-block (BSR) system: SpMV, block-Jacobi PCG as one
// persistent cooperative launch, and the FP64 residual of the iterative refinement.
//
// Replaces the linear solve behind NIST.linearSolve (solvers/nonlinearimplicitstatic.py:727-751;
// the reference's solvers are MKL PARDISO / SuperLU / GMRES+AMG, config/linsolve.py).
//
// Dirichlet DOFs are eliminated symmetrically: every Krylov vector vanishes on them and
// the operator's Dirichlet rows are masked to zero, so the free-free block is solved.
// Reductions are deterministic (per-CTA partials summed in a fixed order by every CTA).
// The persistent kernels over a grid are launched cooperatively (all CTAs resident) and their waits are bounded; the form
// that is one cluster is a plain launch that waits at the hardware's cluster barrier only.

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "cluster.cuh"
#include "ef_common.cuh"
#include "pcg_plan.h"
#include "pcg_scalars.h"
#include "reduce.cuh"

namespace ef {

constexpr int kKB = 512;         // threads per CTA of the Krylov kernels
constexpr int kRowLanes = 8;     // lanes per block row in the SpMV
constexpr int kBatch = 4;        // blocks per lane whose loads are issued together

// y_row = A_row x for the block row `m`, lanes l = 0..7 of a row group; returns partial sums
// CG = true loads x through L2 only (x was written by other CTAs of a persistent kernel)
template <typename MT, typename XT, typename AT, bool CG>
__device__ __forceinline__ void bsr_row(int m, int l, const int32_t* __restrict__ rowPtr,
                                        const int32_t* __restrict__ colIdx, const MT* __restrict__ vals,
                                        const XT* __restrict__ x, AT& y0, AT& y1, AT& y2) {
    y0 = y1 = y2 = (AT)0;
    const int s = rowPtr[m], e = rowPtr[m + 1];
    for (int base = s; base < e; base += kRowLanes * kBatch) {
        int cc[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            const int k = base + l + j * kRowLanes;
            cc[j] = k < e ? 3 * colIdx[k] : -1;
        }
        AT xv[kBatch][3];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            if (cc[j] >= 0) {
                const int c = cc[j];
                if (CG) {
                    xv[j][0] = (AT)__ldcg(x + c);
                    xv[j][1] = (AT)__ldcg(x + c + 1);
                    xv[j][2] = (AT)__ldcg(x + c + 2);
                } else {
                    xv[j][0] = (AT)x[c];
                    xv[j][1] = (AT)x[c + 1];
                    xv[j][2] = (AT)x[c + 2];
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            if (cc[j] >= 0) {
                const MT* v = vals + (int64_t)(base + l + j * kRowLanes) * 9;
                y0 += (AT)v[0] * xv[j][0] + (AT)v[1] * xv[j][1] + (AT)v[2] * xv[j][2];
                y1 += (AT)v[3] * xv[j][0] + (AT)v[4] * xv[j][1] + (AT)v[5] * xv[j][2];
                y2 += (AT)v[6] * xv[j][0] + (AT)v[7] * xv[j][1] + (AT)v[8] * xv[j][2];
            }
        }
    }
#pragma unroll
    for (int o = kRowLanes / 2; o > 0; o >>= 1) {
        y0 += __shfl_xor_sync(0xffffffffu, y0, o);
        y1 += __shfl_xor_sync(0xffffffffu, y1, o);
        y2 += __shfl_xor_sync(0xffffffffu, y2, o);
    }
}

// y = beta_b * b - A x (masked rows -> 0) in AT accumulation; one launch, grid-stride rows.
// With b == nullptr: y = A x.  mask may be nullptr (no masking).
template <typename MT, typename XT, typename AT>
__global__ void __launch_bounds__(kKB) bsr_residual_kernel(int nNodes, const int32_t* __restrict__ rowPtr,
                                                           const int32_t* __restrict__ colIdx,
                                                           const MT* __restrict__ vals, const XT* __restrict__ x,
                                                           const double* __restrict__ b,
                                                           const uint8_t* __restrict__ mask, double* __restrict__ y) {
    const int lane = threadIdx.x % kRowLanes;
    const int groupsPerCTA = kKB / kRowLanes;
    const int nGroups = gridDim.x * groupsPerCTA;
    int g = blockIdx.x * groupsPerCTA + threadIdx.x / kRowLanes;
    // all lanes of a warp iterate the same number of times (shuffles need full warps)
    const int iters = (nNodes + nGroups - 1) / nGroups;
    for (int it = 0; it < iters; ++it, g += nGroups) {
        const int m = g < nNodes ? g : nNodes - 1;
        AT y0, y1, y2;
        bsr_row<MT, XT, AT, false>(m, lane, rowPtr, colIdx, vals, x, y0, y1, y2);
        if (g < nNodes && lane < 3) {
            const int d = 3 * m + lane;
            const AT yy = lane == 0 ? y0 : (lane == 1 ? y1 : y2);
            double out = b ? b[d] - (double)yy : (double)yy;
            if (mask && mask[d]) out = 0.0;
            y[d] = out;
        }
    }
}

// ---- block-Jacobi PCG, persistent over all iterations ------------------------------------------
//
// What bounds an iteration is latency, not bandwidth: the systems it runs on (up to some ten
// thousand block rows per SM) stay in L1 and L2, and two reductions that every CTA needs before it
// goes on (p.q, then r.z with r.r) cut the iteration into two short phases.  So:
//  * every CTA owns a contiguous range of block rows in all phases: its part of the matrix, x, r and
//    q is read by this SM alone and stays in its L1; only z and p, which other CTAs gather, go
//    through L2;
//  * a reduction is also the grid barrier: every CTA publishes its partial sum in a slot of its
//    own, polls the slots of all CTAs and sums them in slot order (the same bits in every CTA): one
//    round trip through L2 instead of a grid barrier, a flag read and a read of the partial sums;
//  * one CTA per SM, and fewer when a CTA's lanes already cover the rows in one pass (pcg_shape).
//  * the scalars of the recurrence belong to one thread of a CTA (grid_sum);
//  * systems that fit into shared memory stay there (pcg_resident_kernel), small ones in one cluster.
// us an iteration (kernel time), before (304 CTAs, cooperative-groups barriers, rows dealt out over the grid, scalars in
// every thread) and now: FP32, 624 nodes 21.4 -> 5.3, 4,836 nodes 23.7 -> 9.1, 22,491 nodes 28.3 -> 10.9; FP64,
// 525 nodes 26.6 -> 7.9, 3,146 nodes 27.4 -> 11.8.  Streaming: FP32, 38,125 nodes 28.1 -> 19.7, 169,781 nodes 78.7 -> 63.3;
// FP64, 22,491 nodes 48.4 -> 38.5, 169,781 nodes 222 -> 144.

constexpr int kPcgMaxCtas = 160;                    // slots of a reduction (one CTA per SM)
constexpr int kPcgMaxCluster = 16;                  // CTAs of the cluster form
constexpr int kPcgPoll = kPcgMaxCtas / 32;          // slots a lane of the polling warp watches
constexpr unsigned kPcgSpinLimit = 1u << 22;        // polls before a barrier gives up (seconds)

// Where a launch reports to, and how often a barrier polls
struct PcgWait {
    PcgResult* res;
    int* flags;
    unsigned limit;
};
constexpr unsigned long long kPcgEmpty = ~0ull;     // an unwritten slot (a NaN that no sum produces)
constexpr size_t kPcgSlotBytes = sizeof(double) * 3 * 2 * kPcgMaxCtas;

template <typename VT>
struct PcgTpb {
    static constexpr int value = sizeof(VT) == 4 ? 1024 : 512;
};

// Sums beyond a warp and the scalars made of them are FP64 for FP32 vectors too (PcgScalars); an unevaluated pair
// of FP32 numbers in their place saves 1.5 us of an iteration (624 nodes 5.3, 4,836 nodes 9.1), but carries 48 bits
// and ends at FP32's range.
// bits of a published sum: never kPcgEmpty
__device__ __forceinline__ unsigned long long slot_bits(double v) {
    return v == v ? (unsigned long long)__double_as_longlong(v) : 0x7ff8000000000000ull;
}
__device__ __forceinline__ double slot_sum(unsigned long long u) { return __longlong_as_double((long long)u); }
// a CTA's slot: two values side by side (one request each way)
__device__ __forceinline__ void slot_store(double* p, unsigned long long a, unsigned long long b) {
    asm volatile("st.release.gpu.global.v2.b64 [%0], {%1, %2};\n" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void slot_load(const double* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];\n" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void slot_clear(double* p) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %1};\n" ::"l"(p), "l"(kPcgEmpty) : "memory");
}

template <typename VT, int TPB>
struct PcgShared {
    VT red[2][sizeof(VT) == 4 ? TPB / 32 : TPB];
    unsigned long long part[2][kPcgMaxCluster][2];  // cluster form: the sums of its CTAs, double buffered
    VT scalar;  // the step length or direction factor of the current phase
    int go;     // 1: go on, 0: the solve ends here, -1: a barrier gave up
};

// Sum of NV values over all threads of the grid in a fixed order; the first thread of every CTA
// gets it (the same bits in every CTA) and turns it into the next step's scalar with `next(sum)`, which
// returns whether to go on.  All writes made before the call are visible to every thread after it.
// FP32 values: a shuffle tree per warp, then the CTA's warps; FP64 values: entry `slot` < count of a
// thread (-1: none) goes through shared memory and one warp adds.  A warp's FP64 instruction takes
// the narrow pipe 16 cycles, so the sums and above all the divisions belong to one warp: done by
// every thread, the two divisions of an iteration alone kept the pipe busy for most of the iteration.
// Slots are triple buffered: passing reduction k means that every CTA has arrived there and so
// has read reduction k - 1, whose slot this CTA then empties; its next use (k + 2) lies behind
// reduction k + 1, which orders the emptying before any poll of it.
// PUB = false: no other CTA's writes are read after this reduction, so the polling warp's acquire fence
// (which orders its own later polls) is taken after the CTA has been let go.
// Few CTAs poll one set of slots: with all 152 on the same lines a reduction takes 1 us longer, so a CTA
// stores into `copies` sets and polls one of them.
// CL: the grid is one cluster; the sums go into every CTA's shared memory, behind the cluster's barrier.
// Returns sh.go: -1 when a CTA did not arrive within the poll limit (EF_FLAG_BARRIER and res->gaveUp are set).
template <typename VT, int TPB, int NV, bool PUB, bool CL, typename F>
__device__ __forceinline__ int grid_sum(const VT (&v)[NV], int slot, int count, PcgShared<VT, TPB>& sh,
                                        double* __restrict__ slots, int copies, int& epoch, const PcgWait& wait, F next) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (sizeof(VT) == 4) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            VT t = v[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) sh.red[j][w] = t;
        }
        count = TPB / 32;
    } else if (slot >= 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) sh.red[j][slot] = v[j];
    }
    __syncthreads();
    if (w == 0) {
        double t[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) t[j] = lane < count ? (double)sh.red[j][lane] : 0.0;
        for (int i = lane + 32; i < count; i += 32)
#pragma unroll
            for (int j = 0; j < NV; ++j) t[j] += (double)sh.red[j][i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < NV; ++j) t[j] += __shfl_xor_sync(0xffffffffu, t[j], o);
        const int n = gridDim.x;
        if (CL) {
            if (lane < n) cluster_store(cluster_addr(sh.part[epoch & 1][blockIdx.x], lane), slot_bits(t[0]), slot_bits(t[NV - 1]));
        } else {
            if (lane < copies)
                slot_store(slots + (lane * 3 + epoch % 3) * 2 * kPcgMaxCtas + 2 * blockIdx.x, slot_bits(t[0]), slot_bits(t[NV - 1]));
            const double* mine = slots + ((int)(blockIdx.x % copies) * 3 + epoch % 3) * 2 * kPcgMaxCtas;
            unsigned long long u[kPcgPoll], v2[kPcgPoll];
#pragma unroll
            for (int i = 0; i < kPcgPoll; ++i) u[i] = v2[i] = lane + 32 * i < n ? kPcgEmpty : 0ull;
            bool all = false;
            for (unsigned spin = 0; !all && spin < wait.limit; ++spin) {
                all = true;
#pragma unroll
                for (int i = 0; i < kPcgPoll; ++i)
                    if (u[i] == kPcgEmpty || v2[i] == kPcgEmpty) slot_load(mine + 2 * (lane + 32 * i), u[i], v2[i]);
#pragma unroll
                for (int i = 0; i < kPcgPoll; ++i) all = all && u[i] != kPcgEmpty && v2[i] != kPcgEmpty;
            }
            if (PUB) __threadfence();  // with the relaxed loads: acquires what the other CTAs released
            const bool arrived = __all_sync(0xffffffffu, all);
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                static_assert(kPcgPoll == 5, "the sum below");
                auto at = [&](int i) { return slot_sum(j == 0 ? u[i] : v2[i]); };
                t[j] = at(0);
                if (n > 32) t[j] = n > 64 ? (at(0) + at(1)) + (at(2) + at(3)) : at(0) + at(1);
                if (n > 128) t[j] += at(4);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int j = 0; j < NV; ++j) t[j] += __shfl_xor_sync(0xffffffffu, t[j], o);
            if (lane == 0) {
                if (!arrived) {
                    atomicOr(wait.flags, EF_FLAG_BARRIER);
                    wait.res->gaveUp = 1;
                }
                sh.go = !arrived ? -1 : (next(t) ? 1 : 0);
            }
        }
    }
    if (CL) {
        cluster_barrier();
        if (w == 0) {
            double t[NV];
#pragma unroll
            for (int j = 0; j < NV; ++j)
                t[j] = lane < (int)gridDim.x ? slot_sum(sh.part[epoch & 1][lane][j]) : 0.0;
#pragma unroll
            for (int o = kPcgMaxCluster / 2; o > 0; o >>= 1)
#pragma unroll
                for (int j = 0; j < NV; ++j) t[j] += __shfl_xor_sync(0xffffffffu, t[j], o);
            if (lane == 0) sh.go = next(t) ? 1 : 0;
        }
    }
    __syncthreads();
    if (!CL && w == 0) {
        if (lane < copies && epoch > 0) slot_clear(slots + (lane * 3 + (epoch + 2) % 3) * 2 * kPcgMaxCtas + 2 * blockIdx.x);
        if (!PUB) __threadfence();
    }
    ++epoch;
    return sh.go;
}

// Block-Jacobi PCG on the free DOFs.  The search direction p_k = z_k + beta_k p_{k-1} is never
// materialised before the product: each row group gathers z and the previous p of its neighbours and
// combines them on the fly, writing p_k for its own row into the other half of a double buffer.
// LPR lanes per block row in the product, a thread per block row in the vector updates.
// b: RHS (zero on Dirichlet DOFs); x: solution (out).  A breakdown (p.q <= 0, e.g. FP32 round-off
// near the attainable accuracy) ends the solve with EF_NOT_CONVERGED and the current iterate.
// slots: kPcgSlotBytes of 0xff bytes.
template <typename VT, int LPR>
__global__ void __launch_bounds__(PcgTpb<VT>::value, 1) pcg_persistent_kernel(
    int nNodes, const int32_t* __restrict__ rowPtr, const int32_t* __restrict__ colIdx, const VT* __restrict__ vals,
    const VT* __restrict__ binv, const uint8_t* __restrict__ mask, const VT* __restrict__ b, VT* x, VT* r, VT* z,
    VT* pA, VT* pB, VT* q, double* slots, int copies, PcgWait wait, int maxIter, double rtol2) {
    constexpr int TPB = PcgTpb<VT>::value;
    constexpr int RPI = TPB / LPR;                    // rows per pass of the product
    constexpr int NB = LPR >= 32 ? 1 : (LPR == 16 ? 2 : 4);  // blocks per lane whose loads are issued together
    __shared__ PcgShared<VT, TPB> sh;
    const int tid = threadIdx.x;
    const int l = tid % LPR, grp = tid / LPR;
    const int per = (nNodes + (int)gridDim.x - 1) / (int)gridDim.x;
    const int r0 = min(nNodes, (int)blockIdx.x * per), r1 = min(nNodes, r0 + per);
    // the lane that holds component comp of its row after row_sum3 (comp 3: none)
    const int comp = l % (LPR / 4) == 0 ? l / (LPR / 4) : 3;
    const int slotA = comp < 3 ? 3 * grp + comp : -1, countA = 3 * min(RPI, r1 - r0);
    const int slotB = tid < r1 - r0 ? tid : -1, countB = min(TPB, r1 - r0);
    int epoch = 0;
    PcgScalars<VT> sca;  // of thread 0

    // init: x = 0, r = b, z = M^-1 r
    VT loc[2] = {(VT)0, (VT)0};
    for (int m = r0 + tid; m < r1; m += TPB) {
        const int d = 3 * m;
        VT rv[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            rv[i] = b[d + i];
            x[d + i] = (VT)0;
            r[d + i] = rv[i];
        }
        const VT* B = binv + (int64_t)m * 9;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            VT zi = B[3 * i] * rv[0] + B[3 * i + 1] * rv[1] + B[3 * i + 2] * rv[2];
            if (mask[d + i]) zi = (VT)0;
            z[d + i] = zi;
            loc[0] += rv[i] * zi;
            loc[1] += rv[i] * rv[i];
        }
    }
    int go = grid_sum<VT, TPB, 2, true, false>(loc, slotB, countB, sh, slots, copies, epoch, wait, [&](const double(&t)[2]) {
        return sca.start(t, rtol2, sh.scalar);
    });
    if (go < 0) return;
    int k = 0;
    VT* pPrev = pB;
    VT* pCur = pA;
    if (go) {
        for (k = 0; k < maxIter; ++k) {
            const VT beta = sh.scalar;
            // q = A p_k with p_k = z + beta p_{k-1} formed on the fly; p_k stored for own rows.
            // Loads are batched (up to NB blocks per lane issued before any use) so that a row
            // costs three dependent memory latencies instead of one per block.
            VT pq[1] = {(VT)0};
            for (int m0 = r0; m0 < r1; m0 += RPI) {
                const bool mine = m0 + grp < r1;
                const int m = mine ? m0 + grp : r1 - 1;
                VT y0 = 0, y1 = 0, y2 = 0;
                const int s0 = rowPtr[m], s1 = rowPtr[m + 1];
                for (int base = s0; base < s1; base += LPR * NB) {
                    int cc[NB];
#pragma unroll
                    for (int j = 0; j < NB; ++j) {
                        const int kk = base + l + j * LPR;
                        cc[j] = kk < s1 ? 3 * colIdx[kk] : -1;
                    }
                    VT xv[NB][3];
#pragma unroll
                    for (int j = 0; j < NB; ++j) {
                        if (cc[j] >= 0) {
                            const int c = cc[j];
                            xv[j][0] = __ldcg(z + c);
                            xv[j][1] = __ldcg(z + c + 1);
                            xv[j][2] = __ldcg(z + c + 2);
                            if (k > 0) {
                                xv[j][0] += beta * __ldcg(pPrev + c);
                                xv[j][1] += beta * __ldcg(pPrev + c + 1);
                                xv[j][2] += beta * __ldcg(pPrev + c + 2);
                            }
                        }
                    }
#pragma unroll
                    for (int j = 0; j < NB; ++j) {
                        if (cc[j] >= 0) {
                            const VT* v = vals + (int64_t)(base + l + j * LPR) * 9;
                            block_fma(v, xv[j][0], xv[j][1], xv[j][2], y0, y1, y2);
                        }
                    }
                }
                VT yy = row_sum3<LPR>(l, y0, y1, y2);
                if (mine && comp < 3) {
                    const int d = 3 * m + comp;
                    VT pd = __ldcg(z + d);
                    if (k > 0) pd += beta * __ldcg(pPrev + d);
                    if (mask[d]) yy = (VT)0;
                    q[d] = yy;
                    pCur[d] = pd;
                    pq[0] += pd * yy;
                }
            }
            go = grid_sum<VT, TPB, 1, true, false>(pq, slotA, countA, sh, slots, copies, epoch, wait, [&](const double(&t)[1]) {
                return sca.step(t, sh.scalar);
            });
            if (go < 0) return;
            if (!go) break;
            const VT alpha = sh.scalar;
            VT l2[2] = {(VT)0, (VT)0};
            for (int m = r0 + tid; m < r1; m += TPB) {
                const int d = 3 * m;
                VT rv[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    x[d + i] += alpha * pCur[d + i];
                    rv[i] = r[d + i] - alpha * q[d + i];
                    r[d + i] = rv[i];
                }
                const VT* B = binv + (int64_t)m * 9;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    VT zi = B[3 * i] * rv[0] + B[3 * i + 1] * rv[1] + B[3 * i + 2] * rv[2];
                    if (mask[d + i]) zi = (VT)0;
                    z[d + i] = zi;
                    l2[0] += rv[i] * zi;
                    l2[1] += rv[i] * rv[i];
                }
            }
            go = grid_sum<VT, TPB, 2, true, false>(l2, slotB, countB, sh, slots, copies, epoch, wait, [&](const double(&t)[2]) {
                return sca.direction(t, sh.scalar);
            });
            if (go < 0) return;
            if (!go) {
                if (sca.done) ++k;
                break;
            }
            VT* t = pPrev;
            pPrev = pCur;
            pCur = t;
        }
        if (k >= maxIter && sca.status == EF_OK && !sca.finished()) sca.status = EF_NOT_CONVERGED;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        wait.res->iterations = k;
        wait.res->status = sca.status;
        wait.res->rr = sca.rr;
        wait.res->bb = sca.bb;
    }
}

// The same PCG for systems whose part per SM fits into its shared memory (pcg_resident_fits): a CTA
// keeps its block rows, their vectors and the search direction of its rows and of the rows they
// couple to (the halo) on chip for the whole solve; an iteration reads nothing but the halo's z from
// L2 and writes nothing but its own rows' z.  The streaming kernel above gathers z and p from L2
// for every block (24 bytes in up to two sectors each), which bounds it once its blocks come from
// L1; and every thread of it forms p for every block, which the FP64 pipe feels.
// Only r.z's reduction publishes data; p.q's needs no fence before the CTA goes on.
// CL: the grid is one cluster of up to 16 CTAs, which read each other's z in shared memory.
// The blocks lie sliced by the warp's lanes: the rows go to warps in groups of 32 / LPR, and step j of a
// group holds lane l's j-th block in nine planes of 32 values (shorter rows are padded with zero blocks),
// so a warp's loads fall on 32 different banks; blocks in row order cost up to twice the cycles.
struct ResidentLayout {
    size_t vals, p, z, r, x, q, binv, lcol, halo, mask, bytes;
};
__host__ __device__ inline ResidentLayout resident_layout(size_t vt, int rows, int halo, int steps) {
    ResidentLayout o;
    size_t at = 0;
    auto take = [&](size_t n) {
        const size_t here = at;
        at = (at + n + 15) / 16 * 16;
        return here;
    };
    o.z = take(vt * 3 * rows);  // first: the same place in every CTA (the cluster form reads it there)
    o.vals = take(vt * 9 * 32 * steps);
    o.p = take(vt * 3 * (rows + halo));
    o.r = take(vt * 6 * rows);
    o.x = take(vt * 3 * rows);
    o.q = take(vt * 3 * rows);
    o.binv = take(vt * 9 * rows);
    o.lcol = take(sizeof(uint16_t) * 32 * steps);
    o.halo = take(sizeof(int32_t) * halo);
    o.mask = take(3 * (size_t)rows);
    o.bytes = at;
    return o;
}

template <typename VT, int LPR, bool CL>
__global__ void __launch_bounds__(PcgTpb<VT>::value, 1) pcg_resident_kernel(
    int nNodes, const int32_t* __restrict__ rowPtr, const uint16_t* __restrict__ lcol,
    const int32_t* __restrict__ haloPtr, const int32_t* __restrict__ haloIdx, const int32_t* __restrict__ groupPtr,
    const VT* __restrict__ vals,
    const VT* __restrict__ binv, const uint8_t* __restrict__ mask, const VT* __restrict__ b, VT* __restrict__ x,
    VT* z, double* slots, int copies, PcgWait wait, int maxIter, double rtol2) {
    constexpr int TPB = PcgTpb<VT>::value;
    constexpr int RPI = TPB / LPR;
    constexpr int RPW = 32 / LPR;  // rows per warp
    __shared__ PcgShared<VT, TPB> sh;
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x;
    const int l = tid % LPR, grp = tid / LPR;
    const int per = (nNodes + (int)gridDim.x - 1) / (int)gridDim.x;
    const int r0 = min(nNodes, (int)blockIdx.x * per), rows = min(nNodes, r0 + per) - r0;
    const int h0 = haloPtr[blockIdx.x], nh = haloPtr[blockIdx.x + 1] - h0;
    const int groups = (per + RPW - 1) / RPW;  // of the largest CTA
    const int32_t* gp = groupPtr + (int64_t)blockIdx.x * (groups + 1);  // first step of each of this CTA's groups
    const ResidentLayout lay = resident_layout(sizeof(VT), rows, nh, gp[groups]);
    VT* sv = reinterpret_cast<VT*>(smem + lay.vals);
    VT* sp = reinterpret_cast<VT*>(smem + lay.p);  // own rows, then the halo
    VT* sz = reinterpret_cast<VT*>(smem + lay.z);
    VT* sr = reinterpret_cast<VT*>(smem + lay.r);
    VT* sr2 = sr + 3 * rows;
    VT* sx = reinterpret_cast<VT*>(smem + lay.x);
    VT* sq = reinterpret_cast<VT*>(smem + lay.q);
    VT* sb = reinterpret_cast<VT*>(smem + lay.binv);
    uint16_t* sc = reinterpret_cast<uint16_t*>(smem + lay.lcol);
    int32_t* sH = reinterpret_cast<int32_t*>(smem + lay.halo);
    uint8_t* sm = smem + lay.mask;
    const int lane = tid & 31, warp = tid >> 5;
    for (int g = warp; g < groups; g += TPB / 32) {
        const int m = g * RPW + lane / LPR;
        const int k0 = m < rows ? rowPtr[r0 + m] : 0, k1 = m < rows ? rowPtr[r0 + m + 1] : 0;
        for (int j = gp[g]; j < gp[g + 1]; ++j) {
            const int64_t kk = k0 + l + (int64_t)(j - gp[g]) * LPR;
            VT* d = sv + 9 * 32 * j + lane;
#pragma unroll
            for (int i = 0; i < 9; ++i) d[32 * i] = kk < k1 ? vals[9 * kk + i] : (VT)0;
            sc[32 * j + lane] = kk < k1 ? lcol[kk] : (uint16_t)0;
        }
    }
    for (int i = tid; i < 9 * rows; i += TPB) sb[i] = binv[9 * (int64_t)r0 + i];
    for (int i = tid; i < nh; i += TPB) {
        const int h = haloIdx[h0 + i];
        sH[i] = CL ? (int)cluster_addr(sz + 3 * (h % per), h / per) : 3 * h;
    }
    for (int i = tid; i < 3 * rows; i += TPB) {
        sm[i] = mask[3 * (int64_t)r0 + i];
        sr[i] = b[3 * (int64_t)r0 + i];
        sx[i] = sq[i] = (VT)0;
    }
    for (int i = tid; i < 3 * (rows + nh); i += TPB) sp[i] = (VT)0;
    // the lane that holds component comp of its row after row_sum3 (comp 3: none)
    const int comp = l % (LPR / 4) == 0 ? l / (LPR / 4) : 3;
    const int slotA = comp < 3 ? 3 * grp + comp : -1, countA = 3 * min(RPI, rows);
    const int slotB = tid < 3 * rows ? tid : -1, countB = min(TPB, 3 * rows);
    int epoch = 0;
    PcgScalars<VT> sca;  // of thread 0
    if (CL) cluster_barrier();  // every CTA's shared memory is there before the first remote access
    __syncthreads();

    // vector updates by a thread per DOF d: r of its node (all three components in each of the node's
    // threads, so that no exchange is needed: the new r goes to the other half of a double buffer),
    // z = M^-1 r to this CTA and to those whose halo it is in; r.z and r.r
    auto update = [&](int d, VT alpha, const VT* rOld, VT* rNew, VT (&s)[2]) {
        const int m = d / 3, i = d - 3 * m;
        VT rv[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) rv[j] = rOld[3 * m + j] - alpha * sq[3 * m + j];
        const VT* B = sb + 9 * m + 3 * i;
        VT zi = B[0] * rv[0] + B[1] * rv[1] + B[2] * rv[2];
        if (sm[d]) zi = (VT)0;
        const VT ri = i == 0 ? rv[0] : (i == 1 ? rv[1] : rv[2]);
        rNew[d] = ri;
        sz[d] = zi;
        if (!CL) z[3 * (int64_t)r0 + d] = zi;
        s[0] += ri * zi;
        s[1] += ri * ri;
    };
    VT loc[2] = {(VT)0, (VT)0};
    for (int d = tid; d < 3 * rows; d += TPB) update(d, (VT)0, sr, sr2, loc);  // q = 0: r = b
    int go = grid_sum<VT, TPB, 2, true, CL>(loc, slotB, countB, sh, slots, copies, epoch, wait, [&](const double(&t)[2]) {
        return sca.start(t, rtol2, sh.scalar);
    });
    if (go < 0) return;
    int k = 0;
    if (go) {
        for (k = 0; k < maxIter; ++k) {
            // p = z + beta p of the halo (z from L2) and of the own rows
            const VT beta = sh.scalar;
            for (int i = tid; i < 3 * nh; i += TPB) {
                const int h = i / 3;
                const VT zi = CL ? cluster_load((unsigned)sH[h] + (unsigned)(sizeof(VT) * (i - 3 * h)), (VT)0)
                                 : __ldcg(z + sH[h] + (i - 3 * h));
                sp[3 * rows + i] = zi + beta * sp[3 * rows + i];
            }
            for (int i = tid; i < 3 * rows; i += TPB) sp[i] = sz[i] + beta * sp[i];
            __syncthreads();
            VT pq[1] = {(VT)0};
            for (int g = warp; g * RPW < rows; g += TPB / 32) {  // (a warp without a row left keeps off the FP64 pipe)
                const int m = g * RPW + lane / LPR;
                const bool mine = m < rows;
                VT y0 = 0, y1 = 0, y2 = 0;
                const int j1 = gp[g + 1];
#pragma unroll 2
                for (int j = gp[g]; j < j1; ++j) {
                    const VT* pv = sp + 3 * (int)sc[32 * j + lane];
                    const VT* d = sv + 9 * 32 * j + lane;
                    const VT v[9] = {d[0], d[32], d[64], d[96], d[128], d[160], d[192], d[224], d[256]};
                    block_fma(v, pv[0], pv[1], pv[2], y0, y1, y2);
                }
                VT yy = row_sum3<LPR>(l, y0, y1, y2);
                if (mine && comp < 3) {
                    const int d = 3 * m + comp;
                    if (sm[d]) yy = (VT)0;
                    sq[d] = yy;
                    pq[0] += sp[d] * yy;
                }
            }
            go = grid_sum<VT, TPB, 1, false, CL>(pq, slotA, countA, sh, slots, copies, epoch, wait, [&](const double(&t)[1]) {
                return sca.step(t, sh.scalar);
            });
            if (go < 0) return;
            if (!go) break;
            const VT alpha = sh.scalar;
            VT l2[2] = {(VT)0, (VT)0};
            VT* t = sr;
            sr = sr2;
            sr2 = t;
            for (int d = tid; d < 3 * rows; d += TPB) {
                sx[d] += alpha * sp[d];
                update(d, alpha, sr, sr2, l2);
            }
            go = grid_sum<VT, TPB, 2, true, CL>(l2, slotB, countB, sh, slots, copies, epoch, wait, [&](const double(&t)[2]) {
                return sca.direction(t, sh.scalar);
            });
            if (go < 0) return;
            if (!go) {
                if (sca.done) ++k;
                break;
            }
        }
        if (k >= maxIter && sca.status == EF_OK && !sca.finished()) sca.status = EF_NOT_CONVERGED;
    }
    if (CL) cluster_barrier();  // no CTA leaves while another may still read its shared memory
    for (int i = tid; i < 3 * rows; i += TPB) x[3 * (int64_t)r0 + i] = sx[i];
    if (blockIdx.x == 0 && tid == 0) {
        wait.res->iterations = k;
        wait.res->status = sca.status;
        wait.res->rr = sca.rr;
        wait.res->bb = sca.bb;
    }
}

// *out = a . b
__global__ void __launch_bounds__(kRedThreads) dot_kernel(int64_t n, const double* __restrict__ a,
                                                          const double* __restrict__ b, double* part, unsigned* ticket,
                                                          double* out) {
    double v[1] = {0.0};
    for (int64_t i = (int64_t)blockIdx.x * kRedThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kRedThreads)
        v[0] += a[i] * b[i];
    if (grid_reduce<1, 0u>(v, part, ticket)) *out = v[0];
}

// The start of a solve in one pass: xd = b on masked DOFs, r = b on free ones, xf = 0;
// out = {b.b, xd.xd, r.r}
__global__ void __launch_bounds__(kRedThreads) solve_begin_kernel(int64_t n, const double* __restrict__ b,
                                                                  const uint8_t* __restrict__ mask,
                                                                  double* __restrict__ xd, double* __restrict__ xf,
                                                                  double* __restrict__ r, double* part, unsigned* ticket,
                                                                  double* out) {
    double v[3] = {0.0, 0.0, 0.0};
    for (int64_t i = (int64_t)blockIdx.x * kRedThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kRedThreads) {
        const double bi = b[i], d = mask[i] ? bi : 0.0, f = mask[i] ? 0.0 : bi;
        xd[i] = d;
        xf[i] = 0.0;
        r[i] = f;
        v[0] += bi * bi;
        v[1] += d * d;
        v[2] += f * f;
    }
    if (grid_reduce<3, 0u>(v, part, ticket)) {
        out[0] = v[0];
        out[1] = v[1];
        out[2] = v[2];
    }
}

// xf += a d, sum = xd + xf: the refinement's new iterate and the point of its residual
template <typename T>
__global__ void refine_update_kernel(int64_t n, double a, const T* __restrict__ d, const double* __restrict__ xd,
                                     double* __restrict__ xf, double* __restrict__ sum) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double f = xf[i] + a * (double)d[i];
    xf[i] = f;
    sum[i] = xd[i] + f;
}

// small vector kernels
template <typename T>
__global__ void masked_copy_kernel(int64_t n, const double* __restrict__ src, const uint8_t* __restrict__ mask,
                                   int keepMasked, double scale, T* __restrict__ dst) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool m = mask && mask[i];
    dst[i] = (T)((m == (keepMasked != 0)) ? src[i] * scale : 0.0);
}

template <typename T>
__global__ void axpy_kernel(int64_t n, double a, const T* __restrict__ xs, double* __restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] += a * (double)xs[i];
}

__global__ void add_kernel(int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                           double* __restrict__ y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = a[i] + b[i];
}

}  // namespace ef

using namespace ef;

static inline int nb(int64_t n, int t) { return (int)((n + t - 1) / t); }

constexpr int kPcgMaxCopies = 16;
// lanes per block row: as many as let a CTA's rows through in one pass (32: a block each), at least 4, and
// in FP64 at most 8 (a row's last steps and lane sums cost its narrow pipe more than a longer chain)
static int pcg_lanes(int rows, int tpb, int vDouble) {
    int lpr = vDouble ? 8 : 32;
    while (lpr > 4 && rows * lpr > tpb) lpr /= 2;
    return lpr;
}

int ef_pcg_slot_sets() { return kPcgMaxCopies; }
size_t ef_pcg_slot_bytes(int sets) { return sets * kPcgSlotBytes; }

ef_status ef_launch_bsr_residual(int nNodes, const int32_t* rowPtr, const int32_t* colIdx, const void* vals,
                                 int mDouble, const double* x, const double* b, const uint8_t* mask, double* y,
                                 int nSM, cudaStream_t s) {
    if (nNodes == 0) return EF_OK;
    const int groups = kKB / kRowLanes;
    int grid = nb(nNodes, groups);
    const int cap = nSM * 8;
    if (grid > cap) grid = cap;
    if (mDouble)
        bsr_residual_kernel<double, double, double><<<grid, kKB, 0, ef::counted(s)>>>(nNodes, rowPtr, colIdx, (const double*)vals,
                                                                       x, b, mask, y);
    else
        bsr_residual_kernel<float, double, double><<<grid, kKB, 0, ef::counted(s)>>>(nNodes, rowPtr, colIdx, (const float*)vals, x,
                                                                      b, mask, y);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

// Lanes per block row, CTAs and slot sets of the PCG on n block rows.  Fewer CTAs make a reduction
// cheaper and an iteration's work per SM larger: 128 rows a CTA in FP32 (4,836 nodes: 9.1 us an
// iteration with 38 CTAs, 9.4 with 76, 10.1 with 152) and 16 in FP64, whose pipe bounds the product (525 nodes: 9.8 us
// with 33 CTAs, 10.5 with 132, 22 with 5), up to one CTA per SM.
static void pcg_shape(int vDouble, int n, int nSM, PcgShape* p) {
    const int tpb = vDouble ? PcgTpb<double>::value : PcgTpb<float>::value;
    const int least = vDouble ? 16 : 128;
    p->cluster = false;
    p->grid = std::max(1, std::min(std::min(nSM, kPcgMaxCtas), (n + least - 1) / least));
    p->copies = p->grid <= 16 ? 1 : (p->grid <= 64 ? 4 : kPcgMaxCopies);
    p->lpr = pcg_lanes((n + p->grid - 1) / p->grid, tpb, vDouble);
}

// the lanes that pcg_lanes gives: 4 to 32 for FP32 vectors, 4 and 8 for FP64 ones
#define EF_PCG(K, ...)                                                                                       \
    (vDouble ? (lpr == 8 ? (const void*)K<double, 8, ##__VA_ARGS__> : (const void*)K<double, 4, ##__VA_ARGS__>) \
     : lpr == 32 ? (const void*)K<float, 32, ##__VA_ARGS__>                                                  \
     : lpr == 16 ? (const void*)K<float, 16, ##__VA_ARGS__>                                                  \
     : lpr == 8  ? (const void*)K<float, 8, ##__VA_ARGS__>                                                   \
                 : (const void*)K<float, 4, ##__VA_ARGS__>)
static const void* pcg_kernel(int vDouble, int lpr) { return EF_PCG(pcg_persistent_kernel); }
static const void* pcg_resident(int vDouble, int lpr, bool cluster) {
    return cluster ? EF_PCG(pcg_resident_kernel, true) : EF_PCG(pcg_resident_kernel, false);
}
#undef EF_PCG

// The resident form's plan for a host block pattern and a given shape: for every CTA the rows outside
// its range that its rows couple to (increasing), the first step of each group of rows (see
// ResidentLayout), and for every block the place of its column among the CTA's rows and halo.  False
// when a CTA's part does not fit into shared memory.
static bool plan_for(int vDouble, const PcgShape& shape, int nNodes, const int32_t* rowPtr, const int32_t* colIdx,
                     PcgResidentPlan& p) {
    const size_t vt = vDouble ? sizeof(double) : sizeof(float);
    const int grid = shape.grid, lpr = shape.lpr;
    const int per = (nNodes + grid - 1) / grid, rpw = 32 / lpr, groups = (per + rpw - 1) / rpw;
    size_t room = 0;
    if (ef::smem_room(pcg_resident(vDouble, lpr, shape.cluster), &room) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    p = PcgResidentPlan();
    p.shape = shape;
    // the steps first: they need no halo, so that a large system's plan is not begun
    p.groupPtr.reserve((size_t)grid * (groups + 1));
    for (int g = 0; g < grid; ++g) {
        const int r0 = std::min(nNodes, g * per), r1 = std::min(nNodes, r0 + per);
        int steps = 0;
        for (int q = 0; q < groups; ++q) {
            p.groupPtr.push_back(steps);
            int w = 0;
            for (int m = r0 + q * rpw; m < std::min(r1, r0 + (q + 1) * rpw); ++m)
                w = std::max(w, (rowPtr[m + 1] - rowPtr[m] + lpr - 1) / lpr);
            steps += w;
        }
        p.groupPtr.push_back(steps);
        if (resident_layout(vt, r1 - r0, 0, steps).bytes > room) return false;
    }
    std::vector<int32_t> place(nNodes, -1);
    p.lcol.resize(rowPtr[nNodes]);
    p.haloPtr.assign(1, 0);
    for (int g = 0; g < grid; ++g) {
        const int r0 = std::min(nNodes, g * per), r1 = std::min(nNodes, r0 + per);
        const size_t h0 = p.haloIdx.size();
        for (int32_t k = rowPtr[r0]; k < rowPtr[r1]; ++k) {
            const int32_t c = colIdx[k];
            if ((c < r0 || c >= r1) && place[c] < 0) {
                place[c] = 0;
                p.haloIdx.push_back(c);
            }
        }
        std::sort(p.haloIdx.begin() + h0, p.haloIdx.end());
        const int nh = (int)(p.haloIdx.size() - h0);
        for (int i = 0; i < nh; ++i) place[p.haloIdx[h0 + i]] = r1 - r0 + i;
        const size_t need = resident_layout(vt, r1 - r0, nh, p.groupPtr[(size_t)g * (groups + 1) + groups]).bytes;
        if (need > room || r1 - r0 + nh > 65535) return false;
        p.smem = std::max(p.smem, need);
        for (int32_t k = rowPtr[r0]; k < rowPtr[r1]; ++k) {
            const int32_t c = colIdx[k];
            p.lcol[k] = (uint16_t)(c >= r0 && c < r1 ? c - r0 : place[c]);
        }
        for (int i = 0; i < nh; ++i) place[p.haloIdx[h0 + i]] = -1;
        p.haloPtr.push_back((int32_t)p.haloIdx.size());
    }
    return true;
}

static cudaLaunchConfig_t cluster_config(const PcgShape& shape, int vDouble, size_t smem, cudaStream_t s,
                                         cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(shape.grid);
    cfg.blockDim = dim3(vDouble ? PcgTpb<double>::value : PcgTpb<float>::value);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = shape.grid;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// The rule of the dispatch.  A system that fits into one cluster's shared memory (about 3,200 rows of 27
// blocks in FP32, 1,600 in FP64) runs there: a reduction through the cluster's barrier costs about half
// of one through L2 (us an iteration in the cluster and in the grid form: FP32, 624 nodes 5.3 and 8.2, 2,730 nodes 6.2
// and 8.6; FP64, 525 nodes 7.8 and 9.8, but 1,440 nodes, for which the FP64 pipes of 16 SMs are few, 12.9 and 10.6).  Else one that fits into all SMs' shared memory runs in the grid form.  Else
// plan.smem is 0: the streaming kernel.
void ef_pcg_resident_plan(int vDouble, int nSM, int nNodes, const int32_t* rowPtr, const int32_t* colIdx,
                          PcgResidentPlan& plan) {
    const int tpb = vDouble ? PcgTpb<double>::value : PcgTpb<float>::value;
    PcgShape shape;
    shape.cluster = true;
    shape.copies = 1;
    // the smallest cluster whose CTAs' lanes cover their rows with 8 (FP64: 16 rows a CTA), at most 16
    const int rows = vDouble ? 16 : tpb / 8;
    for (shape.grid = 1; shape.grid < kPcgMaxCluster && shape.grid * rows < nNodes;) shape.grid *= 2;
    shape.lpr = pcg_lanes((nNodes + shape.grid - 1) / shape.grid, tpb, vDouble);
    if (plan_for(vDouble, shape, nNodes, rowPtr, colIdx, plan)) {
        const void* k = pcg_resident(vDouble, shape.lpr, true);
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = cluster_config(shape, vDouble, plan.smem, 0, &attr);
        int fit = 0;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&fit, k, &cfg) == cudaSuccess && fit > 0)
            return;
        (void)cudaGetLastError();
    }
    pcg_shape(vDouble, nNodes, nSM, &shape);
    if (!plan_for(vDouble, shape, nNodes, rowPtr, colIdx, plan)) plan = PcgResidentPlan();
}

// EF_PCG_POLLS: another limit, for the tests of a wait that runs out
static PcgWait pcg_wait(void* res, int* flags) {
    const char* e = getenv("EF_PCG_POLLS");
    return PcgWait{(PcgResult*)res, flags, e ? (unsigned)strtoul(e, nullptr, 10) : kPcgSpinLimit};
}

// The resident form with its plan on the device; shape and smem as ef_pcg_resident_plan returned them (which has
// allowed the kernel that much shared memory and the cluster's size)
ef_status ef_launch_pcg_resident(int vDouble, const PcgShape& shape, int nNodes, const int32_t* rowPtr,
                                 const uint16_t* lcol, const int32_t* haloPtr, const int32_t* haloIdx,
                                 const int32_t* groupPtr, size_t smem, const void* vals, const void* binv,
                                 const uint8_t* mask, const void* b, void* x, void* z, double* slots, void* res,
                                 int maxIter, double rtol2, int* flags, cudaStream_t s) {
    int copies = shape.copies;
    PcgWait wait = pcg_wait(res, flags);
    void* args[] = {&nNodes, &rowPtr, &lcol, &haloPtr, &haloIdx, &groupPtr, &vals, &binv, &mask, &b, &x, &z,
                    &slots, &copies, &wait, &maxIter, &rtol2};
    const void* k = pcg_resident(vDouble, shape.lpr, shape.cluster);
    ef::note_launches(1);
    if (shape.cluster) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = cluster_config(shape, vDouble, smem, s, &attr);
        EF_CUDA(cudaLaunchKernelExC(&cfg, k, args));
        return EF_OK;
    }
    EF_CUDA(cudaMemsetAsync(slots, 0xff, copies * kPcgSlotBytes, s));
    EF_CUDA(cudaLaunchCooperativeKernel(k, shape.grid, vDouble ? PcgTpb<double>::value : PcgTpb<float>::value, args, smem, s));
    return EF_OK;
}

// slots: ef_pcg_slot_bytes(slotSets) of device memory (set here, stream ordered)
ef_status ef_launch_pcg(int vDouble, int nSM, int nNodes, const int32_t* rowPtr, const int32_t* colIdx,
                        const void* vals, const void* binv, const uint8_t* mask, const void* b, void* x, void* r,
                        void* z, void* pA, void* pB, void* q, double* slots, int slotSets, void* res, int maxIter,
                        double rtol2, int* flags, cudaStream_t s) {
    PcgShape shape;
    pcg_shape(vDouble, nNodes, nSM, &shape);
    int copies = std::min(shape.copies, slotSets);
    PcgWait wait = pcg_wait(res, flags);
    void* args[] = {&nNodes, &rowPtr, &colIdx, &vals, &binv, &mask, &b, &x, &r, &z, &pA, &pB, &q,
                    &slots, &copies, &wait, &maxIter, &rtol2};
    EF_CUDA(cudaMemsetAsync(slots, 0xff, copies * kPcgSlotBytes, s));
    ef::note_launches(1);
    EF_CUDA(cudaLaunchCooperativeKernel(pcg_kernel(vDouble, shape.lpr), shape.grid,
                                        vDouble ? PcgTpb<double>::value : PcgTpb<float>::value, args, 0, s));
    return EF_OK;
}

ef_status ef_launch_dot(int64_t n, const double* a, const double* b, double* part, int nPart, unsigned* ticket,
                        double* out, cudaStream_t s) {
    dot_kernel<<<reduce_grid(n, nPart), kRedThreads, 0, ef::counted(s)>>>(n, a, b, part, ticket, out);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_solve_begin(int64_t n, const double* b, const uint8_t* mask, double* xd, double* xf, double* r,
                                double* part, int nPart, unsigned* ticket, double* out, cudaStream_t s) {
    solve_begin_kernel<<<reduce_grid(n, nPart), kRedThreads, 0, ef::counted(s)>>>(n, b, mask, xd, xf, r, part, ticket,
                                                                                out);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_refine_update(int64_t n, double a, const void* d, int dDouble, const double* xd, double* xf,
                                  double* sum, cudaStream_t s) {
    if (n == 0) return EF_OK;
    if (dDouble)
        refine_update_kernel<double><<<nb(n, 256), 256, 0, ef::counted(s)>>>(n, a, (const double*)d, xd, xf, sum);
    else
        refine_update_kernel<float><<<nb(n, 256), 256, 0, ef::counted(s)>>>(n, a, (const float*)d, xd, xf, sum);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_masked_copy(int64_t n, const double* src, const uint8_t* mask, int keepMasked, double scale,
                                void* dst, int dstDouble, cudaStream_t s) {
    if (n == 0) return EF_OK;
    if (dstDouble)
        masked_copy_kernel<double><<<nb(n, 256), 256, 0, ef::counted(s)>>>(n, src, mask, keepMasked, scale, (double*)dst);
    else
        masked_copy_kernel<float><<<nb(n, 256), 256, 0, ef::counted(s)>>>(n, src, mask, keepMasked, scale, (float*)dst);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_axpy(int64_t n, double a, const void* xs, int xDouble, double* y, cudaStream_t s) {
    if (n == 0) return EF_OK;
    if (xDouble)
        axpy_kernel<double><<<nb(n, 256), 256, 0, ef::counted(s)>>>(n, a, (const double*)xs, y);
    else
        axpy_kernel<float><<<nb(n, 256), 256, 0, ef::counted(s)>>>(n, a, (const float*)xs, y);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_add(int64_t n, const double* a, const double* b, double* y, cudaStream_t s) {
    if (n == 0) return EF_OK;
    add_kernel<<<nb(n, 256), 256, 0, ef::counted(s)>>>(n, a, b, y);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

// ---------------------------------------------------------------------------------------------
// Allocation-free block-Jacobi PCG (ef_pcg_solve_noalloc).
//
// Some callers cannot allocate device memory at solve time: a host framework that has reserved
// the device memory for its own pool, or a latency-critical loop that must not take the
// device-wide synchronisation that cudaMalloc/cudaFree imply.  This entry point solves with the
// same persistent PCG kernel as ef_solve, but its work vectors live in a fixed file-scope device
// array instead of a context workspace, so the call itself allocates nothing.
// ---------------------------------------------------------------------------------------------

#include <mutex>

#define EF_NOALLOC_SCRATCH_BYTES (8u << 20)  // 8 MiB held by every device that loads the library
static __device__ __align__(256) unsigned char g_noallocScratch[EF_NOALLOC_SCRATCH_BYTES];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noallocMutex;
void* g_noallocPtr[kMaxDevices] = {};
int g_noallocSMs[kMaxDevices] = {};

inline size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }
}  // namespace

extern "C" int64_t ef_pcg_noalloc_max_nodes(void) {
    // layout: the reduction slots (kPcgSlotBytes, in 2 x 16 KiB), the result record, then five FP64
    // work vectors of 3*nNodes entries each
    // (the last 256 bytes hold the call's device flags word)
    const size_t fixed = 2 * align256(4 * sizeof(double) * 512) + align256(sizeof(PcgResult)) + 256;
    return (int64_t)((EF_NOALLOC_SCRATCH_BYTES - fixed - 5 * 256) / (5 * 3 * sizeof(double)));
}

extern "C" ef_status ef_pcg_solve_noalloc(int64_t nNodes, const int32_t* rowPtr, const int32_t* colIdx,
                                          const double* vals, const double* binv, const uint8_t* mask,
                                          const double* b, double* x, int maxIter, double rtol, ef_solve_info* info,
                                          void* stream) {
    if (nNodes <= 0 || !rowPtr || !colIdx || !vals || !binv || !mask || !b || !x || maxIter < 0 || !(rtol >= 0.0)) {
        ef_set_error("ef_pcg_solve_noalloc: invalid arguments");
        return EF_ERR_ARG;
    }
    if (nNodes > ef_pcg_noalloc_max_nodes()) {
        ef_set_error("ef_pcg_solve_noalloc: " + std::to_string(nNodes) + " block rows exceed the fixed scratch capacity of " +
                     std::to_string(ef_pcg_noalloc_max_nodes()) + " block rows (8 MiB); use ef_solve");
        return EF_ERR_ARG;
    }
    int dev = 0;
    EF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        ef_set_error("ef_pcg_solve_noalloc: device index out of range");
        return EF_ERR_ARG;
    }
    {
        // once per device, with that device current: the device address of the scratch array
        std::lock_guard<std::mutex> lock(g_noallocMutex);
        if (!g_noallocPtr[dev]) {
            void* p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_noallocScratch);
            if (e != cudaSuccess || !p) {
                ef_set_error(std::string("ef_pcg_solve_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
                return EF_ERR_CUDA;
            }
            EF_CUDA(cudaDeviceGetAttribute(&g_noallocSMs[dev], cudaDevAttrMultiProcessorCount, dev));
            // a kernel's code goes to the device when it is first used: all of them now, so that no later call does that
            for (int lpr = 4; lpr <= 8; lpr *= 2) {
                cudaFuncAttributes fa;
                EF_CUDA(cudaFuncGetAttributes(&fa, pcg_kernel(1, lpr)));
            }
            g_noallocPtr[dev] = p;
        }
    }
    unsigned char* base = (unsigned char*)g_noallocPtr[dev];
    const size_t slotBytes = 2 * align256(4 * sizeof(double) * 512);
    double* slots = (double*)base;
    PcgResult* res = (PcgResult*)(base + slotBytes);
    unsigned char* vec = base + slotBytes + align256(sizeof(PcgResult));
    const size_t vb = align256(3 * (size_t)nNodes * sizeof(double));
    double* r = (double*)(vec + 0 * vb);
    double* z = (double*)(vec + 1 * vb);
    double* pA = (double*)(vec + 2 * vb);
    double* pB = (double*)(vec + 3 * vb);
    double* q = (double*)(vec + 4 * vb);
    // device flags word: the last 256 bytes of the scratch array, cleared for this call
    int* flags = (int*)(base + EF_NOALLOC_SCRATCH_BYTES - 256);
    cudaStream_t s = (cudaStream_t)stream;
    EF_CUDA(cudaMemsetAsync(flags, 0, sizeof(int), s));
    const ef_status ls = ef_launch_pcg(1, g_noallocSMs[dev], (int)nNodes, rowPtr, colIdx, vals, binv, mask, b, x, r, z,
                                       pA, pB, q, slots, 2, res, maxIter, rtol * rtol, flags, s);
    if (ls != EF_OK) return ls;
    PcgResult hr;
    int hf = 0;
    EF_CUDA(cudaMemcpyAsync(&hr, res, sizeof(hr), cudaMemcpyDeviceToHost, s));
    EF_CUDA(cudaMemcpyAsync(&hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, s));
    EF_CUDA(cudaStreamSynchronize(s));
    if (hf & EF_FLAG_BARRIER) {
        ef_set_error("ef_pcg_solve_noalloc: grid barrier timed out");
        return EF_ERR_DEVICE;
    }
    const double rel = hr.bb > 0.0 ? sqrt(hr.rr / hr.bb) : 0.0;
    if (info) {
        info->iterations = hr.iterations;
        info->refinements = 0;
        info->relResidual = rel;
        info->status = hr.status;
        info->kernelMs = 0.0;
        info->kernelLaunches = 1;
    }
    if (hr.status != EF_OK) {
        char msg[160];
        snprintf(msg, sizeof msg, "ef_pcg_solve_noalloc: status %d after %d iterations, relative residual %.3e",
                 hr.status, hr.iterations, rel);
        ef_set_error(msg);
    }
    return hr.status == EF_OK ? EF_OK : (ef_status)hr.status;
}
