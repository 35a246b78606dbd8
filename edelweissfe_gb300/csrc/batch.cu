// Batched solve of many independent small problems held in one context.
//
// The problems are disjoint meshes whose nodes occupy contiguous ranges [nodePtr[p],
// nodePtr[p+1]) of the context's 3x3-block system, so the assembled system is block diagonal by
// problem.  One persistent launch solves all of them: every cluster of CTAs takes the next problem of a
// list sorted by decreasing size (a ticket counter) and runs block-Jacobi PCG on it, its CTAs sharing
// the rows, with reductions through the cluster's distributed shared memory only, so problems of uneven
// size need no grid barrier.  Each problem has its own step lengths, its own stopping test
// (|r| <= rtol |b| on the problem's own right-hand side) and its own iteration count.  Reductions are
// fixed shuffle trees in a fixed order over CTAs: deterministic for a given cluster size (chosen from the
// problems' sizes, ef_batch_cluster_size) and tile shape (threads per CTA, lanes per block row), which a
// timing autotuner picks; which cluster takes a problem does not enter.
//
// What bounds it: the FP64 pipe (2 lanes per SM and cycle: 9 fused multiply-adds a block are 4.5 cycles of
// an SM; the 72 bytes of a block at 1/152 of the measured HBM rate are 3.3) and, before clusters, the
// largest problems, each of which had one SM (and a sum of products took four FP64 instructions where a chain
// of fused multiply-adds takes three).  Load increments, before and now: 160 cubes of 4..16 elements an
// edge 1.03 -> 0.31 s, 11 cubes of 4..9 elements 69 -> 9 ms; one solve of 1024 cubes 164 -> 83 ms.
//
// The per-problem Newton checks of the reference's NIST driver (solvers/nonlinearimplicitstatic.py
// :625-725) need max|R|, sum|F| and max|ddU| per problem: batch_norms_kernel, one CTA per problem.

#include <algorithm>
#include <cmath>
#include <functional>
#include <vector>

#include "cluster.cuh"
#include "ef_common.cuh"
#include "pcg_plan.h"

namespace ef {

constexpr int kBatchMaxCluster = 8;

template <int TPB>
struct BatchShared {
    double red[2][TPB];
    double part[2][kBatchMaxCluster][2];  // sums of the cluster's CTAs, double buffered
    double scalar;                        // the step length or direction factor of the current phase
    int go;
    int next[2];                          // the cluster's problem, double buffered
};

// Sums of NV values over the cluster's threads, in a fixed order; the first thread of every CTA gets them
// and makes the next scalar with `next(sum)`, which returns whether to go on.  Entry tid < count of each
// CTA counts.  One warp adds and one thread divides: a warp's FP64 instruction takes the pipe 16 cycles.
// Behind it every thread sees what the cluster wrote before it.
template <int TPB, int NV, bool MULTI, typename F>
__device__ __forceinline__ bool batch_sum(const double (&v)[NV], int count, BatchShared<TPB>& sh, int nCta, int rank,
                                          int& epoch, F next) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if ((int)threadIdx.x < count)
#pragma unroll
        for (int j = 0; j < NV; ++j) sh.red[j][threadIdx.x] = v[j];
    __syncthreads();
    double t[NV];
    if (w == 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) t[j] = lane < count ? sh.red[j][lane] : 0.0;
        for (int i = lane + 32; i < count; i += 32)
#pragma unroll
            for (int j = 0; j < NV; ++j) t[j] += sh.red[j][i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < NV; ++j) t[j] += __shfl_xor_sync(0xffffffffu, t[j], o);
        if (MULTI && lane < nCta)
            cluster_store(cluster_addr(sh.part[epoch & 1][rank], lane), (unsigned long long)__double_as_longlong(t[0]),
                          (unsigned long long)__double_as_longlong(t[NV - 1]));
    }
    if (MULTI) {
        cluster_barrier();
        if (w == 0) {
#pragma unroll
            for (int j = 0; j < NV; ++j) t[j] = lane < nCta ? sh.part[epoch & 1][lane][j] : 0.0;
#pragma unroll
            for (int o = kBatchMaxCluster / 2; o > 0; o >>= 1)
#pragma unroll
                for (int j = 0; j < NV; ++j) t[j] += __shfl_xor_sync(0xffffffffu, t[j], o);
        }
    }
    if (threadIdx.x == 0) sh.go = next(t) ? 1 : 0;
    __syncthreads();
    ++epoch;
    return sh.go != 0;
}

// TPB threads per CTA; the products use LPR lanes per block row (strided over the row's blocks,
// combined by a fixed shuffle tree), the vector updates one thread per DOF.  The blocks are read from
// a sliced copy (batch_slice_kernel): rows in groups of 32 / LPR, step j of a group holding lane l's j-th
// block in nine planes of 32 values, so that a warp's loads are contiguous (from the block rows they
// touch 18 lines each).  Up to 512 threads' worth of registers (128 a thread) keep two steps of loads in
// flight; with 64 the same shapes took a fifth longer.  MULTI: clusters of more than one CTA; p is then gathered through L2.
// SLICED = false: no memory for the sliced copy; the blocks are read from the block rows themselves, lane l's j-th
// block in the same order (the same sums; ms of a solve with the copy and without: one cube of 8 elements an edge 1.44 and
// 1.59, 160 of 4..16 33.0 and 33.5, with one lane per row 66.5 and 89.9).
template <int TPB, int LPR, bool MULTI, bool SLICED>
__global__ void __launch_bounds__(TPB, 512 / TPB) batched_pcg_kernel(
    int nProb, const int32_t* __restrict__ nodePtr, const int32_t* __restrict__ order,
    const int32_t* __restrict__ groupBase, const int32_t* __restrict__ groupPtr, const int32_t* __restrict__ rowPtr,
    const int32_t* __restrict__ col, const double* __restrict__ vals, const double* __restrict__ binv, const uint8_t* __restrict__ mask,
    const double* __restrict__ b, double* x, double* rA, double* rB, double* z, double* p, double* q, int maxIter,
    double rtol2, int* __restrict__ itersOut, double* __restrict__ relOut, int* ticket) {
    constexpr int RPW = 32 / LPR;  // rows of a group
    __shared__ __align__(16) BatchShared<TPB> sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int l = lane % LPR;
    const int nCta = MULTI ? (int)cluster_size() : 1, rank = MULTI ? (int)cluster_rank() : 0;
    int epoch = 0;
    if (MULTI) cluster_barrier();  // every CTA's shared memory is there before the first remote store
    for (int turn = 0;; ++turn) {
        if (rank == 0 && tid == 0) {
            const int k = atomicAdd(ticket, 1);
            for (int c = 0; c < nCta; ++c) {
                if (MULTI)
                    cluster_store(cluster_addr(&sh.next[turn & 1], c), (unsigned)k);
                else
                    sh.next[turn & 1] = k;
            }
        }
        if (MULTI)
            cluster_barrier();
        else
            __syncthreads();
        const int k = sh.next[turn & 1];
        if (k >= nProb) break;
        const int pid = order[k];
        const int n0 = nodePtr[pid], n1 = nodePtr[pid + 1];
        const int nGroups = (n1 - n0 + RPW - 1) / RPW, per = (nGroups + nCta - 1) / nCta;
        const int g0 = min(nGroups, rank * per), g1 = min(nGroups, g0 + per);
        const int r0 = min(n1, n0 + g0 * RPW), r1 = min(n1, n0 + g1 * RPW);
        const int32_t* gp = groupPtr + groupBase[pid];
        const int countV = min(TPB, 3 * (r1 - r0));
        // of thread 0 of every CTA
        double rz = 0.0, rr = 0.0, bb = 0.0;
        bool ok = true;
        double* r = rA;
        double* r2 = rB;
        double s2[2] = {0.0, 0.0};
        for (int d = 3 * r0 + tid; d < 3 * r1; d += TPB) {
            const int m = d / 3, i = d - 3 * m;
            double rv[3];
#pragma unroll
            for (int j = 0; j < 3; ++j) rv[j] = mask[3 * m + j] ? 0.0 : b[3 * m + j];
            const double* B = binv + (int64_t)m * 9 + 3 * i;
            const double ri = i == 0 ? rv[0] : (i == 1 ? rv[1] : rv[2]);
            const double zi = mask[d] ? 0.0 : B[0] * rv[0] + B[1] * rv[1] + B[2] * rv[2];
            x[d] = 0.0;
            r[d] = ri;
            z[d] = zi;
            p[d] = zi;
            s2[0] += ri * zi;
            s2[1] += ri * ri;
        }
        bool go = batch_sum<TPB, 2, MULTI>(s2, countV, sh, nCta, rank, epoch, [&](const double(&t)[2]) {
            rz = t[0];
            rr = bb = t[1];
            return bb > 0.0 && rr > rtol2 * bb;
        });
        int it = 0;
        while (go && it < maxIter) {
            // q = A p on free rows; p.q
            double pq[1] = {0.0};
            for (int g = g0 + warp; g < g1; g += TPB / 32) {
                const int m = n0 + g * RPW + lane / LPR;
                // block j of the lane: step j of the sliced copy, or entry j of the block row
                const int j0 = SLICED ? gp[g] : (m < r1 ? rowPtr[m] + l : 0);
                const int j1 = SLICED ? gp[g + 1] : (m < r1 ? rowPtr[m + 1] : 0);
                double y0 = 0.0, y1 = 0.0, y2 = 0.0;
#pragma unroll 2
                for (int j = j0; j < j1; j += SLICED ? 1 : LPR) {
                    const double* v = vals + (SLICED ? (int64_t)288 * j + lane : (int64_t)9 * j);
                    const double* pv = p + 3 * (int64_t)__ldg(col + (SLICED ? 32 * (int64_t)j + lane : (int64_t)j));
                    double a[9];
#pragma unroll
                    for (int i = 0; i < 9; ++i) a[i] = __ldg(v + (SLICED ? 32 * i : i));
                    const double p0 = MULTI ? __ldcg(pv) : pv[0], p1 = MULTI ? __ldcg(pv + 1) : pv[1],
                                 p2 = MULTI ? __ldcg(pv + 2) : pv[2];
                    block_fma(a, p0, p1, p2, y0, y1, y2);
                }
                if constexpr (LPR == 1) {
                    if (m < r1) {
                        const double yy[3] = {y0, y1, y2};
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            const int d = 3 * m + i;
                            const double qi = mask[d] ? 0.0 : yy[i];
                            q[d] = qi;
                            pq[0] += p[d] * qi;
                        }
                    }
                } else {
                    const double yy = row_sum3<LPR>(l, y0, y1, y2);
                    if (l % (LPR / 4) == 0 && l / (LPR / 4) < 3 && m < r1) {
                        const int d = 3 * m + l / (LPR / 4);
                        const double qi = mask[d] ? 0.0 : yy;
                        q[d] = qi;
                        pq[0] += p[d] * qi;
                    }
                }
            }
            go = batch_sum<TPB, 1, MULTI>(pq, min(TPB, 32 * (g1 - g0)), sh, nCta, rank, epoch, [&](const double(&t)[1]) {
                sh.scalar = rz / t[0];
                ok = t[0] == t[0];
                return t[0] > 0.0;  // breakdown or NaN: stop with the current iterate
            });
            if (!go) break;
            const double alpha = sh.scalar;
            s2[0] = s2[1] = 0.0;
            for (int d = 3 * r0 + tid; d < 3 * r1; d += TPB) {
                // r of the node's three DOFs in each of its threads; the new r goes to the other buffer
                const int m = d / 3, i = d - 3 * m;
                double rv[3];
#pragma unroll
                for (int j = 0; j < 3; ++j) rv[j] = r[3 * m + j] - alpha * q[3 * m + j];
                const double* B = binv + (int64_t)m * 9 + 3 * i;
                const double ri = i == 0 ? rv[0] : (i == 1 ? rv[1] : rv[2]);
                const double zi = mask[d] ? 0.0 : B[0] * rv[0] + B[1] * rv[1] + B[2] * rv[2];
                x[d] += alpha * p[d];
                r2[d] = ri;
                z[d] = zi;
                s2[0] += ri * zi;
                s2[1] += ri * ri;
            }
            double* t = r;
            r = r2;
            r2 = t;
            go = batch_sum<TPB, 2, MULTI>(s2, countV, sh, nCta, rank, epoch, [&](const double(&t)[2]) {
                sh.scalar = t[0] / rz;
                rz = t[0];
                rr = t[1];
                return rr > rtol2 * bb;
            });
            ++it;
            if (!go) break;
            const double beta = sh.scalar;
            for (int d = 3 * r0 + tid; d < 3 * r1; d += TPB) p[d] = z[d] + beta * p[d];
            if (MULTI)
                cluster_barrier();  // p complete before the next product
            else
                __syncthreads();
        }
        if (rank == 0 && tid == 0) {
            itersOut[pid] = it;
            relOut[pid] = !ok ? __longlong_as_double(0x7ff8000000000000LL) : (bb > 0.0 ? sqrt(rr / bb) : 0.0);
        }
    }
}

// The sliced copy's values and columns from the block rows: a warp per group of 32 / LPR rows (padding: zero
// blocks in the group's first row's column)
template <int LPR>
__global__ void __launch_bounds__(256) batch_slice_kernel(int nGroups, const int32_t* __restrict__ groupRow,
                                                          const int32_t* __restrict__ groupEnd,
                                                          const int32_t* __restrict__ groupStep,
                                                          const int32_t* __restrict__ rowPtr,
                                                          const int32_t* __restrict__ colIdx,
                                                          const double* __restrict__ bsr, double* __restrict__ vals,
                                                          int32_t* __restrict__ col) {
    const int lane = threadIdx.x & 31;
    for (int g = (blockIdx.x * 256 + threadIdx.x) >> 5; g < nGroups; g += gridDim.x * 8) {
        const int row0 = groupRow[g], m = row0 + lane / LPR;
        const int k0 = m < groupEnd[g] ? rowPtr[m] : 0, k1 = m < groupEnd[g] ? rowPtr[m + 1] : 0;
        const int j0 = groupStep[2 * g], j1 = groupStep[2 * g + 1];
        for (int j = j0; j < j1; ++j) {
            const int64_t kk = k0 + lane % LPR + (int64_t)(j - j0) * LPR;
            double* d = vals + (int64_t)288 * j + lane;
#pragma unroll
            for (int i = 0; i < 9; ++i) d[32 * i] = kk < k1 ? bsr[9 * kk + i] : 0.0;
            col[32 * (int64_t)j + lane] = kk < k1 ? colIdx[kk] : row0;
        }
    }
}

// out[p] = {max |R|, sum |F|, max |ddU|} over the DOFs of problem p (ddU may be null)
__global__ void __launch_bounds__(256) batch_norms_kernel(int nProb, const int32_t* __restrict__ nodePtr,
                                                          const double* __restrict__ R, const double* __restrict__ F,
                                                          const double* __restrict__ D, double* __restrict__ out) {
    __shared__ double red[3][8];
    const int pid = blockIdx.x;
    if (pid >= nProb) return;
    const int d0 = 3 * nodePtr[pid], d1 = 3 * nodePtr[pid + 1];
    double a = 0.0, s = 0.0, c = 0.0;
    for (int d = d0 + (int)threadIdx.x; d < d1; d += 256) {
        a = fmax(a, fabs(R[d]));
        s += fabs(F[d]);
        if (D) c = fmax(c, fabs(D[d]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fmax(a, __shfl_xor_sync(0xffffffffu, a, o));
        s += __shfl_xor_sync(0xffffffffu, s, o);
        c = fmax(c, __shfl_xor_sync(0xffffffffu, c, o));
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        red[0][w] = a;
        red[1][w] = s;
        red[2][w] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double A = 0.0, S = 0.0, C = 0.0;
        for (int i = 0; i < 8; ++i) {
            A = fmax(A, red[0][i]);
            S += red[1][i];
            C = fmax(C, red[2][i]);
        }
        out[3 * pid] = A;
        out[3 * pid + 1] = S;
        out[3 * pid + 2] = C;
    }
}

template <int TPB, int LPR, bool MULTI, bool SLICED>
static ef_status launch_batched(const BatchPlanDev& pl, int cluster, int nSM, int nProb, const int32_t* rowPtr,
                                const int32_t* col, const double* vals, const double* binv, const uint8_t* mask, const double* b, double* x, double* r, double* r2, double* z,
                                double* p, double* q, int maxIter, double rtol2, int* iters, double* rel, int* ticket,
                                cudaStream_t s) {
    auto k = batched_pcg_kernel<TPB, LPR, MULTI, SLICED>;
    int perSM = 0;
    EF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k, TPB, 0));
    // as many clusters as are resident at once; a cluster that is scheduled later finds the list empty
    const int clusters = std::max(1, std::min(nProb, std::max(1, perSM) * nSM / cluster));
    EF_CUDA(cudaMemsetAsync(ticket, 0, sizeof(int), s));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * cluster);
    cfg.blockDim = dim3(TPB);
    cfg.stream = ef::counted(s);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = cluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    EF_CUDA(cudaLaunchKernelEx(&cfg, k, nProb, pl.nodePtr, pl.order, pl.groupBase, pl.groupPtr, rowPtr, col, vals, binv, mask,
                               b, x, r, r2, z, p, q, maxIter, rtol2, iters, rel, ticket));
    return EF_OK;
}

}  // namespace ef

using namespace ef;

// tile shapes of the batched PCG: (threads per CTA, lanes per block row in the products)
static const int kBatchTiles[][2] = {{128, 1}, {128, 4}, {128, 8}, {256, 4}, {256, 8}, {512, 8}, {512, 4}};
int ef_batch_num_tiles() { return (int)(sizeof(kBatchTiles) / sizeof(kBatchTiles[0])); }
void ef_batch_tile_shape(int tile, int* tpb, int* lpr) {
    *tpb = kBatchTiles[tile][0];
    *lpr = kBatchTiles[tile][1];
}

// Cluster size for problems of these sizes (nodes) (1 / 2 / 4 / 8 CTAs, ms of a solve in the best tile: 160
// cubes of 4..16 elements an edge 43.3 / 23.4 / 17.1 / 16.6, 11 of 4..9 4.4 / 2.5 / 1.5 / 0.96, 1024 of 4..16
// 83 / 81 / 84 / 90): the smallest of 1, 2, 4 and 8 CTAs whose schedule ends
// within a tenth of the earliest.  An iteration of n nodes is taken as 190 n / C cycles of FP64 work and
// 5,000 (one CTA) or 9,000 (a cluster's three barriers) of reductions, the number of iterations as n^(1/3)
// times a constant; problems go to clusters in decreasing size, nSM / C of them at a time.
int ef_batch_cluster_size(int nSM, const std::vector<int>& sizes) {
    std::vector<int> n = sizes;
    std::sort(n.begin(), n.end(), [](int a, int b) { return a > b; });
    double time[4], best = 0.0;
    for (int c = 0; c < 4; ++c) {
        const int C = 1 << c;
        std::vector<double> end(std::max(1, std::min<int>(nSM / C, (int)n.size())), 0.0);  // a min-heap
        for (int v : n) {
            std::pop_heap(end.begin(), end.end(), std::greater<double>());
            end.back() += std::cbrt((double)v) * (190.0 * v / C + (C == 1 ? 5000.0 : 9000.0));
            std::push_heap(end.begin(), end.end(), std::greater<double>());
        }
        time[c] = *std::max_element(end.begin(), end.end());
        best = c == 0 ? time[c] : std::min(best, time[c]);
    }
    for (int c = 0; c < 4; ++c)
        if (time[c] <= 1.1 * best) return 1 << c;
    return 1;
}

ef_status ef_launch_batched_pcg(int tile, const BatchPlanDev& pl, int cluster, int nSM, int nProb, const int32_t* rowPtr,
                                const int32_t* colIdx, const double* bsr, const double* binv, const uint8_t* mask,
                                const double* b, double* x, double* r, double* r2, double* z, double* p, double* q,
                                int maxIter, double rtol2, int* iters, double* rel, int* ticket, cudaStream_t s) {
    if (nProb == 0) return EF_OK;
    const int sliceGrid = std::max(1, std::min((pl.nGroups + 7) / 8, 16 * nSM));
    const bool sliced = pl.vals != nullptr;
#define EF_BT_LAUNCH(T, L, M, S)                                                                                      \
    launch_batched<T, L, M, S>(pl, cluster, nSM, nProb, rowPtr, S ? pl.col : colIdx, S ? pl.vals : bsr, binv, mask, b, x, \
                               r, r2, z, p, q, maxIter, rtol2, iters, rel, ticket, s)
#define EF_BT(T, L)                                                                                                   \
    do {                                                                                                              \
        if (sliced && pl.nGroups > 0)                                                                                 \
            batch_slice_kernel<L><<<sliceGrid, 256, 0, ef::counted(s)>>>(pl.nGroups, pl.groupRow, pl.groupEnd,        \
                                                                         pl.groupStep, rowPtr, colIdx, bsr, pl.vals,  \
                                                                         pl.col);                                     \
        EF_CUDA(cudaGetLastError());                                                                                  \
        if (cluster > 1) return sliced ? EF_BT_LAUNCH(T, L, true, true) : EF_BT_LAUNCH(T, L, true, false);            \
        return sliced ? EF_BT_LAUNCH(T, L, false, true) : EF_BT_LAUNCH(T, L, false, false);                           \
    } while (0)
    switch (tile) {
        case 0: EF_BT(128, 1);
        case 1: EF_BT(128, 4);
        case 2: EF_BT(128, 8);
        case 3: EF_BT(256, 4);
        case 4: EF_BT(256, 8);
        case 5: EF_BT(512, 8);
        case 6: EF_BT(512, 4);
        default:
            ef_set_error("batched PCG: unknown tile shape");
            return EF_ERR_ARG;
    }
#undef EF_BT
#undef EF_BT_LAUNCH
}

ef_status ef_launch_batch_norms(int nProb, const int32_t* nodePtr, const double* R, const double* F, const double* D,
                                double* out, cudaStream_t s) {
    if (nProb == 0) return EF_OK;
    batch_norms_kernel<<<nProb, 256, 0, ef::counted(s)>>>(nProb, nodePtr, R, F, D, out);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}
