// Assembly kernels: residual condensation, VIJ export, reference-order CSR scatter,
// Dirichlet rows, atomic-free 3x3-block (BSR) scatter, and deterministic norms.
//
// Reference semantics (EdelweissFE):
//   solvers/nonlinearimplicitstaticparallelmk2.pyx:186-193  P[I] += Pe, F[I] += |Pe| (element order)
//   numerics/dofmanager.py:47-82,522-557                      VIJ layout
//   numerics/csrgenerator.pyx:100-115                         data[x[k]] += V[k], increasing k
//   solvers/nonlinearimplicitstaticparallelmk2.pyx:66-109     Dirichlet rows
//
// No float atomics anywhere: every output element is owned by one thread that
// sums its contributions in a fixed (reference) order, so results are
// bit-reproducible run to run.

#include "ef_common.cuh"
#include "reduce.cuh"

#include <algorithm>

namespace ef {

// Sum over the sources of one DOF (component c of node m) in source order, and of their absolute values; the
// loads of eight sources are in flight together (an interior hex8 node has eight), where one source after the
// other cost eight trips to memory
template <bool ABS>
__device__ __forceinline__ void condense_dof(int64_t k0, int64_t k1, int c, const int64_t* __restrict__ src,
                                             const float* __restrict__ w, const double* __restrict__ Pe, double& p,
                                             double& f) {
    p = f = 0.0;
    for (int64_t k = k0; k < k1; k += 8) {
        double v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (k + j < k1) {
                v[j] = Pe[src[k + j] + c];
                if (w) v[j] *= (double)w[k + j];  // tied node: weighted share of the slave's element vectors
            }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (k + j < k1) {
                p += v[j];
                if (ABS) f += fabs(v[j]);
            }
    }
}

// P[d] = sum_k Pe[src_k + c], F likewise with |.| (F may be null); a thread per DOF
template <bool ABS>
__global__ void __launch_bounds__(kRedThreads) condense_kernel(int64_t nNodes, const int32_t* __restrict__ nodeDof,
                                                               const int64_t* __restrict__ ptr,
                                                               const int64_t* __restrict__ src,
                                                               const float* __restrict__ w, const double* __restrict__ Pe,
                                                               double* __restrict__ P, double* __restrict__ F) {
    const int64_t t = (int64_t)blockIdx.x * kRedThreads + threadIdx.x;
    if (t >= 3 * nNodes) return;
    const int64_t m = t / 3;
    const int c = (int)(t - 3 * m);
    double p, f;
    condense_dof<ABS>(ptr[m], ptr[m + 1], c, src, w, Pe, p, f);
    const int d = nodeDof[m] + c;
    P[d] = p;
    if (ABS) F[d] = f;
}

// r = b - (condensed ye) on free DOFs, 0 on masked ones (b may be null: r = condensed ye) and, with out,
// *out = sum r^2: the refinement residual from its element vectors in one pass
__global__ void __launch_bounds__(kRedThreads) condense_residual_kernel(
    int64_t nNodes, const int32_t* __restrict__ nodeDof, const int64_t* __restrict__ ptr,
    const int64_t* __restrict__ src, const float* __restrict__ w, const double* __restrict__ ye,
    const double* __restrict__ b, const uint8_t* __restrict__ mask, double* __restrict__ r, double* part,
    unsigned* ticket, double* out) {
    double v[1] = {0.0};
    for (int64_t t = (int64_t)blockIdx.x * kRedThreads + threadIdx.x; t < 3 * nNodes;
         t += (int64_t)gridDim.x * kRedThreads) {
        const int64_t m = t / 3;
        const int c = (int)(t - 3 * m);
        const int d = nodeDof[m] + c;
        double y = 0.0, f;
        if (!mask[d]) {
            condense_dof<false>(ptr[m], ptr[m + 1], c, src, w, ye, y, f);
            if (b) y = b[d] - y;
        }
        r[d] = y;
        v[0] += y * y;
    }
    if (!out) return;
    if (grid_reduce<1, 0u>(v, part, ticket)) *out = v[0];
}

// adds the condensed element vectors into V (V[d] += sum), used for body forces
__global__ void condense_add_kernel(int64_t nNodes, const int32_t* __restrict__ nodeDof,
                                    const int64_t* __restrict__ ptr, const int64_t* __restrict__ src,
                                    const float* __restrict__ w, const double* __restrict__ Pe, int64_t lo, int64_t hi,
                                    double* __restrict__ V) {
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nNodes) return;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    bool any = false;
    for (int64_t k = ptr[m]; k < ptr[m + 1]; ++k) {
        const int64_t s = src[k];
        if (s < lo || s >= hi) continue;
        const double* pe = Pe + s;
        const double wk = w ? (double)w[k] : 1.0;
        p0 += wk * pe[0];
        p1 += wk * pe[1];
        p2 += wk * pe[2];
        any = true;
    }
    if (!any) return;
    const int d = nodeDof[m];
    V[d] += p0;
    V[d + 1] += p1;
    V[d + 2] += p2;
}

// element blocks (symmetric storage, pair p(a,b), a<=b) -> reference VIJ layout in FP64
template <typename KT>
__global__ void vij_export_kernel(int nEl, int nn, int np, const KT* __restrict__ Kblk, double* __restrict__ Kvij) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)nEl * np) return;
    const int e = (int)(t / np);
    const int p = (int)(t % np);
    int a = 0, start = 0;
    while (start + (nn - a) <= p) {
        start += nn - a;
        ++a;
    }
    const int b = a + (p - start);
    const int nd = 3 * nn;
    const KT* kb = Kblk + t * 9;
    double* ke = Kvij + (int64_t)e * nd * nd;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            const double v = (double)kb[i * 3 + j];
            ke[(3 * a + i) * nd + 3 * b + j] = v;
            if (a != b) ke[(3 * b + j) * nd + 3 * a + i] = v;
        }
}

// ---- reference-order scalar scatter: data[s] = ((0 + V[k0]) + V[k1]) + ... for k0 < k1 < ... ----------
//
// Slots take 1 to 8 (and more) values; a warp whose lanes' counts differ keeps the narrow FP64 pipe (16 cycles an
// instruction) as long as its longest lane.  So the 256 slots of a CTA are dealt out by count (a
// counting sort in shared memory), the first value is taken over without an addition (0 + v is v but for -0,
// which becomes 0), and the loads of four values are in flight together.  Reading the element blocks directly
// (DIRECT) leaves out the VIJ vector: 576 values of a hex8 element written and read back, from 36 blocks of 9.
// 10,240 hex8 elements: VIJ export and scatter 23 + 48 us, now 39 us.

constexpr int kCsrThreads = 256;
constexpr int kCsrBuckets = 10;  // counts 0..8, and more

// VIJ value k from the element blocks (ND: 3 nodes of every group's element, 0: by group)
template <typename KT, int ND>
__device__ __forceinline__ double vij_value(int k, const CsrGroups& G, const KT* __restrict__ Kblk) {
    int g = 0;
    if (ND == 0)
        while (k >= G.vijEnd[g]) ++g;
    const unsigned nd = ND ? ND : G.nd[g];
    const unsigned r = (unsigned)(k - (g ? G.vijEnd[g - 1] : 0));
    const unsigned e = r / (nd * nd), ab = r - e * (nd * nd);
    const unsigned a = ab / nd, b = ab - a * nd;  // value a * nd + b is Ke[a][b]
    const unsigned na = a / 3, i = a - 3 * na, nb = b / 3, j = b - 3 * nb;
    const unsigned lo = min(na, nb), hi = max(na, nb), nn = nd / 3;
    const unsigned p = lo * nn - lo * (lo - 1) / 2 + (hi - lo);
    const int64_t blk = G.keOffset[g] + (int64_t)e * (nn * (nn + 1) / 2) + p;
    return (double)Kblk[blk * 9 + (na <= nb ? 3 * i + j : 3 * j + i)];
}

// DEAL = false: a thread takes its own slot (csr_deal)
template <typename KT, int ND, bool DIRECT, bool DEAL>
__global__ void __launch_bounds__(kCsrThreads) csr_scatter_kernel(int64_t nnz, const int64_t* __restrict__ seg,
                                                                  const int32_t* __restrict__ perm, CsrGroups G,
                                                                  const KT* __restrict__ V, double* __restrict__ data) {
    __shared__ int start[kCsrThreads];
    __shared__ int len[kCsrThreads];
    __shared__ unsigned char order[kCsrThreads];
    __shared__ int first[kCsrThreads / 32][kCsrBuckets];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int64_t s0 = (int64_t)blockIdx.x * kCsrThreads;
    const int64_t t0 = s0 + tid < nnz ? seg[s0 + tid] : 0;
    const int n0 = s0 + tid < nnz ? (int)(seg[s0 + tid + 1] - t0) : 0;
    int mine = tid;
    if constexpr (DEAL) {
        start[tid] = (int)t0;  // (fewer than 2^31 VIJ values)
        len[tid] = n0;
        const int bucket = min(n0, kCsrBuckets - 1);
        int rank = 0;
#pragma unroll
        for (int b = 0; b < kCsrBuckets; ++b) {
            const unsigned m = __ballot_sync(0xffffffffu, bucket == b);
            if (bucket == b) rank = __popc(m & ((1u << lane) - 1));
            if (lane == 0) first[w][b] = __popc(m);
        }
        __syncthreads();
        if (w == 0) {  // exclusive sums over (bucket, warp)
            int tot = 0;
            if (lane < kCsrBuckets)
                for (int q = 0; q < kCsrThreads / 32; ++q) tot += first[q][lane];
            int base = tot;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, base, o);
                if (lane >= o) base += v;
            }
            base -= tot;
            if (lane < kCsrBuckets)
                for (int q = 0; q < kCsrThreads / 32; ++q) {
                    const int c = first[q][lane];
                    first[q][lane] = base;
                    base += c;
                }
        }
        __syncthreads();
        order[first[w][bucket] + rank] = (unsigned char)tid;
        __syncthreads();
        mine = order[tid];
    }
    if (s0 + mine >= nnz) return;
    const int n = DEAL ? len[mine] : n0;
    const int32_t* pk = perm + (DEAL ? start[mine] : (int)t0);
    double acc = 0.0;
    for (int t = 0; t < n; t += 4) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (t + u < n) {
                const int k = pk[t + u];
                v[u] = DIRECT ? vij_value<KT, ND>(k, G, V) : (double)V[k];
            }
        if (t == 0) {
            acc = __double_as_longlong(v[0]) == (long long)0x8000000000000000ull ? 0.0 : v[0];
        } else {
            acc += v[0];
        }
#pragma unroll
        for (int u = 1; u < 4; ++u)
            if (t + u < n) acc += v[u];
    }
    data[s0 + mine] = acc;
}

// a warp per row
__global__ void csr_dirichlet_rows_kernel(int64_t nRows, const int64_t* __restrict__ rows,
                                          const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                                          double* __restrict__ data) {
    const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= nRows) return;
    const int64_t r = rows[t];
    for (int32_t j = indptr[r] + (threadIdx.x & 31); j < indptr[r + 1]; j += 32) data[j] = (indices[j] == r) ? 1.0 : 0.0;
}

// BSR block s = sum over its element-block contributions (element order); src encodes
// (global element-block index << 1) | transpose
template <typename KT>
__global__ void bsr_scatter_kernel(int64_t nBlocks, const int64_t* __restrict__ seg, const int64_t* __restrict__ src,
                                   const float* __restrict__ w, const KT* __restrict__ Kblk, KT* __restrict__ vals) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nBlocks) return;
    KT acc[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) acc[i] = (KT)0;
    for (int64_t t = seg[s]; t < seg[s + 1]; ++t) {
        const int64_t c = src[t];
        const KT* kb = Kblk + (c >> 1) * 9;
        const KT wt = w ? (KT)w[t] : (KT)1;  // tie weight (products of 1/2), exact in either type
        KT v[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] = wt * kb[i];
        if (c & 1) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) acc[i * 3 + j] += v[j * 3 + i];
        } else {
#pragma unroll
            for (int i = 0; i < 9; ++i) acc[i] += v[i];
        }
    }
    KT* o = vals + s * 9;
#pragma unroll
    for (int i = 0; i < 9; ++i) o[i] = acc[i];
}

// block-Jacobi setup: inverse of each diagonal 3x3 block with Dirichlet rows/columns
// replaced by the identity (inverted in FP64)
template <typename KT>
__global__ void bj_setup_kernel(int64_t nNodes, const int64_t* __restrict__ diagPos, const int32_t* __restrict__ nodeDof,
                                const uint8_t* __restrict__ mask, const KT* __restrict__ vals, KT* __restrict__ inv,
                                int* __restrict__ flags) {
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nNodes) return;
    const KT* D = vals + diagPos[m] * 9;
    const int d = nodeDof[m];
    const bool f[3] = {mask[d] != 0, mask[d + 1] != 0, mask[d + 2] != 0};
    double A[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) A[i][j] = (f[i] || f[j]) ? (i == j ? 1.0 : 0.0) : (double)D[i * 3 + j];
    const double c00 = A[1][1] * A[2][2] - A[1][2] * A[2][1];
    const double c01 = A[1][2] * A[2][0] - A[1][0] * A[2][2];
    const double c02 = A[1][0] * A[2][1] - A[1][1] * A[2][0];
    const double det = A[0][0] * c00 + A[0][1] * c01 + A[0][2] * c02;
    if (!(fabs(det) > 0.0)) {
        atomicOr(flags, EF_FLAG_NAN);
    }
    const double id = 1.0 / det;
    KT* o = inv + m * 9;
    o[0] = (KT)(c00 * id);
    o[3] = (KT)(c01 * id);
    o[6] = (KT)(c02 * id);
    o[1] = (KT)((A[0][2] * A[2][1] - A[0][1] * A[2][2]) * id);
    o[4] = (KT)((A[0][0] * A[2][2] - A[0][2] * A[2][0]) * id);
    o[7] = (KT)((A[0][1] * A[2][0] - A[0][0] * A[2][1]) * id);
    o[2] = (KT)((A[0][1] * A[1][2] - A[0][2] * A[1][1]) * id);
    o[5] = (KT)((A[0][2] * A[1][0] - A[0][0] * A[1][2]) * id);
    o[8] = (KT)((A[0][0] * A[1][1] - A[0][1] * A[1][0]) * id);
}

// out = {max |R|, sum |F|, max |D|} (each may be null -> 0)
__global__ void __launch_bounds__(kRedThreads) norms_kernel(int64_t n, const double* __restrict__ R,
                                                            const double* __restrict__ F, const double* __restrict__ D,
                                                            double* part, unsigned* ticket, double* out) {
    double v[3] = {0.0, 0.0, 0.0};
    for (int64_t i = (int64_t)blockIdx.x * kRedThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kRedThreads) {
        if (R) v[0] = fmax(v[0], fabs(R[i]));
        if (F) v[1] += fabs(F[i]);
        if (D) v[2] = fmax(v[2], fabs(D[i]));
    }
    if (grid_reduce<3, 5u>(v, part, ticket)) {
        out[0] = v[0];
        out[1] = v[1];
        out[2] = v[2];
    }
}

// R = P + PExt with the Dirichlet rows set to 0 (dir[i] != 0), the norms of the convergence check (max |R|,
// sum |F|, max |ddU|; solvers/nonlinearimplicitstatic.py:418-436, :625-725) and, by the thread that gets
// them, the reference's test for the displacement field (:656-682, computeSpatialAveragedFluxes :771-792):
// out = {converged, nGrew, fluxResidual, fieldCorrection, spatialAveragedFlux}
__global__ void __launch_bounds__(kRedThreads) newton_check_kernel(int64_t n, const double* __restrict__ P,
                                                                   const double* __restrict__ PExt,
                                                                   const uint8_t* __restrict__ dir,
                                                                   const double* __restrict__ F,
                                                                   const double* __restrict__ D, double* __restrict__ R,
                                                                   double* part, unsigned* ticket, NewtonTest q,
                                                                   double* out) {
    double v[3] = {0.0, 0.0, 0.0};
    for (int64_t i = (int64_t)blockIdx.x * kRedThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kRedThreads) {
        const double r = dir[i] ? 0.0 : (PExt ? P[i] + PExt[i] : P[i]);
        R[i] = r;
        v[0] = fmax(v[0], fabs(r));
        v[1] += fabs(F[i]);
        if (D) v[2] = fmax(v[2], fabs(D[i]));
    }
    if (!grid_reduce<3, 5u>(v, part, ticket)) return;
    const double avg = fmax(1e-10, v[1] / q.nAccFluxes);
    const double tol = q.iteration < 15 ? q.fluxTol : q.fluxTolAlt;
    const double corr = D ? v[2] : 0.0;
    const bool convCorr = corr < q.corrTol;
    const bool convFlux = v[0] <= fmax(tol * avg, q.fluxFloor);
    out[0] = (convCorr && convFlux) ? 1.0 : 0.0;
    out[1] = q.nGrew + (v[0] > q.prevResidual ? 1.0 : 0.0);
    out[2] = v[0];
    out[3] = corr;
    out[4] = avg;
}

// R = P + PExt, then R[dofs[k]] = values[k] (the prescribed increments of the first iteration)
__global__ void newton_first_residual_kernel(int64_t n, const double* __restrict__ P, const double* __restrict__ PExt,
                                             double* __restrict__ R) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) R[i] = PExt ? P[i] + PExt[i] : P[i];
}
__global__ void scatter_values_kernel(int64_t n, const int64_t* __restrict__ dofs, const double* __restrict__ v,
                                      double* __restrict__ R) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) R[dofs[k]] = v[k];
}

// x[slave] = (x[a] + x[b]) / 2 per component (tied nodes)
__global__ void tie_fill_kernel(int64_t n, const int32_t* __restrict__ slave, const int32_t* __restrict__ ma,
                                const int32_t* __restrict__ mb, double* __restrict__ x) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * n) return;
    const int64_t k = t / 3;
    const int c = (int)(t % 3);
    x[3 * (int64_t)slave[k] + c] = 0.5 * (x[3 * (int64_t)ma[k] + c] + x[3 * (int64_t)mb[k] + c]);
}

}  // namespace ef

using namespace ef;

static inline int nblk(int64_t n, int t) { return (int)((n + t - 1) / t); }

ef_status ef_launch_condense(int64_t nNodes, const int32_t* nodeDof, const int64_t* ptr, const int64_t* src,
                             const float* w, const double* Pe, double* P, double* F, cudaStream_t s) {
    if (nNodes == 0) return EF_OK;
    if (F)
        condense_kernel<true><<<nblk(3 * nNodes, kRedThreads), kRedThreads, 0, ef::counted(s)>>>(nNodes, nodeDof, ptr, src,
                                                                                                w, Pe, P, F);
    else
        condense_kernel<false><<<nblk(3 * nNodes, kRedThreads), kRedThreads, 0, ef::counted(s)>>>(nNodes, nodeDof, ptr, src,
                                                                                                 w, Pe, P, F);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

// nPart: the number of CTAs' results `part` has room for
ef_status ef_launch_condense_residual(int64_t nNodes, const int32_t* nodeDof, const int64_t* ptr, const int64_t* src,
                                      const float* w, const double* ye, const double* b, const uint8_t* mask, double* r,
                                      double* part, int nPart, unsigned* ticket, double* out, cudaStream_t s) {
    if (nNodes == 0) return EF_OK;
    const int grid = std::min(nblk(3 * nNodes, kRedThreads), nPart);
    condense_residual_kernel<<<grid, kRedThreads, 0, ef::counted(s)>>>(nNodes, nodeDof, ptr, src, w, ye, b, mask, r, part,
                                                                      ticket, out);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_condense_add(int64_t nNodes, const int32_t* nodeDof, const int64_t* ptr, const int64_t* src,
                                 const float* w, const double* Pe, int64_t lo, int64_t hi, double* V, cudaStream_t s) {
    if (nNodes == 0) return EF_OK;
    condense_add_kernel<<<nblk(nNodes, 256), 256, 0, ef::counted(s)>>>(nNodes, nodeDof, ptr, src, w, Pe, lo, hi, V);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_vij_export(int nEl, int nn, int np, const void* Kblk, int kDouble, double* Kvij, cudaStream_t s) {
    const int64_t n = (int64_t)nEl * np;
    if (n == 0) return EF_OK;
    if (kDouble)
        vij_export_kernel<double><<<nblk(n, 256), 256, 0, ef::counted(s)>>>(nEl, nn, np, (const double*)Kblk, Kvij);
    else
        vij_export_kernel<float><<<nblk(n, 256), 256, 0, ef::counted(s)>>>(nEl, nn, np, (const float*)Kblk, Kvij);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

// Dealing a CTA's slots out by count pays where they have many values: of a VIJ vector us without and with at
// 2.3 values a slot (10,240 hex8 elements) 58.8 and 51.2, at 1.95 (125 hex8) 16.8 and 15.6, at 1.64 (2,880 hex20) 77.0 and
// 88.2, at 1.58 (546 hex20) 24.2 and 26.5
static bool csr_deal(int64_t nVIJ, int64_t nnz) { return 10 * nVIJ > 17 * nnz; }

ef_status ef_launch_csr_scatter(int64_t nVIJ, int64_t nnz, const int64_t* seg, const int32_t* perm, const double* V,
                                double* data, cudaStream_t s) {
    if (nnz == 0) return EF_OK;
    auto k = csr_deal(nVIJ, nnz) ? csr_scatter_kernel<double, 0, false, true> : csr_scatter_kernel<double, 0, false, false>;
    k<<<nblk(nnz, kCsrThreads), kCsrThreads, 0, ef::counted(s)>>>(nnz, seg, perm, CsrGroups{}, V, data);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_csr_from_blocks(int64_t nnz, const int64_t* seg, const int32_t* perm, const CsrGroups& G,
                                    const void* Kblk, int kDouble, double* data, cudaStream_t s) {
    if (nnz == 0) return EF_OK;
    const int nd = G.n == 1 ? G.nd[0] : 0;
#define EF_CSR(T_, N_)                                                                                            \
    csr_scatter_kernel<T_, N_, true, true><<<nblk(nnz, kCsrThreads), kCsrThreads, 0, ef::counted(s)>>>(nnz, seg, perm, G, \
                                                                                               (const T_*)Kblk, data)
    if (kDouble) {
        if (nd == 24)
            EF_CSR(double, 24);
        else if (nd == 60)
            EF_CSR(double, 60);
        else
            EF_CSR(double, 0);
    } else {
        if (nd == 24)
            EF_CSR(float, 24);
        else if (nd == 60)
            EF_CSR(float, 60);
        else
            EF_CSR(float, 0);
    }
#undef EF_CSR
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_csr_dirichlet_rows(int64_t nRows, const int64_t* rows, const int32_t* indptr,
                                       const int32_t* indices, double* data, cudaStream_t s) {
    if (nRows == 0) return EF_OK;
    csr_dirichlet_rows_kernel<<<nblk(32 * nRows, 256), 256, 0, ef::counted(s)>>>(nRows, rows, indptr, indices, data);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_bsr_scatter(int64_t nBlocks, const int64_t* seg, const int64_t* src, const float* w,
                                const void* Kblk, int kDouble, void* vals, cudaStream_t s) {
    if (nBlocks == 0) return EF_OK;
    if (kDouble)
        bsr_scatter_kernel<double><<<nblk(nBlocks, 256), 256, 0, ef::counted(s)>>>(nBlocks, seg, src, w,
                                                                                   (const double*)Kblk, (double*)vals);
    else
        bsr_scatter_kernel<float><<<nblk(nBlocks, 256), 256, 0, ef::counted(s)>>>(nBlocks, seg, src, w,
                                                                                  (const float*)Kblk, (float*)vals);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_bj_setup(int64_t nNodes, const int64_t* diagPos, const int32_t* nodeDof, const uint8_t* mask,
                             const void* vals, int kDouble, void* inv, int* flags, cudaStream_t s) {
    if (nNodes == 0) return EF_OK;
    if (kDouble)
        bj_setup_kernel<double><<<nblk(nNodes, 256), 256, 0, ef::counted(s)>>>(nNodes, diagPos, nodeDof, mask,
                                                                   (const double*)vals, (double*)inv, flags);
    else
        bj_setup_kernel<float><<<nblk(nNodes, 256), 256, 0, ef::counted(s)>>>(nNodes, diagPos, nodeDof, mask, (const float*)vals,
                                                                  (float*)inv, flags);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_norms(int64_t n, const double* R, const double* F, const double* D, double* part, int nPart,
                          unsigned* ticket, double* out, cudaStream_t s) {
    norms_kernel<<<reduce_grid(n, nPart), kRedThreads, 0, ef::counted(s)>>>(n, R, F, D, part, ticket, out);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_newton_check(int64_t n, const double* P, const double* PExt, const uint8_t* dir, const double* F,
                                 const double* D, double* R, double* part, int nPart, unsigned* ticket,
                                 const NewtonTest& q, double* out, cudaStream_t s) {
    newton_check_kernel<<<reduce_grid(n, nPart), kRedThreads, 0, ef::counted(s)>>>(n, P, PExt, dir, F, D, R, part, ticket,
                                                                                 q, out);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_newton_first(int64_t n, const double* P, const double* PExt, int64_t nDir, const int64_t* dofs,
                                 const double* values, double* R, cudaStream_t s) {
    if (n > 0) newton_first_residual_kernel<<<nblk(n, 256), 256, 0, ef::counted(s)>>>(n, P, PExt, R);
    if (nDir > 0) scatter_values_kernel<<<nblk(nDir, 256), 256, 0, ef::counted(s)>>>(nDir, dofs, values, R);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_tie_fill(int64_t n, const int32_t* slave, const int32_t* ma, const int32_t* mb, double* x,
                             cudaStream_t s) {
    if (n == 0) return EF_OK;
    tie_fill_kernel<<<nblk(3 * n, 256), 256, 0, ef::counted(s)>>>(n, slave, ma, mb, x);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

// element results (utils/elementresultcollector.pyx:38-120): one thread per requested
// (element, quadrature point) p = i * nQ + j, table[p * count + k] = state var first + k of point
// elements[i] * nQP + qps[j]; the SoA state makes the reads of a warp contiguous for consecutive
// points, the strided writes of a thread merge in L2
__global__ void results_gather_kernel(int64_t nPts, int nQ, int nQP, int64_t nq, int first, int count,
                                      const int32_t* __restrict__ elements, const int32_t* __restrict__ qps,
                                      const double* __restrict__ state, double* __restrict__ table) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nPts) return;
    const int64_t i = p / nQ;
    const int j = (int)(p - i * nQ);
    const double* src = state + (int64_t)first * nq + (int64_t)elements[i] * nQP + qps[j];
    double* out = table + p * count;
    for (int k = 0; k < count; ++k) out[k] = src[(int64_t)k * nq];
}

ef_status ef_launch_results_gather(int64_t nPts, int nQ, int nQP, int64_t nq, int first, int count,
                                   const int32_t* elements, const int32_t* qps, const double* state, double* table,
                                   cudaStream_t s) {
    if (nPts == 0) return EF_OK;
    results_gather_kernel<<<nblk(nPts, 256), 256, 0, ef::counted(s)>>>(nPts, nQ, nQP, nq, first, count, elements, qps,
                                                                        state, table);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}
