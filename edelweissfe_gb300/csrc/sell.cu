// Sliced-ELL copies of the fine 3x3-block system and the fine-level kernels that stream them.
//
// The fine system's block rows are grouped into slices of 32; a slice is as wide as its longest
// row (shorter rows are padded with zero blocks whose column is the row itself) and its entries
// are stored column-major: entry j of the slice's row i sits at slot e0 + 32 j + i.  A warp takes
// one slice, a lane one row, so at every step j the warp reads 32 consecutive column indices and
// 32 consecutive blocks -- fully coalesced, with no row-pointer load ahead of them -- and, on a
// mesh numbered along a grid line, gathers x from 32 consecutive nodes.  An optional row
// permutation (rows sorted by length within windows) keeps the padding small on meshes whose row
// lengths vary; on the structured hex8 box it is the identity and costs one coalesced load.
//
// Two value copies, refreshed from the FP32 block values after every assembly:
//  * FP32, nine planes per slot column: value k of slot t at 9 (t - i) + 32 k + i (i = t mod 32),
//    for the FGMRES product y = K z;
//  * BF16 split: one 16-byte word with values 0..7 per slot and value 8 in a second array, for the
//    multigrid's fine smoothing sweeps and residuals (a preconditioner only).
// Summation per row runs over the row's blocks in column order with one accumulator per output
// component: deterministic, not the same rounding as the CSR kernels.

#include <cuda_bf16.h>
#include <stdint.h>

#include <type_traits>

#include "amg_sa_body.h"
#include "early.cuh"
#include "ef_common.cuh"

namespace ef {

constexpr int kSellThreads = 128;  // four warps per CTA
// Split slices: S warps per slice, each taking a contiguous share of the slice's entries, four
// warps per CTA up to S = 4 and S warps (one slice) above

// FP32 planes of K; the BF16 copy holds K, or with binv the blocks of K (M D^-1) (the block
// inverse of the slot's column node with the rows of masked DOFs zeroed), for the residual of the
// block-Jacobi sweep from zero: r - K (w M D^-1 r) = r - w (K M D^-1) r
// diaN > 0 (diagonal form): the FP32 planes hold only the diagonals from the middle one on (see
// sell_spmv3_dia_kernel)
__global__ void sell_refresh_kernel(int64_t nE, const int32_t* __restrict__ src, const float* __restrict__ bsr,
                                    float* __restrict__ v9, uint4* __restrict__ v8, __nv_bfloat16* __restrict__ v1,
                                    const int32_t* __restrict__ col, const float* __restrict__ binv,
                                    const uint8_t* __restrict__ mask, int diaN) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nE) return;
    const int64_t b = src[t];
    float a[9];
    if (b >= 0) {
#pragma unroll
        for (int k = 0; k < 9; ++k) a[k] = bsr[b * 9 + k];
    } else {
#pragma unroll
        for (int k = 0; k < 9; ++k) a[k] = 0.f;
    }
    const int64_t i = t & 31;
    if (diaN == 0) {
        float* d = v9 + 9 * (t - i) + i;
#pragma unroll
        for (int k = 0; k < 9; ++k) d[32 * k] = a[k];
    } else {
        const int sl = (int)(t >> 5) / diaN, j = (int)(t >> 5) - sl * diaN, h = diaN / 2;
        if (j >= h) {
            float* d = v9 + (int64_t)288 * ((int64_t)sl * (h + 1) + j - h) + i;
#pragma unroll
            for (int k = 0; k < 9; ++k) d[32 * k] = a[k];
        }
    }
    if (v8 && binv) {
        const int64_t c = col[t];
        const float* D = binv + 9 * c;
        float sa[9];
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                float z = 0.f;
#pragma unroll
                for (int u = 0; u < 3; ++u) z += mask[3 * c + u] ? 0.f : a[3 * p + u] * D[3 * u + q];
                sa[3 * p + q] = z;
            }
#pragma unroll
        for (int k = 0; k < 9; ++k) a[k] = sa[k];
    }
    if (v8) {
        __nv_bfloat162 h[4] = {__floats2bfloat162_rn(a[0], a[1]), __floats2bfloat162_rn(a[2], a[3]),
                               __floats2bfloat162_rn(a[4], a[5]), __floats2bfloat162_rn(a[6], a[7])};
        v8[t] = *reinterpret_cast<const uint4*>(h);
        v1[t] = __float2bfloat16_rn(a[8]);
    }
}

// Diagonal form of the slices (structured meshes): every block column is its row plus one of a few
// node offsets, slot column j of every slice holding offset dia[j] (zero blocks where the row has
// no such neighbour), so the column is computed, not loaded, and the x gathers of a warp are 32
// consecutive nodes.  The rows are in natural order; a column outside the nodes is clamped (its
// block is zero).
__device__ __forceinline__ int dia_column(int row, int d, int nN) { return min(max(row + d, 0), nN - 1); }

// The slice and entry range of this warp: warp h of the S warps of a slice takes entries
// [j0, j1) = [ceil(h w / S), ceil((h + 1) w / S)) of its width w.  Returns false past the last
// slice.
struct SellPart {
    int sl, h, lane, j0, j1;
    int64_t e0;
};
constexpr int sell_split_threads(int S) { return S <= 4 ? kSellThreads : 32 * S; }
template <int S>
__device__ __forceinline__ bool sell_part(int nSlices, const int64_t* __restrict__ off, SellPart& p) {
    constexpr int spc = sell_split_threads(S) / (32 * S);
    p.lane = threadIdx.x & 31;
    const int wi = threadIdx.x >> 5;
    p.sl = blockIdx.x * spc + wi / S;
    p.h = wi % S;
    if (p.sl >= nSlices) return false;
    p.e0 = off[p.sl];
    const int w = (int)((off[p.sl + 1] - p.e0) >> 5);
    p.j0 = (p.h * w + S - 1) / S;
    p.j1 = ((p.h + 1) * w + S - 1) / S;
    return true;
}

// the partial sums of warps 1..S-1 of a slice go through shared memory to warp 0, which adds them
// after its own in warp order (a fixed order: deterministic)
template <int S>
__device__ __forceinline__ bool sell_combine(const SellPart& p, bool active, float& y0, float& y1, float& y2) {
    if constexpr (S == 1) {
        return active;
    } else {
        constexpr int spc = sell_split_threads(S) / (32 * S);
        __shared__ float part[spc][S - 1][3][32];
        const int ls = (threadIdx.x >> 5) / S;
        if (active && p.h > 0) {
            part[ls][p.h - 1][0][p.lane] = y0;
            part[ls][p.h - 1][1][p.lane] = y1;
            part[ls][p.h - 1][2][p.lane] = y2;
        }
        __syncthreads();
        if (!active || p.h != 0) return false;
#pragma unroll
        for (int q = 0; q < S - 1; ++q) {
            y0 += part[ls][q][0][p.lane];
            y1 += part[ls][q][1][p.lane];
            y2 += part[ls][q][2][p.lane];
        }
        return true;
    }
}

// the end of a product's row m: the scale, the copy of x, the mask and, with binv, D^-1
template <bool COPY>
__device__ __forceinline__ void sell_product_end(int m, const float* __restrict__ x, const uint8_t* __restrict__ mask,
                                                 float* __restrict__ y, float* __restrict__ xcopy,
                                                 const float* __restrict__ scale, const float* __restrict__ binv, float y0,
                                                 float y1, float y2) {
    const int d = 3 * m;
    if (scale) {
        const float sc = *scale;
        y0 *= sc;
        y1 *= sc;
        y2 *= sc;
        if (COPY) {
            xcopy[d + 0] = sc * x[d + 0];
            xcopy[d + 1] = sc * x[d + 1];
            xcopy[d + 2] = sc * x[d + 2];
        }
    } else if (COPY) {
        xcopy[d + 0] = x[d + 0];
        xcopy[d + 1] = x[d + 1];
        xcopy[d + 2] = x[d + 2];
    }
    y0 = mask[d + 0] ? 0.f : y0;
    y1 = mask[d + 1] ? 0.f : y1;
    y2 = mask[d + 2] ? 0.f : y2;
    if (binv) {  // y = D^-1 (K x) with the row's block inverse (the power iteration on D^-1 K)
        const float* B = binv + 9 * (int64_t)m;
        const float z0 = B[0] * y0 + B[1] * y1 + B[2] * y2;
        const float z1 = B[3] * y0 + B[4] * y1 + B[5] * y2;
        const float z2 = B[6] * y0 + B[7] * y1 + B[8] * y2;
        y0 = mask[d + 0] ? 0.f : z0;
        y1 = mask[d + 1] ? 0.f : z1;
        y2 = mask[d + 2] ? 0.f : z2;
    }
    y[d + 0] = y0;
    y[d + 1] = y1;
    y[d + 2] = y2;
}

__device__ __forceinline__ void sell_block_add(const float (&a)[9], const float (&xv)[3], float& y0, float& y1, float& y2) {
    y0 += a[0] * xv[0] + a[1] * xv[1] + a[2] * xv[2];
    y1 += a[3] * xv[0] + a[4] * xv[1] + a[5] * xv[2];
    y2 += a[6] * xv[0] + a[7] * xv[1] + a[8] * xv[2];
}

// The slot columns of a warp are taken two at a time, all their loads first (the second clamped to the last one and
// left out of the sum where the count is odd): an unrolled loop falls back to one column after the other for its
// remainder, which with a slice split over several warps is most of it.  More than two take registers from
// the warps that hide the loads.  us before, with two and with four columns: the product at 169,781 nodes 32.8, 26.8 and
// 26.8, of 81-block rows at 26,745 nodes 20.7, 18.5 and 19.8; the preconditioner (its residual) 82.4, 78.2 and 79.4 at
// 169,781 nodes, 31.6, 30.0 and 33.8 at 18,081.  What bounds them then is the latency of the gathers: the 82 MB that a
// residual of 169,781 nodes reads take 14.5 us (5.7 TB/s) by themselves; a ring of slices in shared memory kept ahead
// by bulk copies was slower (preconditioner 100 us), as fewer warps gather.
constexpr int kSellBatch = 2;

// The first two columns are loaded ahead of the wait for the kernel before (early.cuh), which gives a product of
// 785 nodes of quadratic elements 8.2 -> 7.4 us, of 7,412 nodes 10.4 -> 9.7, of 19,456 nodes of a tied mesh 13.8 -> 12.6.  The
// same in the diagonal form gains nothing, and in the residual and the post-smoothing it costs the large
// systems more (cycle at 169,781 nodes 71.2 -> 74.3 and 72.4 us) than it gives the small.
// y = sc K x on the free DOFs (0 on masked rows); COPY: xcopy = sc x as well; sc = *scale (1 without
// one: the FGMRES basis vector x then carries its normalisation factor); S warps per slice
template <bool COPY, int S>
__global__ void __launch_bounds__(sell_split_threads(S)) sell_spmv3_kernel(
    int nN, int nSlices, const int64_t* __restrict__ off, const int32_t* __restrict__ perm,
    const int32_t* __restrict__ col, const float* __restrict__ v9, const float* __restrict__ x,
    const uint8_t* __restrict__ mask, float* __restrict__ y, float* __restrict__ xcopy,
    const float* __restrict__ scale, const float* __restrict__ binv) {
    SellPart p;
    const bool active = sell_part<S>(nSlices, off, p);
    float y0 = 0.f, y1 = 0.f, y2 = 0.f;
    float a[kSellBatch][9];
    int c3[kSellBatch];
    const int32_t* cs = col + p.e0 + p.lane;
    const float* vs = v9 + 9 * p.e0 + p.lane;
    auto load = [&](int j, auto ahead) {
#pragma unroll
        for (int u = 0; u < kSellBatch; ++u) {
            const int k = min(j + u, p.j1 - 1);
            c3[u] = 3 * (ahead() ? early_cs(cs + 32 * k) : __ldcs(cs + 32 * k));
#pragma unroll
            for (int i = 0; i < 9; ++i)
                a[u][i] = ahead() ? early_cs(vs + 288 * k + 32 * i) : __ldcs(vs + 288 * k + 32 * i);
        }
    };
    const bool some = active && p.j0 < p.j1;
    if (some) load(p.j0, std::true_type());
    ef::dep_entry();
    if (some)
        for (int j = p.j0;;) {
            float xv[kSellBatch][3];
#pragma unroll
            for (int u = 0; u < kSellBatch; ++u)
#pragma unroll
                for (int i = 0; i < 3; ++i) xv[u][i] = x[c3[u] + i];
#pragma unroll
            for (int u = 0; u < kSellBatch; ++u)
                if (j + u < p.j1) sell_block_add(a[u], xv[u], y0, y1, y2);
            j += kSellBatch;
            if (j >= p.j1) break;
            load(j, std::false_type());
        }
    if (!sell_combine<S>(p, active, y0, y1, y2)) return;
    const int r = p.sl * 32 + p.lane;
    if (r >= nN) return;
    sell_product_end<COPY>(perm ? perm[r] : r, x, mask, y, xcopy, scale, binv, y0, y1, y2);
}

// The product in the diagonal form from half the matrix.  K is symmetric to the bit (both blocks of a pair of
// nodes sum the same element blocks in the same order; where ties or collapsed elements give a pair several blocks of one
// element, to the rounding of that sum), so only the diagonals j >= diaN / 2 are stored: the block of
// diagonal -d in row r is the transpose of the one of diagonal d in row r - d, which the rows a little
// further up have just brought into L1 and L2.  The order of a row's sums is the full form's: the same bits.
// Half the values leave HBM (86 MB of them at 169,781 nodes, full form 165 MB) and L2 the rest.  STREAM (above 60,000 nodes, where
// an iteration's matrices no longer fit into L2 and would evict the basis): the blocks are marked for early eviction
// and taken two at a time; below, one after the other from cached lines (11,849 nodes: 6.7 us against 7.5 two at a
// time, 38,125 nodes: 9.1 against 10.4).  us of a product, full form and now: 11,849 nodes 8.3 -> 6.7, 38,125 nodes
// 12.7 -> 9.1, 88,209 nodes 23.0 -> 16.7, 169,781 nodes 35.8 -> 26.8.
template <bool COPY, int S, bool STREAM>
__global__ void __launch_bounds__(sell_split_threads(S)) sell_spmv3_dia_kernel(
    int nN, int nSlices, int diaN, const float* __restrict__ v9, const float* __restrict__ x,
    const uint8_t* __restrict__ mask, float* __restrict__ y, float* __restrict__ xcopy,
    const float* __restrict__ scale, const int32_t* __restrict__ dia, const float* __restrict__ binv) {
    ef::dep_entry();
    constexpr int spc = sell_split_threads(S) / (32 * S);
    SellPart p;
    p.lane = threadIdx.x & 31;
    const int wi = threadIdx.x >> 5;
    p.sl = blockIdx.x * spc + wi / S;
    p.h = wi % S;
    const bool active = p.sl < nSlices;
    p.j0 = (p.h * diaN + S - 1) / S;
    p.j1 = ((p.h + 1) * diaN + S - 1) / S;
    const int row = p.sl * 32 + p.lane;
    const int mid = diaN / 2, stored = mid + 1;  // diagonals of a slice
    auto ld = [](const float* a) { return STREAM ? __ldcs(a) : *a; };
    float y0 = 0.f, y1 = 0.f, y2 = 0.f;
    if (active) {
        if constexpr (STREAM) {
            for (int j = p.j0; j < p.j1; j += kSellBatch) {
                float a[kSellBatch][9], xv[kSellBatch][3];
                bool in[kSellBatch];
#pragma unroll
                for (int u = 0; u < kSellBatch; ++u) {
                    const int k = min(j + u, p.j1 - 1);
                    const int c = row + __ldg(dia + k), cc = min(max(c, 0), nN - 1);
                    // below the middle: transposed from row c (a block of rows before 0: none)
                    const bool below = k < mid;
                    const int rr = below ? cc : row;
                    const float* vv = v9 + (int64_t)288 * ((int64_t)(rr >> 5) * stored + (below ? mid - k : k - mid)) + (rr & 31);
                    in[u] = j + u < p.j1 && (!below || c == cc);
                    a[u][0] = ld(vv);
                    a[u][1] = ld(vv + (below ? 96 : 32));
                    a[u][2] = ld(vv + (below ? 192 : 64));
                    a[u][3] = ld(vv + (below ? 32 : 96));
                    a[u][4] = ld(vv + 128);
                    a[u][5] = ld(vv + (below ? 224 : 160));
                    a[u][6] = ld(vv + (below ? 64 : 192));
                    a[u][7] = ld(vv + (below ? 160 : 224));
                    a[u][8] = ld(vv + 256);
#pragma unroll
                    for (int i = 0; i < 3; ++i) xv[u][i] = x[3 * cc + i];
                }
#pragma unroll
                for (int u = 0; u < kSellBatch; ++u)
                    if (in[u]) sell_block_add(a[u], xv[u], y0, y1, y2);
            }
        } else {
            const int jm = min(p.j1, max(p.j0, mid));
#pragma unroll 3
            for (int j = p.j0; j < jm; ++j) {  // below the middle: transposed from row r + dia[j] (a block of rows before 0: none)
                const int c = row + __ldg(dia + j);
                const int cc = min(max(c, 0), nN - 1);
                const float* vv = v9 + (int64_t)288 * ((int64_t)(cc >> 5) * stored + (mid - j)) + (cc & 31);
                const float a0 = ld(vv), a1 = ld(vv + 32), a2 = ld(vv + 64), a3 = ld(vv + 96), a4 = ld(vv + 128);
                const float a5 = ld(vv + 160), a6 = ld(vv + 192), a7 = ld(vv + 224), a8 = ld(vv + 256);
                const float x0 = x[3 * cc], x1 = x[3 * cc + 1], x2 = x[3 * cc + 2];
                if (c == cc) {
                    y0 += a0 * x0 + a3 * x1 + a6 * x2;
                    y1 += a1 * x0 + a4 * x1 + a7 * x2;
                    y2 += a2 * x0 + a5 * x1 + a8 * x2;
                }
            }
            const float* vs = v9 + (int64_t)288 * ((int64_t)p.sl * stored - mid) + p.lane;
#pragma unroll 3
            for (int j = max(p.j0, mid); j < p.j1; ++j) {
                const int c3 = 3 * dia_column(row, __ldg(dia + j), nN);
                const float* vv = vs + 288 * j;
                const float a0 = ld(vv), a1 = ld(vv + 32), a2 = ld(vv + 64), a3 = ld(vv + 96), a4 = ld(vv + 128);
                const float a5 = ld(vv + 160), a6 = ld(vv + 192), a7 = ld(vv + 224), a8 = ld(vv + 256);
                const float x0 = x[c3], x1 = x[c3 + 1], x2 = x[c3 + 2];
                y0 += a0 * x0 + a1 * x1 + a2 * x2;
                y1 += a3 * x0 + a4 * x1 + a5 * x2;
                y2 += a6 * x0 + a7 * x1 + a8 * x2;
            }
        }
    }
    if (!sell_combine<S>(p, active, y0, y1, y2)) return;
    if (row >= nN) return;
    sell_product_end<COPY>(row, x, mask, y, xcopy, scale, binv, y0, y1, y2);
}

// y += one BF16 block times x (values 0..7 in q, value 8 in b8)
__device__ __forceinline__ void sell_bf16_step(const uint4& q, __nv_bfloat16 b8, float x0, float x1, float x2, float& y0,
                                               float& y1, float& y2) {
    const float w8 = __bfloat162float(b8);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
    const float2 a01 = __bfloat1622float2(h[0]), a23 = __bfloat1622float2(h[1]);
    const float2 a45 = __bfloat1622float2(h[2]), a67 = __bfloat1622float2(h[3]);
    y0 += a01.x * x0 + a01.y * x1 + a23.x * x2;
    y1 += a23.y * x0 + a45.x * x1 + a45.y * x2;
    y2 += a67.x * x0 + a67.y * x1 + w8 * x2;
}

// the end of a row m of sell_level3_bf16_kernel: K x = (y0, y1, y2)
__device__ __forceinline__ void sell_level3_end(int m, const float* __restrict__ x, const float* __restrict__ r,
                                                const uint8_t* __restrict__ mask, float* __restrict__ t,
                                                const float* __restrict__ binv, float omega, float ys, float y0, float y1,
                                                float y2) {
    const int d = 3 * m;
    const bool k0 = mask[d], k1 = mask[d + 1], k2 = mask[d + 2];
    const float t0 = k0 ? 0.f : r[d] - ys * y0, t1 = k1 ? 0.f : r[d + 1] - ys * y1,
                t2 = k2 ? 0.f : r[d + 2] - ys * y2;
    if (!binv) {
        t[d] = t0;
        t[d + 1] = t1;
        t[d + 2] = t2;
        return;
    }
    const float* B = binv + 9 * (int64_t)m;
    const float z0 = B[0] * t0 + B[1] * t1 + B[2] * t2;
    const float z1 = B[3] * t0 + B[4] * t1 + B[5] * t2;
    const float z2 = B[6] * t0 + B[7] * t1 + B[8] * t2;
    const float x0 = x[d], x1 = x[d + 1], x2 = x[d + 2];
    t[d] = k0 ? x0 : x0 + omega * z0;
    t[d + 1] = k1 ? x1 : x1 + omega * z1;
    t[d + 2] = k2 ? x2 : x2 + omega * z2;
}

// t = r - ys K x on the fine level (0 on masked rows), or with binv a damped block-Jacobi sweep
// t = x + omega D^-1 (r - K x) (masked DOFs keep x), from the BF16 split copy; S warps per slice
template <int S, bool DIA>
__global__ void __launch_bounds__(sell_split_threads(S)) sell_level3_bf16_kernel(
    int nN, int nSlices, const int64_t* __restrict__ off, const int32_t* __restrict__ perm,
    const int32_t* __restrict__ col, const uint4* __restrict__ v8, const __nv_bfloat16* __restrict__ v1,
    const float* __restrict__ x, const float* __restrict__ r, const uint8_t* __restrict__ mask, float* __restrict__ t,
    const float* __restrict__ binv, float omega, float ys, const int32_t* __restrict__ dia) {
    ef::dep_entry();
    SellPart p;
    const bool active = sell_part<S>(nSlices, off, p);
    float y0 = 0.f, y1 = 0.f, y2 = 0.f;
    if (active) {
        const int32_t* cs = col + p.e0 + p.lane;
        const uint4* qs = v8 + p.e0 + p.lane;
        const __nv_bfloat16* ws = v1 + p.e0 + p.lane;
        const int row = p.sl * 32 + p.lane;
        for (int j = p.j0; j < p.j1; j += kSellBatch) {
            uint4 q[kSellBatch];
            __nv_bfloat16 b8[kSellBatch];
            float xv[kSellBatch][3];
#pragma unroll
            for (int u = 0; u < kSellBatch; ++u) {
                const int k = min(j + u, p.j1 - 1);
                const int c3 = 3 * (DIA ? dia_column(row, __ldg(dia + k), nN) : __ldcs(cs + 32 * k));
                q[u] = __ldcs(qs + 32 * k);
                b8[u] = ws[32 * k];
                xv[u][0] = x[c3];
                xv[u][1] = x[c3 + 1];
                xv[u][2] = x[c3 + 2];
            }
#pragma unroll
            for (int u = 0; u < kSellBatch; ++u)
                if (j + u < p.j1) sell_bf16_step(q[u], b8[u], xv[u][0], xv[u][1], xv[u][2], y0, y1, y2);
        }
    }
    if (!sell_combine<S>(p, active, y0, y1, y2)) return;
    const int rr = p.sl * 32 + p.lane;
    if (rr >= nN) return;
    sell_level3_end(perm ? perm[rr] : rr, x, r, mask, t, binv, omega, ys, y0, y1, y2);
}

// ---- fused fine-level post-smoothing x = w D^-1 (r + t) + C e (amg_sa_body.h) ----------------
//
// C (3 x 6 blocks, the pattern of A P) in BF16, sliced like the fine system: slices of 32 finer
// rows (in the order perm: sorted by length within windows), slot e0 + 32 j + i holding slice row
// i's j-th block (padding: zero block, column 0); per slot one 16-byte word with values 0..7, one
// with values 8..15 and one 4-byte word with 16..17.

__device__ __forceinline__ uint32_t bf16x2_bits(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// slot t: C of AP block src[t] (or zeros)
__global__ void sa_post_setup_kernel(int64_t nSlot, const int32_t* __restrict__ src, const int32_t* __restrict__ apRow,
                                     const int32_t* __restrict__ apToP, const float* __restrict__ Pv,
                                     const float* __restrict__ APv, const float* __restrict__ binv, float omega,
                                     float alpha, uint4* __restrict__ q0, uint4* __restrict__ q1,
                                     uint32_t* __restrict__ q2) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nSlot) return;
    float C[18];
    const int64_t a = src[t];
    if (a >= 0) {
        sa_post_block<3>(a, apRow, apToP, Pv, APv, binv, omega, alpha, C);
    } else {
#pragma unroll
        for (int p = 0; p < 18; ++p) C[p] = 0.f;
    }
    q0[t] = make_uint4(bf16x2_bits(C[0], C[1]), bf16x2_bits(C[2], C[3]), bf16x2_bits(C[4], C[5]),
                       bf16x2_bits(C[6], C[7]));
    q1[t] = make_uint4(bf16x2_bits(C[8], C[9]), bf16x2_bits(C[10], C[11]), bf16x2_bits(C[12], C[13]),
                       bf16x2_bits(C[14], C[15]));
    q2[t] = bf16x2_bits(C[16], C[17]);
}

__device__ __forceinline__ float2 bf16x2_floats(uint32_t v) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
}

// y += C e of one block
__device__ __forceinline__ void sa_post_step(const float* ev, const uint4& u, const uint4& v, uint32_t w2,
                                             float& y0, float& y1, float& y2) {
    const float e0 = ev[0], e1 = ev[1], e2 = ev[2], e3 = ev[3], e4 = ev[4], e5 = ev[5];
    const float2 c01 = bf16x2_floats(u.x), c23 = bf16x2_floats(u.y), c45 = bf16x2_floats(u.z);
    const float2 c67 = bf16x2_floats(u.w), c89 = bf16x2_floats(v.x), cab = bf16x2_floats(v.y);
    const float2 ccd = bf16x2_floats(v.z), cef = bf16x2_floats(v.w), cgh = bf16x2_floats(w2);
    y0 += c01.x * e0 + c01.y * e1 + c23.x * e2 + c23.y * e3 + c45.x * e4 + c45.y * e5;
    y1 += c67.x * e0 + c67.y * e1 + c89.x * e2 + c89.y * e3 + cab.x * e4 + cab.y * e5;
    y2 += ccd.x * e0 + ccd.y * e1 + cef.x * e2 + cef.y * e3 + cgh.x * e4 + cgh.y * e5;
}

// the end of row m: x = w D^-1 (r + t) + y
__device__ __forceinline__ void sa_post_end(int m, const float* __restrict__ r, const float* __restrict__ t,
                                            const float* __restrict__ binv, const uint8_t* __restrict__ mask, float omega,
                                            float* __restrict__ x, float y0, float y1, float y2) {
    const int d = 3 * m;
    const float s0 = r[d] + t[d], s1 = r[d + 1] + t[d + 1], s2 = r[d + 2] + t[d + 2];
    const float* B = binv + 9 * (int64_t)m;
    const float z0 = B[0] * s0 + B[1] * s1 + B[2] * s2;
    const float z1 = B[3] * s0 + B[4] * s1 + B[5] * s2;
    const float z2 = B[6] * s0 + B[7] * s1 + B[8] * s2;
    x[d] = mask[d] ? 0.f : omega * z0 + y0;
    x[d + 1] = mask[d + 1] ? 0.f : omega * z1 + y1;
    x[d + 2] = mask[d + 2] ? 0.f : omega * z2 + y2;
}

// x = w D^-1 (r + t) + sum over the row's C blocks of C e[col] (masked DOFs 0); S warps per slice
template <int S>
__global__ void __launch_bounds__(sell_split_threads(S)) sa_post_fused_kernel(
    int nN, int nSlices, const int64_t* __restrict__ off, const int32_t* __restrict__ perm,
    const int32_t* __restrict__ col,
    const uint4* __restrict__ q0, const uint4* __restrict__ q1, const uint32_t* __restrict__ q2,
    const float* __restrict__ e, const float* __restrict__ r, const float* __restrict__ t,
    const float* __restrict__ binv, const uint8_t* __restrict__ mask, float omega, float* __restrict__ x) {
    ef::dep_entry();
    SellPart p;
    const bool active = sell_part<S>(nSlices, off, p);
    float y0 = 0.f, y1 = 0.f, y2 = 0.f;
    if (active) {
        const int32_t* cs = col + p.e0 + p.lane;
        const uint4* a0 = q0 + p.e0 + p.lane;
        const uint4* a1 = q1 + p.e0 + p.lane;
        const uint32_t* a2 = q2 + p.e0 + p.lane;
#pragma unroll 2
        for (int j = p.j0; j < p.j1; ++j) {
            const float* ev = e + 6 * (int64_t)__ldcs(cs + 32 * j);
            sa_post_step(ev, __ldcs(a0 + 32 * j), __ldcs(a1 + 32 * j), __ldcs(a2 + 32 * j), y0, y1, y2);
        }
    }
    if (!sell_combine<S>(p, active, y0, y1, y2)) return;
    const int rr = p.sl * 32 + p.lane;
    if (rr >= nN) return;
    sa_post_end(perm ? perm[rr] : rr, r, t, binv, mask, omega, x, y0, y1, y2);
}

}  // namespace ef

using namespace ef;

static inline unsigned sell_split_grid(int nSlices, int S) {
    const int spc = sell_split_threads(S) / (32 * S);
    return (unsigned)((nSlices + spc - 1) / spc);
}

ef_status ef_launch_sell_refresh(int64_t nE, const int32_t* src, const float* bsr, float* v9, void* v8, void* v1,
                                 const int32_t* col, const float* binv, const uint8_t* mask, int diaN, cudaStream_t s) {
    if (nE <= 0) return EF_OK;
    sell_refresh_kernel<<<(unsigned)((nE + 255) / 256), 256, 0, ef::counted(s)>>>(
        nE, src, bsr, v9, (uint4*)v8, (__nv_bfloat16*)v1, col, binv, mask, diaN);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_sell_spmv3(int nN, int nSlices, const int64_t* off, const int32_t* perm, const int32_t* col,
                               const float* v9, const float* x, const uint8_t* mask, float* y, float* xcopy, int split,
                               cudaStream_t s, const float* scale, const int32_t* dia, int diaN, const float* binv) {
    if (nSlices <= 0) return EF_OK;
#define EF_SPMV3(C_, S_)                                                                                              \
    do {                                                                                                              \
        if (dia && nN > 60000)                                                                                        \
            EF_CUDA(ef::launch_dep(sell_spmv3_dia_kernel<C_, S_, true>, sell_split_grid(nSlices, S_),                 \
                                   sell_split_threads(S_), 0, s, nN, nSlices, diaN, v9, x, mask, y, xcopy, scale,     \
                                   dia, binv));                                                                       \
        else if (dia)                                                                                                 \
            EF_CUDA(ef::launch_dep(sell_spmv3_dia_kernel<C_, S_, false>, sell_split_grid(nSlices, S_),                \
                                   sell_split_threads(S_), 0, s, nN, nSlices, diaN, v9, x, mask, y, xcopy, scale,     \
                                   dia, binv));                                                                       \
        else                                                                                                          \
            EF_CUDA(ef::launch_dep(sell_spmv3_kernel<C_, S_>, sell_split_grid(nSlices, S_), sell_split_threads(S_),   \
                                   0, s, nN, nSlices, off, perm, col, v9, x, mask, y, xcopy, scale, binv));           \
    } while (0)
#define EF_SPMV3_S(C_)      \
    if (split == 2)         \
        EF_SPMV3(C_, 2);    \
    else if (split == 4)    \
        EF_SPMV3(C_, 4);    \
    else if (split == 8)    \
        EF_SPMV3(C_, 8);    \
    else if (split == 16)   \
        EF_SPMV3(C_, 16);   \
    else if (split == 32)   \
        EF_SPMV3(C_, 32);   \
    else                    \
        EF_SPMV3(C_, 1)
    if (xcopy) {
        EF_SPMV3_S(true);
    } else {
        EF_SPMV3_S(false);
    }
#undef EF_SPMV3_S
#undef EF_SPMV3
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_sell_level3_bf16(int nN, int nSlices, const int64_t* off, const int32_t* perm, const int32_t* col,
                                     const void* v8, const void* v1, const float* x, const float* r,
                                     const uint8_t* mask, float* t, const float* binv, float omega, int split,
                                     cudaStream_t s, float ys, const int32_t* dia) {
    if (nSlices <= 0) return EF_OK;
#define EF_L3(S_)                                                                                                    \
    do {                                                                                                             \
        if (dia)                                                                                                     \
            EF_CUDA(ef::launch_dep(sell_level3_bf16_kernel<S_, true>, sell_split_grid(nSlices, S_),                  \
                                   sell_split_threads(S_), 0, s, nN, nSlices, off, perm, col, (const uint4*)v8,      \
                                   (const __nv_bfloat16*)v1, x, r, mask, t, binv, omega, ys, dia));                  \
        else                                                                                                         \
            EF_CUDA(ef::launch_dep(sell_level3_bf16_kernel<S_, false>, sell_split_grid(nSlices, S_),                 \
                                   sell_split_threads(S_), 0, s, nN, nSlices, off, perm, col, (const uint4*)v8,      \
                                   (const __nv_bfloat16*)v1, x, r, mask, t, binv, omega, ys, dia));                  \
    } while (0)
    if (split == 1)
        EF_L3(1);
    else if (split == 2)
        EF_L3(2);
    else if (split == 8)
        EF_L3(8);
    else if (split == 16)
        EF_L3(16);
    else if (split == 32)
        EF_L3(32);
    else
        EF_L3(4);
#undef EF_L3
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_sa_post_setup(int64_t nSlot, const int32_t* src, const int32_t* apRow, const int32_t* apToP,
                                  const float* Pv, const float* APv, const float* binv, float omega, float alpha,
                                  void* q0, void* q1, void* q2, cudaStream_t s) {
    if (nSlot <= 0) return EF_OK;
    sa_post_setup_kernel<<<(unsigned)((nSlot + 255) / 256), 256, 0, ef::counted(s)>>>(
        nSlot, src, apRow, apToP, Pv, APv, binv, omega, alpha, (uint4*)q0, (uint4*)q1, (uint32_t*)q2);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

ef_status ef_launch_sa_post_fused(int nN, int nSlices, const int64_t* off, const int32_t* perm, const int32_t* col,
                                  const void* q0, const void* q1, const void* q2, const float* e, const float* r,
                                  const float* t, const float* binv, const uint8_t* mask, float omega, float* x,
                                  int split, cudaStream_t s) {
    if (nSlices <= 0) return EF_OK;
#define EF_POST(S_)                                                                                              \
    EF_CUDA(ef::launch_dep(sa_post_fused_kernel<S_>, sell_split_grid(nSlices, S_), sell_split_threads(S_), 0, s, \
                           nN, nSlices, off, perm, col, (const uint4*)q0, (const uint4*)q1, (const uint32_t*)q2, e, r, \
                           t, binv, mask, omega, x))
    if (split == 1)
        EF_POST(1);
    else if (split == 2)
        EF_POST(2);
    else if (split == 8)
        EF_POST(8);
    else if (split >= 16)
        EF_POST(16);
    else
        EF_POST(4);
#undef EF_POST
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}
