// Batched small-strain displacement element kernels (C3D8 / C3D20 families).
//
// One kernel launch evaluates every element of a group: shape-function
// gradients, strain increment, the constitutive update per Gauss point
// (linear elastic or J2 radial return in FP64), the element residual Pe in
// FP64 and the element stiffness Ke (FP32 or FP64) as 3x3 node-pair blocks.
//
// Reference semantics (EdelweissFE):
//   elements/displacementelement/element.py:290-346   computeYourself
//   elements/displacementelement/_elementcomputationmatrices.py:306-366,679-817 (hex8)
//   elements/displacementelement/_elementcomputationmatrices.py:369-495,820+   (hex20)
//   materials/linearelastic/linearelastic.py:95-125,185-210
//   materials/vonmises/vonmises.py:35-56,105-124,186-254
//
// Thread mapping: TPE threads per element (8 for <= 8 Gauss points, 32
// otherwise); thread `lane` of an element owns Gauss point `lane` for the
// constitutive phase and node `lane` for the residual phase; in the stiffness
// phase the node pairs of all the CTA's elements are dealt out over its threads.
// Per-element scratch lives in shared memory; the state is structure-of-arrays [var][element*nQP + qp] so
// that the constitutive phase reads and writes it coalesced.

#include <math.h>

#include "dfloat_bits.h"
#include "ef_common.cuh"
#include "materials.h"

namespace ef {

constexpr int kBlock = 128;

template <int NN>
struct PairTab {
    static constexpr int NP = NN * (NN + 1) / 2;
};

__device__ __forceinline__ int pair_a(int p, int nn) {
    // inverse of p(a,b) = a*nn - a*(a-1)/2 + (b-a), a <= b
    int a = 0;
    int start = 0;
    while (start + (nn - a) <= p) {
        start += nn - a;
        ++a;
    }
    return a;
}

// Double-float arithmetic (Dekker 1971; Knuth's TwoSum): a value is an unevaluated pair of
// FP32 numbers hi + lo with |lo| <= ulp(hi) / 2, about 48 significant bits.  The element kernel
// forms its strain and residual contractions this way on the FP32 pipe, because the FP64 pipe
// of this GPU (2 lanes per SM and cycle) bounds the kernel.  The rounded operations are written
// with the _rn intrinsics so that the compiler cannot contract them into FMAs.
struct DF {
    float hi, lo;
};

__host__ __device__ __forceinline__ float2 df_split(double d) {
    const float hi = (float)d;
    return make_float2(hi, (float)(d - (double)hi));
}

__device__ __forceinline__ double df_value(const DF& a) { return (double)a.hi + (double)a.lo; }

// the same conversions by integer operations on the bit patterns (dfloat_bits.h), which keep them
// off the FP64 pipe; hi is truncated instead of rounded (the pair still holds 47 bits)
__device__ __forceinline__ float2 df_split_i(double d) {
    uint32_t h, l;
    split_bits((uint64_t)__double_as_longlong(d), &h, &l);
    return make_float2(__uint_as_float(h), __uint_as_float(l));
}
__device__ __forceinline__ double widen_i(float f) { return __longlong_as_double((long long)widen_bits(__float_as_uint(f))); }
__device__ __forceinline__ double df_value_i(const DF& a) { return widen_i(a.hi) + widen_i(a.lo); }
__device__ __forceinline__ float2 df_split_sel(double d, int intConv) { return intConv ? df_split_i(d) : df_split(d); }
__device__ __forceinline__ double df_value_sel(const DF& a, int intConv) {
    return intConv ? df_value_i(a) : df_value(a);
}
// NaN test: a floating-point compare (FP64 pipe), or with intConv the exponent-all-ones,
// nonzero-fraction test on the bit pattern (integer pipe)
__device__ __forceinline__ bool is_nan_sel(double x, int intConv) {
    if (intConv) return ((unsigned long long)__double_as_longlong(x) << 1) > (0x7FF0000000000000ull << 1);
    return !(x == x);
}

// acc += a * b for a = (ah, al), b = (bh, bl): the product ah bh exactly (its rounding error from
// an FMA), the cross terms ah bl + al bh in FP32 (relative 2^-24 of the product), al bl dropped
// (2^-48); the sum with acc.hi by TwoSum, every error term into acc.lo
__device__ __forceinline__ void df_fma(DF& acc, float2 a, float2 b) {
    const float p = __fmul_rn(a.x, b.x);
    const float pe = __fmaf_rn(a.x, b.x, -p);
    const float x = __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x));
    const float s = __fadd_rn(acc.hi, p);
    const float bv = __fsub_rn(s, acc.hi);
    const float err = __fadd_rn(__fsub_rn(acc.hi, __fsub_rn(s, bv)), __fsub_rn(p, bv));
    acc.hi = s;
    acc.lo = __fadd_rn(acc.lo, __fadd_rn(err, __fadd_rn(pe, x)));
}

// Gauss-point geometry in FP64: J = dN/dS x (reference formulation, including the C3D20
// row-2 Jacobian term), det J and g_a = dN_a/dx = inv(J) dN_a/dS.
template <int NN>
__device__ __forceinline__ double qp_geometry(const ElemTables* __restrict__ T, int q, const double (*xr)[3],
                                              double (*g)[3]) {
    double J[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double s = 0;
#pragma unroll
            for (int a = 0; a < NN; ++a) s += T->dNdS_d[q][r][a] * xr[a][c];
            J[r][c] = s;
        }
    if (NN == 20 && T->quirk) {
        // reference _J3D20 (_elementcomputationmatrices.py:481-495) row-2 term a5*zeta instead of a5*xi
        const double f = T->quirkFac[q];
#pragma unroll
        for (int c = 0; c < 3; ++c) J[2][c] += f * 0.25 * (-xr[9][c] + xr[11][c] + xr[13][c] - xr[15][c]);
    }
    const double c00 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
    const double c01 = J[1][2] * J[2][0] - J[1][0] * J[2][2];
    const double c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
    const double det = J[0][0] * c00 + J[0][1] * c01 + J[0][2] * c02;
    const double id = 1.0 / det;
    double iJ[3][3];
    iJ[0][0] = c00 * id;
    iJ[1][0] = c01 * id;
    iJ[2][0] = c02 * id;
    iJ[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) * id;
    iJ[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * id;
    iJ[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) * id;
    iJ[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * id;
    iJ[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) * id;
    iJ[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * id;
    for (int a = 0; a < NN; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            g[a][c] = iJ[c][0] * T->dNdS_d[q][0][a] + iJ[c][1] * T->dNdS_d[q][1][a] + iJ[c][2] * T->dNdS_d[q][2][a];
    return det;
}

// Geometry cache, computed once per element group (initializeElement, element.py:194-205):
// geo[(e*NQ + q) * (3*NN + 1) + 3a + c] = dN_a/dx_c, last entry = w_q det J.
template <int NN, int NQ>
__global__ void geometry_kernel(const ElemTables* __restrict__ T, int nEl, const int32_t* __restrict__ nodeDof,
                                const double* __restrict__ X, double* __restrict__ geo, float2* __restrict__ geoS,
                                int* __restrict__ flags) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)nEl * NQ) return;
    const int64_t e = t / NQ;
    const int q = (int)(t % NQ);
    double xr[NN][3];
    const int d0 = nodeDof[e * NN];
    for (int a = 0; a < NN; ++a) {
        const int d = nodeDof[e * NN + a];
#pragma unroll
        for (int c = 0; c < 3; ++c) xr[a][c] = X[d + c] - X[d0 + c];
    }
    double g[NN][3];
    const double det = qp_geometry<NN>(T, q, xr, g);
    if (!(det > 0.0)) atomicOr(flags, EF_FLAG_BADDET);
    double* o = geo + t * (3 * NN + 1);
    for (int a = 0; a < NN; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) o[3 * a + c] = g[a][c];
    o[3 * NN] = T->w[q] * det;
    if (geoS) {
        float2* os = geoS + t * (3 * NN + 1);
        for (int k = 0; k <= 3 * NN; ++k) os[k] = df_split(o[k]);
    }
}

// x with its sign flipped where neg has the sign bit (integer pipe)
__device__ __forceinline__ double flip_sign(double x, int neg) {
    return __hiloint2double(__double2hiint(x) ^ neg, __double2loint(x));
}

template <int NN, int NQ, typename KT>
struct SSShared {
    static constexpr int TPE = (NQ <= 8) ? 8 : 32;
    // FP64: small CTAs (8 elements of 8 Gauss points, 2 of 27, whose scratch is twice as large), which deal the FP64 pipe's
    // work out evenly over the SMs where an SM gets few elements (2,500 hex8: 113 -> 93 us with 4 or 8 of them for 16)
    static constexpr int BLOCK = sizeof(KT) == 8 ? 64 : kBlock;
    static constexpr int EPB = BLOCK / TPE;
    static constexpr int NG = NQ * NN * 3 + 1;
    // per-element rows padded by one entry, so that the elements of a warp fall on different banks
    float2 du[EPB][NN * 3 + 1];       // dU split into FP32 pairs, [3a + i]
    float2 sw[EPB][NQ * 6 + 1];       // sigma w detJ split into FP32 pairs, [6q + i]
    KT tn[EPB][NQ][9];                // FP32 and FP64 with one Gauss point: lt*w, mt*w, c1*w, n[6]; FP64: c2, c1, w (its sign)
    union {
        float2 g[EPB][NG];            // dN/dx split into FP32 pairs, [(q NN + a) 3 + c] (the FP32 stiffness reads hi)
        struct {                      // the FP64 stiffness, once the residual is done with g
            double gd[EPB][NG];       // sqrt(|w detJ|) dN/dx (one Gauss point: dN/dx)
            double vd[sizeof(KT) == 8 ? EPB : 1][sizeof(KT) == 8 ? NG : 1];  // n . gd, where plastic
        } d;
    } u;
};

// Element loop of one group: strain increment, constitutive update, Pe (FP64) and Ke blocks (KT).
template <int NN, int NQ, typename KT, int MAT, bool VIJ>
__global__ void __launch_bounds__(SSShared<NN, NQ, KT>::BLOCK, sizeof(KT) == 8 ? (NQ <= 8 ? 6 : 4) : 5) small_strain_kernel(
    int nEl, const int32_t* __restrict__ nodeDof, const float2* __restrict__ geoS, const double* __restrict__ geo,
    const double* __restrict__ dU,
    const double* __restrict__ stateIn, double* __restrict__ stateOut, PropsArg props,
    const double* __restrict__ propsTable, const int32_t* __restrict__ elemRow, KT* __restrict__ Kout,
    double* __restrict__ Pe, double* __restrict__ tang, int* __restrict__ flags, int intConv) {
    constexpr int TPE = (NQ <= 8) ? 8 : 32;
    constexpr int EPB = SSShared<NN, NQ, KT>::EPB;
    constexpr int NP = PairTab<NN>::NP;
    constexpr int ND = 3 * NN;
    constexpr int NG = 3 * NN + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SSShared<NN, NQ, KT>& sh = *reinterpret_cast<SSShared<NN, NQ, KT>*>(smem_raw);
    const int tid = threadIdx.x;
    const int le = tid / TPE;
    const int lane = tid % TPE;
    const int e = blockIdx.x * EPB + le;
    const bool valid = e < nEl;

    if (valid) {
        for (int a = lane; a < NN; a += TPE) {
            const int d = nodeDof[(int64_t)e * NN + a];
            sh.du[le][3 * a + 0] = df_split_sel(dU[d + 0], intConv);
            sh.du[le][3 * a + 1] = df_split_sel(dU[d + 1], intConv);
            sh.du[le][3 * a + 2] = df_split_sel(dU[d + 2], intConv);
        }
    }
    __syncthreads();

    MatOut mo;
    mo.c1 = mo.c2 = 0.0;
    const double* pv = propsTable ? propsTable + 8 * (int64_t)elemRow[valid ? e : 0] : props.v;
    // ---- Gauss-point phase ---------------------------------------------------
    if (valid && lane < NQ) {
        const int q = lane;
        const float2* gq = geoS + ((int64_t)e * NQ + q) * NG;
        // displacement-increment gradient H = sum_a dU_a (x) g_a in double-float arithmetic
        DF H[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) H[i][j] = DF{0.f, 0.f};
#pragma unroll 4
        for (int a = 0; a < NN; ++a) {
            float2 ga[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                ga[c] = gq[3 * a + c];
                sh.u.g[le][(q * NN + a) * 3 + c] = ga[c];
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const float2 u = sh.du[le][3 * a + i];
#pragma unroll
                for (int j = 0; j < 3; ++j) df_fma(H[i][j], u, ga[j]);
            }
        }
        const float2 wq = gq[3 * NN];
        const double wdet = df_value_sel(DF{wq.x, wq.y}, intConv);
        const double de[6] = {df_value_sel(H[0][0], intConv), df_value_sel(H[1][1], intConv),
                              df_value_sel(H[2][2], intConv),
                              df_value_sel(H[0][1], intConv) + df_value_sel(H[1][0], intConv),
                              df_value_sel(H[0][2], intConv) + df_value_sel(H[2][0], intConv),
                              df_value_sel(H[1][2], intConv) + df_value_sel(H[2][1], intConv)};
        const int64_t nQPtot = (int64_t)nEl * NQ;
        const int64_t qi = (int64_t)e * NQ + q;
        double sig[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) sig[i] = stateIn[i * nQPtot + qi];
        if (MAT == MAT_VON_MISES) {
            double kap = stateIn[12 * nQPtot + qi];
            if (!mat_von_mises(pv, sig, &kap, de, mo)) {
                atomicOr(flags, EF_FLAG_RETURNMAP);
                atomicMin(flags + 1, __float_as_int(props.cutback));
            }
            stateOut[12 * nQPtot + qi] = kap;
            if (is_nan_sel(kap, intConv)) atomicOr(flags, EF_FLAG_NAN);
        } else {
            mat_linear_elastic(pv, sig, de, mo);
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            stateOut[i * nQPtot + qi] = sig[i];
            stateOut[(6 + i) * nQPtot + qi] = stateIn[(6 + i) * nQPtot + qi] + de[i];
            if (is_nan_sel(sig[i], intConv)) atomicOr(flags, EF_FLAG_NAN);
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) sh.sw[le][6 * q + i] = df_split_sel(sig[i] * wdet, intConv);
        if (tang) {
            // FP64 tangent of this Gauss point for the exact (matrix-free) refinement residual
            tang[0 * nQPtot + qi] = mo.lt * wdet;
            tang[1 * nQPtot + qi] = mo.mt * wdet;
            tang[2 * nQPtot + qi] = mo.c1 * wdet;
#pragma unroll
            for (int i = 0; i < 6; ++i) tang[(3 + i) * nQPtot + qi] = mo.c1 != 0.0 ? mo.n[i] : 0.0;
        }
        if (sizeof(KT) == 8 && NQ > 1) {
            sh.tn[le][q][0] = (KT)mo.c2;
            sh.tn[le][q][1] = (KT)mo.c1;
            sh.tn[le][q][2] = (KT)wdet;
        } else {
            sh.tn[le][q][0] = (KT)(mo.lt * wdet);
            sh.tn[le][q][1] = (KT)(mo.mt * wdet);
            sh.tn[le][q][2] = (KT)(mo.c1 * wdet);
            if (mo.c1 != 0.0) {
#pragma unroll
                for (int i = 0; i < 6; ++i) sh.tn[le][q][3 + i] = (KT)mo.n[i];
            }
        }
    }
    __syncthreads();

    // ---- residual: Pe_a = -sum_q (sigma w detJ) . g_qa  (double-float accumulation) ----
    for (int a = valid ? lane : NN; a < NN; a += TPE) {
        DF f0{0.f, 0.f}, f1{0.f, 0.f}, f2{0.f, 0.f};
#pragma unroll 2
        for (int q = 0; q < NQ; ++q) {
            const float2* s = &sh.sw[le][6 * q];
            const float2* gg = &sh.u.g[le][(q * NN + a) * 3];
            const float2 gx = gg[0], gy = gg[1], gz = gg[2];
            df_fma(f0, s[0], gx);
            df_fma(f0, s[3], gy);
            df_fma(f0, s[4], gz);
            df_fma(f1, s[3], gx);
            df_fma(f1, s[1], gy);
            df_fma(f1, s[5], gz);
            df_fma(f2, s[4], gx);
            df_fma(f2, s[5], gy);
            df_fma(f2, s[2], gz);
        }
        double* pe = Pe + (int64_t)e * ND + 3 * a;
        pe[0] = -df_value_sel(f0, intConv);
        pe[1] = -df_value_sel(f1, intConv);
        pe[2] = -df_value_sel(f2, intConv);
    }

    auto store = [&](int e, int p, int a, int b, const KT (&k)[3][3]) {
        if (VIJ) {
            // reference VIJ layout: value a*n+b of the element slice holds Ke[a][b]
            KT* ke = Kout + (int64_t)e * ND * ND;
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    ke[(3 * a + i) * ND + 3 * b + j] = k[i][j];
                    if (a != b) ke[(3 * b + j) * ND + 3 * a + i] = k[i][j];
                }
        } else {
            KT* kb = Kout + ((int64_t)e * NP + p) * 9;
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) kb[i * 3 + j] = k[i][j];
        }
    };
    // the pairs of nodes of the CTA's elements, dealt out over all threads: a warp has those of one or two elements (the
    // plastic branch is then rarely taken for some of its lanes only) and 36 pairs an element leave no lanes idle (10,240
    // hex8 J2 elements in FP64 312 -> 292 us, 160,000 in FP32, where the FP64 constitutive update bounds it, 478 -> 474)
    const int nItems = min(EPB, nEl - (int)blockIdx.x * EPB) * NP;
    if constexpr (sizeof(KT) == 8 && NQ == 1) {
        // ---- stiffness of one Gauss point in FP64: there is nothing to sum, so the three terms are formed per pair, 30
        // instructions and 12 more where plastic (as sums of outer products 30 and 60), from the FP64 gradients and va,
        // which the element's lanes make by nodes.  C3D8R J2 elements, us with both formed per pair from the split
        // geometry, as sums of outer products and now: 10,240 135, 150 and 88, 54,000 514, 587 and 306
        __syncthreads();  // the residual has read g
        for (int a = valid ? lane : NN; a < NN; a += TPE) {
            const double* gq = geo + (int64_t)e * (3 * NN + 1) + 3 * a;
            const double g0 = gq[0], g1 = gq[1], g2 = gq[2];
            double* gd = &sh.u.d.gd[le][3 * a];
            gd[0] = g0;
            gd[1] = g1;
            gd[2] = g2;
            const KT* tn = sh.tn[le][0];
            if (tn[2] != 0.0) {
                double* vd = &sh.u.d.vd[le][3 * a];
                vd[0] = fma(tn[7], g2, fma(tn[6], g1, tn[3] * g0));
                vd[1] = fma(tn[8], g2, fma(tn[4], g1, tn[6] * g0));
                vd[2] = fma(tn[5], g2, fma(tn[8], g1, tn[7] * g0));
            }
        }
        __syncthreads();
        for (int item = tid; item < nItems; item += SSShared<NN, NQ, KT>::BLOCK) {
            const int le = item / NP, p = item - le * NP;
            const int a = pair_a(p, NN);
            const int b = a + (p - (a * NN - a * (a - 1) / 2));
            const KT* tn = sh.tn[le][0];
            const double *ga = &sh.u.d.gd[le][3 * a], *gb = &sh.u.d.gd[le][3 * b];
            const double lt = tn[0], mt = tn[1], c1 = tn[2];
            const double la[3] = {lt * ga[0], lt * ga[1], lt * ga[2]}, mb[3] = {mt * gb[0], mt * gb[1], mt * gb[2]};
            const double s = fma(ga[2], mb[2], fma(ga[1], mb[1], ga[0] * mb[0]));
            KT k[3][3];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) k[i][j] = fma(la[i], gb[j], i == j ? fma(mb[i], ga[j], s) : mb[i] * ga[j]);
            if (MAT == MAT_VON_MISES && c1 != 0.0) {
                const double *va = &sh.u.d.vd[le][3 * a], *vb = &sh.u.d.vd[le][3 * b];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const double cv = c1 * va[i];
#pragma unroll
                    for (int j = 0; j < 3; ++j) k[i][j] = fma(-cv, vb[j], k[i][j]);
                }
            }
            store(blockIdx.x * EPB + le, p, a, b, k);
        }
        return;
    } else if constexpr (sizeof(KT) == 8) {
        // ---- stiffness in FP64, which the FP64 pipe bounds: K_ab = sum_q lt ga(x)gb + mt (gb(x)ga + ga.gb I)
        // - c1 va(x)vb with lt = lam + c2/3, mt = G - c2/2 and lam, G of the element, so that
        //   K = lam A + G (A^T + tr A I) + B/3 - (B^T + tr B I)/2 - V,
        //   A = sum_q ga(x)gb, B = sum_q c2 ga(x)gb, V = sum_q c1 va(x)vb, g with sqrt(|w detJ|) in it and the sign
        // of w detJ (negative in an inverted element, which the element status reports) given to ga and va, va with
        // sqrt(|c1|) in it:
        // 9 instructions per pair of nodes and elastic Gauss point, 30 where plastic, against 58 and 88 with the
        // three terms formed per pair from the split geometry (10,240 hex8 J2 elements, half of them plastic: 659 us with
        // the FP64 pipe 87 % busy, 292 now with it 75 to 80 %; 2,500 elements 92).  The FP64 geometry (not its 48-bit split) is
        // scaled once per Gauss point and node, va = n . ga likewise.
        __syncthreads();  // the residual has read g
        if (valid && lane < NQ) {
            const int q = lane;
            const double* gq = geo + ((int64_t)e * NQ + q) * (3 * NN + 1);
            const double sw = sqrt(fabs(gq[3 * NN]));
            const bool plasticQ = mo.c1 != 0.0 || mo.c2 != 0.0;
            double n[6];
            if (plasticQ) {
                const double rc = sqrt(fabs(mo.c1));
#pragma unroll
                for (int i = 0; i < 6; ++i) n[i] = rc * mo.n[i];
            }
#pragma unroll 2
            for (int a = 0; a < NN; ++a) {
                const double g0 = sw * gq[3 * a], g1 = sw * gq[3 * a + 1], g2 = sw * gq[3 * a + 2];
                double* gd = &sh.u.d.gd[le][(q * NN + a) * 3];
                gd[0] = g0;
                gd[1] = g1;
                gd[2] = g2;
                if (plasticQ) {
                    double* vd = &sh.u.d.vd[le][(q * NN + a) * 3];
                    vd[0] = fma(n[4], g2, fma(n[3], g1, n[0] * g0));
                    vd[1] = fma(n[5], g2, fma(n[1], g1, n[3] * g0));
                    vd[2] = fma(n[2], g2, fma(n[5], g1, n[4] * g0));
                }
            }
        }
        __syncthreads();
        for (int item = tid; item < nItems; item += SSShared<NN, NQ, KT>::BLOCK) {
            const int le = item / NP, p = item - le * NP, e = blockIdx.x * EPB + le;
            const double* pv = propsTable ? propsTable + 8 * (int64_t)elemRow[e] : props.v;
            const double lam = pv[6], G = pv[7];
            const int a = pair_a(p, NN);
            const int b = a + (p - (a * NN - a * (a - 1) / 2));
            double A[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, B[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
            double V[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
            bool plastic = false;
            for (int q = 0; q < NQ; ++q) {
                const double* gA = &sh.u.d.gd[le][(q * NN + a) * 3];
                const double* gB = &sh.u.d.gd[le][(q * NN + b) * 3];
                const int neg = __double2hiint(sh.tn[le][q][2]) & 0x80000000;
                const double ga[3] = {flip_sign(gA[0], neg), flip_sign(gA[1], neg), flip_sign(gA[2], neg)};
                const double gb[3] = {gB[0], gB[1], gB[2]};
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) A[i][j] = fma(ga[i], gb[j], A[i][j]);
                const double c2 = sh.tn[le][q][0], c1 = sh.tn[le][q][1];
                if (MAT == MAT_VON_MISES && (__double2hiint(c2) | __double2hiint(c1)) != 0) {
                    plastic = true;
                    const double* vA = &sh.u.d.vd[le][(q * NN + a) * 3];
                    const double* vB = &sh.u.d.vd[le][(q * NN + b) * 3];
                    const double cg[3] = {c2 * ga[0], c2 * ga[1], c2 * ga[2]};
                    const int neg1 = neg ^ (__double2hiint(c1) & 0x80000000);
                    const double cv[3] = {flip_sign(vA[0], neg1), flip_sign(vA[1], neg1), flip_sign(vA[2], neg1)};
                    const double vb[3] = {vB[0], vB[1], vB[2]};
#pragma unroll
                    for (int i = 0; i < 3; ++i)
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            B[i][j] = fma(cg[i], gb[j], B[i][j]);
                            V[i][j] = fma(cv[i], vb[j], V[i][j]);
                        }
                }
            }
            KT k[3][3];
            const double s = G * (A[0][0] + A[1][1] + A[2][2]);
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) k[i][j] = fma(G, A[j][i], i == j ? fma(lam, A[i][j], s) : lam * A[i][j]);
            if (plastic) {
                const double h = -0.5 * (B[0][0] + B[1][1] + B[2][2]);
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const double t = fma(-0.5, B[j][i], fma(1.0 / 3.0, B[i][j], (i == j ? h : 0.0) - V[i][j]));
                        k[i][j] += t;
                    }
            }
            store(e, p, a, b, k);
        }
        return;
    }
    // ---- stiffness: K_ab = sum_q lt ga(x)gb + mt (gb(x)ga + ga.gb I) - c1 va(x)vb ----
    for (int item = tid; item < nItems; item += SSShared<NN, NQ, KT>::BLOCK) {
        const int le = item / NP, p = item - le * NP;
        const int a = pair_a(p, NN);
        const int b = a + (p - (a * NN - a * (a - 1) / 2));
        KT k[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        for (int q = 0; q < NQ; ++q) {
            const KT* tn = sh.tn[le][q];
            const float2* gA = &sh.u.g[le][(q * NN + a) * 3];
            const float2* gB = &sh.u.g[le][(q * NN + b) * 3];
            const KT ga0 = (KT)gA[0].x, ga1 = (KT)gA[1].x, ga2 = (KT)gA[2].x;
            const KT gb0 = (KT)gB[0].x, gb1 = (KT)gB[1].x, gb2 = (KT)gB[2].x;
            const KT lt = tn[0], mt = tn[1], c1 = tn[2];
            const KT s = mt * (ga0 * gb0 + ga1 * gb1 + ga2 * gb2);
            const KT la[3] = {lt * ga0, lt * ga1, lt * ga2};
            const KT ma[3] = {mt * gb0, mt * gb1, mt * gb2};
            const KT gaa[3] = {ga0, ga1, ga2};
            const KT gbb[3] = {gb0, gb1, gb2};
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) k[i][j] += la[i] * gbb[j] + ma[i] * gaa[j];
#pragma unroll
            for (int i = 0; i < 3; ++i) k[i][i] += s;
            if (c1 != (KT)0) {
                const KT* n = tn + 3;
                const KT va[3] = {n[0] * ga0 + n[3] * ga1 + n[4] * ga2, n[3] * ga0 + n[1] * ga1 + n[5] * ga2,
                                  n[4] * ga0 + n[5] * ga1 + n[2] * ga2};
                const KT vb[3] = {n[0] * gb0 + n[3] * gb1 + n[4] * gb2, n[3] * gb0 + n[1] * gb1 + n[5] * gb2,
                                  n[4] * gb0 + n[5] * gb1 + n[2] * gb2};
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) k[i][j] -= c1 * va[i] * vb[j];
            }
        }
        store(blockIdx.x * EPB + le, p, a, b, k);
    }
}

// y_e = K_e x_e with the FP64 Gauss-point tangents stored by the assembly (matrix-free, FP64).
// Used for the residual of the iterative refinement, so that a mixed-precision solve is exact
// for the FP64 tangent.
template <int NN, int NQ>
struct ApplyShared {
    static constexpr int TPE = (NQ <= 8) ? 8 : 32;
    static constexpr int EPB = kBlock / TPE;
    // per-element rows padded by one entry (bank spread of the elements of a warp)
    double xv[EPB][NN * 3 + 1];
    double g[EPB][NQ * NN * 3 + 1];
    double sw[EPB][NQ * 6 + 1];
};

template <int NN, int NQ>
__global__ void __launch_bounds__(kBlock) small_strain_apply_kernel(int nEl, const int32_t* __restrict__ nodeDof,
                                                                    const double* __restrict__ geo,
                                                                    const double* __restrict__ x,
                                                                    const double* __restrict__ tang,
                                                                    double* __restrict__ ye) {
    constexpr int TPE = (NQ <= 8) ? 8 : 32;
    constexpr int EPB = kBlock / TPE;
    constexpr int ND = 3 * NN;
    constexpr int NG = 3 * NN + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ApplyShared<NN, NQ>& sh = *reinterpret_cast<ApplyShared<NN, NQ>*>(smem_raw);
    const int tid = threadIdx.x;
    const int le = tid / TPE;
    const int lane = tid % TPE;
    const int e = blockIdx.x * EPB + le;
    const bool valid = e < nEl;
    if (valid) {
        for (int a = lane; a < NN; a += TPE) {
            const int d = nodeDof[(int64_t)e * NN + a];
            sh.xv[le][3 * a + 0] = x[d + 0];
            sh.xv[le][3 * a + 1] = x[d + 1];
            sh.xv[le][3 * a + 2] = x[d + 2];
        }
    }
    __syncthreads();
    if (valid && lane < NQ) {
        const int q = lane;
        const double* gq = geo + ((int64_t)e * NQ + q) * NG;
        double H[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
        for (int a = 0; a < NN; ++a) {
#pragma unroll
            for (int c = 0; c < 3; ++c) sh.g[le][(q * NN + a) * 3 + c] = gq[3 * a + c];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) H[i][j] += sh.xv[le][3 * a + i] * sh.g[le][(q * NN + a) * 3 + j];
        }
        const double ep[6] = {H[0][0], H[1][1], H[2][2], H[0][1] + H[1][0], H[0][2] + H[2][0], H[1][2] + H[2][1]};
        const int64_t nQPtot = (int64_t)nEl * NQ;
        const int64_t qi = (int64_t)e * NQ + q;
        const double lt = tang[qi], mt = tang[nQPtot + qi], c1 = tang[2 * nQPtot + qi];
        const double tr = ep[0] + ep[1] + ep[2];
        double ne = 0.0, n[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) n[i] = 0.0;
        if (c1 != 0.0) {
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                n[i] = tang[(3 + i) * nQPtot + qi];
                ne += n[i] * ep[i];
            }
        }
        // sigma = (lt 1x1 + 2 mt I_s - c1 n x n) eps   (weights already in lt, mt, c1)
#pragma unroll
        for (int i = 0; i < 3; ++i) sh.sw[le][6 * q + i] = lt * tr + 2.0 * mt * ep[i] - c1 * n[i] * ne;
#pragma unroll
        for (int i = 3; i < 6; ++i) sh.sw[le][6 * q + i] = mt * ep[i] - c1 * n[i] * ne;
    }
    __syncthreads();
    if (!valid) return;
    for (int a = lane; a < NN; a += TPE) {
        double f0 = 0, f1 = 0, f2 = 0;
        for (int q = 0; q < NQ; ++q) {
            const double* s = &sh.sw[le][6 * q];
            const double* gg = &sh.g[le][(q * NN + a) * 3];
            const double gx = gg[0], gy = gg[1], gz = gg[2];
            f0 += s[0] * gx + s[3] * gy + s[4] * gz;
            f1 += s[3] * gx + s[1] * gy + s[5] * gz;
            f2 += s[4] * gx + s[5] * gy + s[2] * gz;
        }
        double* o = ye + (int64_t)e * ND + 3 * a;
        o[0] = f0;
        o[1] = f1;
        o[2] = f2;
    }
}

// The same product with the contractions in double-float arithmetic on the FP32 pipe (the FP64
// pipe of this GPU executes 2 lanes per SM and cycle): x split once into FP32 pairs, the
// geometry read from the split cache, H = sum_a x_a (x) g_a and y_a = sum_q sigma_q . g_qa as
// double-float sums (about 48 significant bits, as the element kernel's strain increment and
// residual), the Gauss-point stress from the FP64 tangent in FP64.
template <int NN, int NQ>
struct ApplyDFShared {
    static constexpr int TPE = (NQ <= 8) ? 8 : 32;
    static constexpr int EPB = kBlock / TPE;
    float2 xv[EPB][NN * 3 + 1];
    float2 g[EPB][NQ * NN * 3 + 1];
    float2 sw[EPB][NQ * 6 + 1];
};

template <int NN, int NQ>
__global__ void __launch_bounds__(kBlock) small_strain_apply_df_kernel(int nEl, const int32_t* __restrict__ nodeDof,
                                                                       const float2* __restrict__ geoS,
                                                                       const double* __restrict__ x,
                                                                       const double* __restrict__ tang,
                                                                       double* __restrict__ ye, int intConv) {
    constexpr int TPE = (NQ <= 8) ? 8 : 32;
    constexpr int EPB = kBlock / TPE;
    constexpr int ND = 3 * NN;
    constexpr int NG = 3 * NN + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ApplyDFShared<NN, NQ>& sh = *reinterpret_cast<ApplyDFShared<NN, NQ>*>(smem_raw);
    const int tid = threadIdx.x;
    const int le = tid / TPE;
    const int lane = tid % TPE;
    const int e = blockIdx.x * EPB + le;
    const bool valid = e < nEl;
    if (valid) {
        for (int a = lane; a < NN; a += TPE) {
            const int d = nodeDof[(int64_t)e * NN + a];
            sh.xv[le][3 * a + 0] = df_split_sel(x[d + 0], intConv);
            sh.xv[le][3 * a + 1] = df_split_sel(x[d + 1], intConv);
            sh.xv[le][3 * a + 2] = df_split_sel(x[d + 2], intConv);
        }
    }
    __syncthreads();
    if (valid && lane < NQ) {
        const int q = lane;
        const float2* gq = geoS + ((int64_t)e * NQ + q) * NG;
        DF H[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) H[i][j] = DF{0.f, 0.f};
#pragma unroll 4
        for (int a = 0; a < NN; ++a) {
            float2 ga[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                ga[c] = gq[3 * a + c];
                sh.g[le][(q * NN + a) * 3 + c] = ga[c];
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const float2 u = sh.xv[le][3 * a + i];
#pragma unroll
                for (int j = 0; j < 3; ++j) df_fma(H[i][j], u, ga[j]);
            }
        }
        const double ep[6] = {df_value_sel(H[0][0], intConv), df_value_sel(H[1][1], intConv),
                              df_value_sel(H[2][2], intConv),
                              df_value_sel(H[0][1], intConv) + df_value_sel(H[1][0], intConv),
                              df_value_sel(H[0][2], intConv) + df_value_sel(H[2][0], intConv),
                              df_value_sel(H[1][2], intConv) + df_value_sel(H[2][1], intConv)};
        const int64_t nQPtot = (int64_t)nEl * NQ;
        const int64_t qi = (int64_t)e * NQ + q;
        const double lt = tang[qi], mt = tang[nQPtot + qi], c1 = tang[2 * nQPtot + qi];
        const double tr = ep[0] + ep[1] + ep[2];
        double ne = 0.0, n[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) n[i] = 0.0;
        if (c1 != 0.0) {
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                n[i] = tang[(3 + i) * nQPtot + qi];
                ne += n[i] * ep[i];
            }
        }
        // sigma = (lt 1x1 + 2 mt I_s - c1 n x n) eps   (weights already in lt, mt, c1)
#pragma unroll
        for (int i = 0; i < 3; ++i) sh.sw[le][6 * q + i] = df_split_sel(lt * tr + 2.0 * mt * ep[i] - c1 * n[i] * ne, intConv);
#pragma unroll
        for (int i = 3; i < 6; ++i) sh.sw[le][6 * q + i] = df_split_sel(mt * ep[i] - c1 * n[i] * ne, intConv);
    }
    __syncthreads();
    if (!valid) return;
    for (int a = lane; a < NN; a += TPE) {
        DF f0{0.f, 0.f}, f1{0.f, 0.f}, f2{0.f, 0.f};
#pragma unroll 2
        for (int q = 0; q < NQ; ++q) {
            const float2* sq = &sh.sw[le][6 * q];
            const float2* gg = &sh.g[le][(q * NN + a) * 3];
            const float2 gx = gg[0], gy = gg[1], gz = gg[2];
            df_fma(f0, sq[0], gx);
            df_fma(f0, sq[3], gy);
            df_fma(f0, sq[4], gz);
            df_fma(f1, sq[3], gx);
            df_fma(f1, sq[1], gy);
            df_fma(f1, sq[5], gz);
            df_fma(f2, sq[4], gx);
            df_fma(f2, sq[5], gy);
            df_fma(f2, sq[2], gz);
        }
        double* o = ye + (int64_t)e * ND + 3 * a;
        o[0] = df_value_sel(f0, intConv);
        o[1] = df_value_sel(f1, intConv);
        o[2] = df_value_sel(f2, intConv);
    }
}

// The same product for elements with 8 Gauss points (TPE = 8 threads per element, a thread per
// Gauss point) without the per-element geometry and stress stages in shared memory (which held
// occupancy near a third): the Gauss-point thread keeps its stress, and for each node a forms
// its term sigma_q . g_qa (geometry re-read from L1) as a double-float value; the 8 threads of
// the element sum the terms by an xor butterfly of double-float additions (TwoSum of the high
// parts: its error term is exact, so both partners of a pair get the same sum and every lane
// ends with the same bits), and thread a keeps node a's result.  Only x is staged.
__device__ __forceinline__ DF df_add(DF a, DF b) {
    const float s = __fadd_rn(a.hi, b.hi);
    const float bv = __fsub_rn(s, a.hi);
    const float err = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bv)), __fsub_rn(b.hi, bv));
    return DF{s, __fadd_rn(__fadd_rn(a.lo, b.lo), err)};
}
__device__ __forceinline__ DF df_shfl_xor8(DF v, int o) {
    return DF{__shfl_xor_sync(0xffffffffu, v.hi, o, 8), __shfl_xor_sync(0xffffffffu, v.lo, o, 8)};
}

template <int NN>
__global__ void __launch_bounds__(kBlock) small_strain_apply_df8_kernel(int nEl, const int32_t* __restrict__ nodeDof,
                                                                        const float2* __restrict__ geoS,
                                                                        const double* __restrict__ x,
                                                                        const double* __restrict__ tang,
                                                                        double* __restrict__ ye, int intConv) {
    constexpr int NQ = 8, TPE = 8, EPB = kBlock / TPE;
    constexpr int ND = 3 * NN;
    constexpr int NG = 3 * NN + 1;
    __shared__ float2 xv[EPB][ND + 1];
    const int tid = threadIdx.x;
    const int le = tid / TPE;
    const int q = tid % TPE;
    const int e0 = blockIdx.x * EPB + le;
    const bool valid = e0 < nEl;
    const int e = valid ? e0 : nEl - 1;  // the last element's lanes keep the shuffles full
    for (int a = q; a < NN; a += TPE) {
        const int d = nodeDof[(int64_t)e * NN + a];
        xv[le][3 * a + 0] = df_split_sel(x[d + 0], intConv);
        xv[le][3 * a + 1] = df_split_sel(x[d + 1], intConv);
        xv[le][3 * a + 2] = df_split_sel(x[d + 2], intConv);
    }
    __syncthreads();
    const float2* gq = geoS + ((int64_t)e * NQ + q) * NG;
    DF H[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) H[i][j] = DF{0.f, 0.f};
#pragma unroll 4
    for (int a = 0; a < NN; ++a) {
        float2 ga[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) ga[c] = gq[3 * a + c];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float2 u = xv[le][3 * a + i];
#pragma unroll
            for (int j = 0; j < 3; ++j) df_fma(H[i][j], u, ga[j]);
        }
    }
    const double ep[6] = {df_value_sel(H[0][0], intConv), df_value_sel(H[1][1], intConv),
                          df_value_sel(H[2][2], intConv),
                          df_value_sel(H[0][1], intConv) + df_value_sel(H[1][0], intConv),
                          df_value_sel(H[0][2], intConv) + df_value_sel(H[2][0], intConv),
                          df_value_sel(H[1][2], intConv) + df_value_sel(H[2][1], intConv)};
    const int64_t nQPtot = (int64_t)nEl * NQ;
    const int64_t qi = (int64_t)e * NQ + q;
    const double lt = tang[qi], mt = tang[nQPtot + qi], c1 = tang[2 * nQPtot + qi];
    const double tr = ep[0] + ep[1] + ep[2];
    double ne = 0.0, n[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) n[i] = 0.0;
    if (c1 != 0.0) {
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            n[i] = tang[(3 + i) * nQPtot + qi];
            ne += n[i] * ep[i];
        }
    }
    float2 sw[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) sw[i] = df_split_sel(lt * tr + 2.0 * mt * ep[i] - c1 * n[i] * ne, intConv);
#pragma unroll
    for (int i = 3; i < 6; ++i) sw[i] = df_split_sel(mt * ep[i] - c1 * n[i] * ne, intConv);
    DF own0{0.f, 0.f}, own1{0.f, 0.f}, own2{0.f, 0.f};
#pragma unroll 2
    for (int a = 0; a < NN; ++a) {
        const float2 gx = gq[3 * a + 0], gy = gq[3 * a + 1], gz = gq[3 * a + 2];
        DF f0{0.f, 0.f}, f1{0.f, 0.f}, f2{0.f, 0.f};
        df_fma(f0, sw[0], gx);
        df_fma(f0, sw[3], gy);
        df_fma(f0, sw[4], gz);
        df_fma(f1, sw[3], gx);
        df_fma(f1, sw[1], gy);
        df_fma(f1, sw[5], gz);
        df_fma(f2, sw[4], gx);
        df_fma(f2, sw[5], gy);
        df_fma(f2, sw[2], gz);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            f0 = df_add(f0, df_shfl_xor8(f0, o));
            f1 = df_add(f1, df_shfl_xor8(f1, o));
            f2 = df_add(f2, df_shfl_xor8(f2, o));
        }
        if ((a & (TPE - 1)) == q) {
            own0 = f0;
            own1 = f1;
            own2 = f2;
        }
        if ((a & (TPE - 1)) == TPE - 1 || a == NN - 1) {
            const int ao = (a & ~(TPE - 1)) + q;  // the node this lane owns in this group of 8
            if (valid && ao <= a) {
                double* o = ye + (int64_t)e * ND + 3 * ao;
                o[0] = df_value_sel(own0, intConv);
                o[1] = df_value_sel(own1, intConv);
                o[2] = df_value_sel(own2, intConv);
            }
        }
    }
}

// Consistent body force of a constant load vector (element.py:348-371): Pe[a,c] = load_c sum_q N_qa detJ_q w_q
template <int NN, int NQ>
__global__ void body_force_kernel(const ElemTables* __restrict__ T, int nEl, const double* __restrict__ geo,
                                  double l0, double l1, double l2, double* __restrict__ Pe) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nEl) return;
    constexpr int NG = 3 * NN + 1;
    double acc[NN];
    for (int a = 0; a < NN; ++a) acc[a] = 0.0;
    for (int q = 0; q < NQ; ++q) {
        const double wdet = geo[((int64_t)e * NQ + q) * NG + 3 * NN];
        for (int a = 0; a < NN; ++a) acc[a] += T->N[q][a] * wdet;
    }
    for (int a = 0; a < NN; ++a) {
        Pe[(int64_t)e * 3 * NN + 3 * a + 0] = l0 * acc[a];
        Pe[(int64_t)e * 3 * NN + 3 * a + 1] = l1 * acc[a];
        Pe[(int64_t)e * 3 * NN + 3 * a + 2] = l2 * acc[a];
    }
}

template <int NN, int NQ, typename KT, int MAT>
static ef_status launch_ss(const Group& g, const double* dU, void* K, int vij, double* Pe, double* tang, int* flags,
                           cudaStream_t s) {
    constexpr int EPB = SSShared<NN, NQ, KT>::EPB;
    const int grid = (g.nEl + EPB - 1) / EPB;
    PropsArg pa;
    for (int i = 0; i < 8; ++i) pa.v[i] = g.props[i];
    pa.cutback = g.cutback;
    const double* sIn = g.state[g.cur];
    double* sOut = g.state[1 - g.cur];
    if (grid == 0) return EF_OK;
    if (!g.geoS) {
        ef_set_error("small-strain kernel: split geometry cache missing");
        return EF_ERR_STATE;
    }
    const size_t smem = sizeof(SSShared<NN, NQ, KT>);
    if (vij) {
        auto k = small_strain_kernel<NN, NQ, KT, MAT, true>;
        EF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<grid, SSShared<NN, NQ, KT>::BLOCK, smem, ef::counted(s)>>>(g.nEl, g.nodeDof, g.geoS, g.geo, dU, sIn, sOut, pa,
                                                                       g.propsTable, g.elemRow, (KT*)K, Pe, tang, flags,
                                                                       g.intConv);
    } else {
        auto k = small_strain_kernel<NN, NQ, KT, MAT, false>;
        EF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<grid, SSShared<NN, NQ, KT>::BLOCK, smem, ef::counted(s)>>>(g.nEl, g.nodeDof, g.geoS, g.geo, dU, sIn, sOut, pa,
                                                                       g.propsTable, g.elemRow, (KT*)K, Pe, tang, flags,
                                                                       g.intConv);
    }
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

template <int NN, int NQ>
static ef_status dispatch_ss(const Group& g, const double* dU, void* K, int kDouble, int vij, double* Pe,
                             double* tang, int* flags, cudaStream_t s) {
    if (g.mat == MAT_VON_MISES)
        return kDouble ? launch_ss<NN, NQ, double, MAT_VON_MISES>(g, dU, K, vij, Pe, tang, flags, s)
                       : launch_ss<NN, NQ, float, MAT_VON_MISES>(g, dU, K, vij, Pe, tang, flags, s);
    if (g.mat == MAT_LINEAR_ELASTIC)
        return kDouble ? launch_ss<NN, NQ, double, MAT_LINEAR_ELASTIC>(g, dU, K, vij, Pe, tang, flags, s)
                       : launch_ss<NN, NQ, float, MAT_LINEAR_ELASTIC>(g, dU, K, vij, Pe, tang, flags, s);
    ef_set_error("material not available for small-strain elements");
    return EF_ERR_ARG;
}

template <int NN, int NQ>
static ef_status launch_apply(const Group& g, const double* x, const double* tang, double* ye, cudaStream_t s) {
    constexpr int EPB = ApplyShared<NN, NQ>::EPB;
    const int grid = (g.nEl + EPB - 1) / EPB;
    if (grid == 0) return EF_OK;
    static const bool fp64 = [] {
        const char* e = getenv("EF_APPLY_FP64");
        return e && atoi(e) != 0;
    }();
    static const bool staged = [] {
        const char* e = getenv("EF_APPLY_STAGED");
        return e && atoi(e) != 0;
    }();
    if (g.geoS && !fp64 && NQ == 8 && !staged) {  // 8 Gauss points: the butterfly form (EF_APPLY_STAGED=1: staged)
        small_strain_apply_df8_kernel<NN><<<(g.nEl + kBlock / 8 - 1) / (kBlock / 8), kBlock, 0, ef::counted(s)>>>(
            g.nEl, g.nodeDof, g.geoS, x, tang, ye, g.intConv);
        EF_CUDA(cudaGetLastError());
        return EF_OK;
    }
    if (g.geoS && !fp64) {  // double-float contractions (default); EF_APPLY_FP64=1: the FP64 kernel
        const size_t smemDF = sizeof(ApplyDFShared<NN, NQ>);
        auto kd = small_strain_apply_df_kernel<NN, NQ>;
        EF_CUDA(cudaFuncSetAttribute(kd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemDF));
        kd<<<grid, kBlock, smemDF, ef::counted(s)>>>(g.nEl, g.nodeDof, g.geoS, x, tang, ye, g.intConv);
        EF_CUDA(cudaGetLastError());
        return EF_OK;
    }
    const size_t smem = sizeof(ApplyShared<NN, NQ>);
    auto k = small_strain_apply_kernel<NN, NQ>;
    EF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<grid, kBlock, smem, ef::counted(s)>>>(g.nEl, g.nodeDof, g.geo, x, tang, ye);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

template <int NN, int NQ>
static ef_status launch_geometry(const Group& g, const ElemTables* T, const double* X, int* flags, cudaStream_t s) {
    const int64_t n = (int64_t)g.nEl * NQ;
    if (n == 0) return EF_OK;
    geometry_kernel<NN, NQ><<<(int)((n + 127) / 128), 128, 0, ef::counted(s)>>>(T, g.nEl, g.nodeDof, X, g.geo, g.geoS,
                                                                              flags);
    EF_CUDA(cudaGetLastError());
    return EF_OK;
}

}  // namespace ef

using namespace ef;

#define EF_FOR_TYPES(M) M(8, 8) M(8, 1) M(8, 27) M(20, 27) M(20, 8)

ef_status ef_launch_geometry(const Group& g, const ElemTables* T, const double* X, int* flags, cudaStream_t s) {
#define EF_G(NN_, NQ_) \
    if (g.nNodes == NN_ && g.nQP == NQ_) return launch_geometry<NN_, NQ_>(g, T, X, flags, s);
    EF_FOR_TYPES(EF_G)
#undef EF_G
    ef_set_error("unsupported element type");
    return EF_ERR_ARG;
}

ef_status ef_launch_small_strain(const Group& g, const double* dU, void* Kout, int kDouble, int kLayoutVIJ,
                                 double* Pe, double* tang, int* flags, cudaStream_t s) {
#define EF_SS(NN_, NQ_) \
    if (g.nNodes == NN_ && g.nQP == NQ_) return dispatch_ss<NN_, NQ_>(g, dU, Kout, kDouble, kLayoutVIJ, Pe, tang, flags, s);
    EF_FOR_TYPES(EF_SS)
#undef EF_SS
    ef_set_error("unsupported element type for the small-strain kernel");
    return EF_ERR_ARG;
}

ef_status ef_launch_small_strain_apply(const Group& g, const double* x, const double* tang, double* ye,
                                       cudaStream_t s) {
#define EF_AP(NN_, NQ_) \
    if (g.nNodes == NN_ && g.nQP == NQ_) return launch_apply<NN_, NQ_>(g, x, tang, ye, s);
    EF_FOR_TYPES(EF_AP)
#undef EF_AP
    ef_set_error("unsupported element type for the tangent apply");
    return EF_ERR_ARG;
}

ef_status ef_launch_body_force(const Group& g, const ElemTables* T, const double load[3], double* Pe, cudaStream_t s) {
    const int grid = (g.nEl + 127) / 128;
    if (grid == 0) return EF_OK;
#define EF_BF(NN_, NQ_)                                                                                   \
    if (g.nNodes == NN_ && g.nQP == NQ_) {                                                               \
        body_force_kernel<NN_, NQ_><<<grid, 128, 0, ef::counted(s)>>>(T, g.nEl, g.geo, load[0], load[1], load[2], Pe); \
        EF_CUDA(cudaGetLastError());                                                                     \
        return EF_OK;                                                                                    \
    }
    EF_FOR_TYPES(EF_BF)
#undef EF_BF
    ef_set_error("unsupported element type for body forces");
    return EF_ERR_ARG;
}
