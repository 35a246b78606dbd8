// Device helpers of the PCG kernels (krylov.cu, batch.cu): distributed shared memory of a thread-block cluster,
// and the product of a 3x3 block row with lanes side by side.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ef {

__device__ __forceinline__ unsigned cluster_size() {
    unsigned v;
    asm("mov.u32 %0, %%cluster_nctaid.x;\n" : "=r"(v));
    return v;
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned v;
    asm("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(v));
    return v;
}
// the address of a shared-memory variable of this CTA in CTA `rank` of its cluster
__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_store(unsigned a, unsigned long long u, unsigned long long v) {
    asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};\n" ::"r"(a), "l"(u), "l"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(unsigned a, unsigned u) {
    asm volatile("st.shared::cluster.b32 [%0], %1;\n" ::"r"(a), "r"(u) : "memory");
}
__device__ __forceinline__ float cluster_load(unsigned a, float) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double cluster_load(unsigned a, double) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];\n" : "=d"(v) : "r"(a) : "memory");
    return v;
}
// every thread of every CTA of the cluster; what they wrote before it is visible behind it
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}

// y += A p of one block as chains of fused multiply-adds (written as a sum of products it is four FP64
// instructions a row instead of three)
template <typename VT>
__device__ __forceinline__ void block_fma(const VT* v, VT p0, VT p1, VT p2, VT& y0, VT& y1, VT& y2) {
    y0 = fma(v[2], p2, fma(v[1], p1, fma(v[0], p0, y0)));
    y1 = fma(v[5], p2, fma(v[4], p1, fma(v[3], p0, y1)));
    y2 = fma(v[8], p2, fma(v[7], p1, fma(v[6], p0, y2)));
}

// Component c of (y0, y1, y2) summed over the LPR lanes of a row, in the lanes whose top two bits of
// the group lane are c (c = 3: none).  The first two steps exchange components instead of summing all three in
// every lane: 3 adds and one per further step against 3 per step.
template <int LPR, typename VT>
__device__ __forceinline__ VT row_sum3(int l, VT y0, VT y1, VT y2) {
    const bool hi = (l & (LPR / 2)) != 0, lo = (l & (LPR / 4)) != 0;
    VT k0 = hi ? y2 : y0, k1 = hi ? (VT)0 : y1;
    k0 += __shfl_xor_sync(0xffffffffu, hi ? y0 : y2, LPR / 2);
    k1 += __shfl_xor_sync(0xffffffffu, hi ? y1 : (VT)0, LPR / 2);
    VT k = lo ? k1 : k0;
    k += __shfl_xor_sync(0xffffffffu, lo ? k0 : k1, LPR / 4);
#pragma unroll
    for (int o = LPR / 8; o > 0; o >>= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
    return k;
}

}  // namespace ef
