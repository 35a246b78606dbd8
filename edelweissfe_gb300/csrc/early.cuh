// Loads that a dependent launch (launch_dep) issues before it waits for the kernel ahead of it.
#pragma once

#include <stdint.h>

namespace ef {

// Loads of matrix values and indices ahead of griddepcontrol.wait: a cycle's small kernels are chains of a few
// dependent loads (row pointer, index, value, vector), and only the vector comes from the kernel before.  The
// matrices are set-up results, and the kernel launched just before one of these never writes them (the rule at
// launch_dep): it is one of the cycle or of the Krylov iteration, or in the power iteration the norm or the scaling of its
// vector.  Volatile, so that they stay ahead of the wait.  us of the
// cycle before and now: 7,412 nodes of quadratic elements 25.3 -> 23.2, hex8 4,225 nodes 19.3 -> 17.2, 11,849 nodes 27.7 ->
// 23.5, 18,081 nodes 30.0 -> 25.5, 169,781 nodes 78.1 -> 71.3.
__device__ __forceinline__ int early(const int32_t* p) {
    int v;
    asm volatile("ld.global.nc.s32 %0, [%1];\n" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t early(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.u32 %0, [%1];\n" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float early(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];\n" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 early(const float2* p) {
    float2 v;
    asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 early(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// values that are read once (evicted first)
__device__ __forceinline__ float early_cs(const float* p) {
    float v;
    asm volatile("ld.global.cs.f32 %0, [%1];\n" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int early_cs(const int32_t* p) {
    int v;
    asm volatile("ld.global.cs.s32 %0, [%1];\n" : "=r"(v) : "l"(p));
    return v;
}
}  // namespace ef
