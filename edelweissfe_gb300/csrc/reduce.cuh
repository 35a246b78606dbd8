// Sums and maxima of a launch's values in one launch, in a fixed order.
//
// Every CTA combines its threads' values (one warp: a warp's FP64 instruction takes this GPU's narrow pipe
// 16 cycles, so the other warps add nothing) and stores the result; the last CTA to arrive, by an atomic
// ticket that nobody waits for, combines the CTAs' results in CTA order.  The two-launch form, whose
// second kernel added the CTAs' results in one thread, spent 14-20 us there (one dependent load and
// addition after another), and the Newton check's 60.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ef {

constexpr int kRedThreads = 256;

template <int NV, unsigned MAXMASK>
struct RedOp {  // value j: the maximum where bit j of MAXMASK is set, else the sum
    static __device__ __forceinline__ double apply(int j, double a, double b) {
        return (MAXMASK >> j) & 1u ? fmax(a, b) : a + b;
    }
};

template <int NV, unsigned MAXMASK>
__device__ __forceinline__ void cta_reduce(double (&v)[NV], double (*red)[kRedThreads]) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int j = 0; j < NV; ++j) red[j][tid] = v[j];
    __syncthreads();
    if (tid < 32) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            double t = red[j][tid];
#pragma unroll
            for (int i = 1; i < kRedThreads / 32; ++i) t = RedOp<NV, MAXMASK>::apply(j, t, red[j][tid + 32 * i]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t = RedOp<NV, MAXMASK>::apply(j, t, __shfl_xor_sync(0xffffffffu, t, o));
            v[j] = t;
        }
    }
}

// All CTAs of kRedThreads threads call it; true in one thread of the launch, whose v then holds the result.
// part: [NV * gridDim.x]; *ticket: 0 between launches.  Sums start at 0 and maxima are of absolute values, so
// a thread without values passes 0.
template <int NV, unsigned MAXMASK>
__device__ __forceinline__ bool grid_reduce(double (&v)[NV], double* part, unsigned* ticket) {
    __shared__ double red[NV][kRedThreads];
    __shared__ bool last;
    cta_reduce<NV, MAXMASK>(v, red);
    if (gridDim.x == 1) return threadIdx.x == 0;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) part[NV * blockIdx.x + j] = v[j];
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = 0.0;
    for (unsigned c = threadIdx.x; c < gridDim.x; c += kRedThreads)
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j] = RedOp<NV, MAXMASK>::apply(j, v[j], __ldcg(part + NV * c + j));
    cta_reduce<NV, MAXMASK>(v, red);
    if (threadIdx.x == 0) *ticket = 0u;
    return threadIdx.x == 0;
}

// CTAs of a reduction over n values: four a thread, up to `most`
inline int reduce_grid(int64_t n, int most) {
    const int64_t g = (n + 4 * kRedThreads - 1) / (4 * kRedThreads);
    return (int)(g < 1 ? 1 : (g > most ? most : g));
}

}  // namespace ef
