// Deterministic block/grid reductions (FP64 accumulation).
#pragma once
#include <cuda_runtime.h>

namespace eqc {

constexpr int SUM_THREADS = 256;   // the largest CTA that sums

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Sum of one number per thread over the CTA (whole warps, at most SUM_THREADS threads); valid in thread 0.
// An FP64 instruction of a warp holds its SM's FP64 pipe for 16 clocks, so one warp adds what every thread
// leaves in shared memory, 12 instructions to a CTA where sums of each warp first take 45.
__device__ __forceinline__ double cta_sum(double v) {
    __shared__ double sh[SUM_THREADS];
    sh[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t[SUM_THREADS / 32];
#pragma unroll
        for (int q = 0; q < SUM_THREADS / 32; ++q) t[q] = 32 * q < blockDim.x ? sh[32 * q + threadIdx.x] : 0.0;
#pragma unroll
        for (int h = SUM_THREADS / 64; h > 0; h >>= 1)
#pragma unroll
            for (int q = 0; q < h; ++q) t[q] += t[q + h];
        v = warp_sum(t[0]);
    }
    __syncthreads();
    return v;
}

// Finishes a reduction (DotAcc) over the grid: every CTA stores its partial, the last one to do so (an atomic
// ticket) sums them, one per thread where there are threads enough, in an order that depends on the
// grid only, and calls fin(total) in thread 0.  part: one entry per CTA.
template <class Acc, class Fin>
__device__ __forceinline__ void grid_sum(const Acc& acc, double* part, unsigned* count, Fin fin) {
    __shared__ bool last;
    const unsigned nblk = gridDim.x * gridDim.y;
    const double s = cta_sum(acc.value());
    if (threadIdx.x == 0) {
        part[blockIdx.y * gridDim.x + blockIdx.x] = s;
        __threadfence();
        const unsigned prev = atomicAdd(count, 1u);
        last = (prev == nblk - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    for (unsigned k = threadIdx.x; k < nblk; k += blockDim.x) t += __ldcg(part + k);
    t = cta_sum(t);
    if (threadIdx.x == 0) {
        fin(t);
        *count = 0u;
    }
}

}  // namespace eqc
