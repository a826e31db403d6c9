// Deterministic block/grid reductions (FP64 accumulation).
#pragma once
#include <cuda_runtime.h>

namespace eqc {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the CTA; result valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double* sh) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    v = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
    if (w == 0) v = warp_sum(v);
    __syncthreads();
    return v;
}

// Sum of a dot-product accumulator (DotAcc) over the CTA (up to 1,024 threads); valid in warp 0's lane 0.
template <class Acc>
__device__ __forceinline__ void block_sum(Acc& acc) {
    __shared__ typename Acc::Part sh[32];
    acc.warp_sum();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) sh[w] = acc.part();
    __syncthreads();
    if (w == 0) {
        acc = Acc();
        if (lane < nw) acc.merge(sh[lane]);
        acc.warp_sum(nw);
    }
    __syncthreads();
}

// Finishes a reduction over the grid: every CTA stores its partial, the last one to do so (an atomic
// ticket) sums them, one per thread where there are threads enough, in an order that depends on the
// grid only, and calls fin(total) in thread 0.  part: 16 bytes per CTA.
template <class Acc, class Fin>
__device__ __forceinline__ void grid_sum(Acc acc, double* part, unsigned* count, Fin fin) {
    __shared__ bool last;
    using Part = typename Acc::Part;
    Part* p = reinterpret_cast<Part*>(part);
    const unsigned nblk = gridDim.x * gridDim.y;
    block_sum(acc);
    if (threadIdx.x == 0) {
        p[blockIdx.y * gridDim.x + blockIdx.x] = acc.part();
        __threadfence();
        const unsigned prev = atomicAdd(count, 1u);
        last = (prev == nblk - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    acc = Acc();
    for (unsigned k = threadIdx.x; k < nblk; k += blockDim.x) acc.merge(__ldcg(p + k));
    block_sum(acc);
    if (threadIdx.x == 0) {
        fin(acc.value());
        *count = 0u;
    }
}

}  // namespace eqc
