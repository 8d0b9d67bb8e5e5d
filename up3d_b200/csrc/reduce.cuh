// Sums over a vector in an order fixed by its length: the dot products of
// the Krylov solvers (krylov.cu) and of the allocation-free CG (noalloc.cu).
//
// dot_grid(n) blocks of DOT_BLOCK threads stride the vector; each block's
// sum goes to its partial, and one block adds the partials.  A block per
// 1024 values: a fixed 592 blocks left most of them idle on small systems
// and the last block 592 partials to add with one warp (8 us a dot at 5 k
// rows, 9.6 us at 625 k).
#pragma once

#include "internal.cuh"

namespace up3d {

constexpr int DOT_BLOCK = 256, DOT_MAX_BLOCKS = 592;
inline unsigned dot_grid(int64_t n) { return grid_for(n, 1024, DOT_MAX_BLOCKS); }

// Sum of v over the block's threads, in thread 0 (warp butterflies, then
// the warp sums in order).  sh: DOT_BLOCK / 32 values; every thread calls.
__device__ __forceinline__ double block_sum(double v, double* sh) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < DOT_BLOCK / 32; ++q) t += sh[q];
    __syncthreads();
    return t;
}

// The sum of nb block partials, in thread 0 of the calling block.
__device__ __forceinline__ double sum_partials(const double* partial, int nb, double* sh) {
    double v = 0.0;
    for (int b = threadIdx.x; b < nb; b += DOT_BLOCK) v += __ldcg(partial + b);
    return block_sum(v, sh);
}

// Called by every thread of every block once the block's partials are
// written: true in the last block to arrive, which then sees them all and
// must re-arm the counter (*counter = 0) for the next launch on the stream.
__device__ __forceinline__ bool last_block(unsigned int* counter) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (last) __threadfence();
    return last;
}

}  // namespace up3d
