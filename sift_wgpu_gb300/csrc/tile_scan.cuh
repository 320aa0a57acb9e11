// tile_scan.cuh — block-wide sums for the ordered lists.
//
// A list's items (mask words, candidate slots) are cut into tiles, and the
// kernel that produces them counts each tile's output items as it goes
// (integer atomics, so the counts do not depend on scheduling). A block of the
// kernel that writes the list then knows its tile's first position from the
// counts of the tiles before it alone: no pass in between, no block waits for
// another.
#pragma once
#include "sift_internal.cuh"

namespace sift {

// The block's sum of one value per thread, in every thread. It synchronises
// the block (also before, so that buf may be read from the last call).
template <int kThreads>
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* buf) {
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) s += buf[w];
    return s;
}

// The sum of the values of the threads before this one.
template <int kThreads>
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* buf) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    __syncthreads();
    if (lane == 31) buf[warp] = x;
    __syncthreads();
    uint32_t r = x - v;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) r += w < warp ? buf[w] : 0u;
    return r;
}

// The counts of tiles from .. to - 1, summed over the block.
template <int kThreads>
__device__ __forceinline__ uint32_t tiles_sum(const uint32_t* __restrict__ tiles, uint32_t from, uint32_t to,
                                              uint32_t* buf) {
    uint32_t part = 0;
#pragma unroll 4
    for (uint32_t i = from + threadIdx.x; i < to; i += kThreads) part += tiles[i];
    return block_sum<kThreads>(part, buf);
}

}  // namespace sift
