// export.cu — a run's exchange with the host: its first and its last kernel.
//
// k_begin starts a run: it copies the run's cell (RunCell: where the image is,
// where the results go) from mapped host memory to device memory and zeroes
// the counters and the tile counts. It takes the place of two memset nodes of
// the graph (a 160 x 120 frame 176 -> 162 us); launched ahead of the graph
// with the cell as a parameter the frame took 174 us.
//
// k_fetch brings a pageable image into the engine's device copy, straight
// from the caller's buffer, ahead of the graph, so that it runs while the
// host still launches the graph. The host link is the limit: 16-byte loads of
// pageable memory by the SMs reach 200 GB/s at any grid of one CTA per SM or
// more (2 MB in 15 us, 17 MB in 86 us; cudaMemcpyAsync of the same memory
// takes 23 and 103 us). The base level's own reads over the link, which fetch
// a tile's halo too, took 252 us at 4096 x 4096.
//
// k_export ends a run: the host does not know the keypoint count of a run
// before it finishes, so a copy engine cannot be told how much to move; this
// kernel reads the count on the device and moves the counters and
// min(count, cap) keypoints over the host link in one launch. (The descriptor
// stage writes descriptors below cap into the same buffer itself,
// describe.cu.) The host then needs one synchronisation per call instead of a
// counter read followed by a sized copy.
#include <algorithm>

#include "sift_internal.cuh"

namespace sift {
namespace {

constexpr int kBeginThreads = 256;

// 16 bytes from p, which may start anywhere: the aligned words that hold
// bytes p .. p + n - 1 (n <= 16), and no others, are read.
__device__ __forceinline__ uint4 load16(const uint8_t* p, int n) {
    const int sh = (int)((uintptr_t)p & 15);
    const ulonglong2* w = reinterpret_cast<const ulonglong2*>(p - sh);
    const ulonglong2 a = w[0];
    if (sh == 0) return make_uint4((unsigned)a.x, (unsigned)(a.x >> 32), (unsigned)a.y, (unsigned)(a.y >> 32));
    ulonglong2 b = make_ulonglong2(0ull, 0ull);
    if (sh + n > 16) b = w[1];
    unsigned long long q0 = a.x, q1 = a.y, q2 = b.x;
    if (sh >= 8) {
        q0 = a.y;
        q1 = b.x;
        q2 = b.y;
    }
    const int s = (sh & 7) * 8;
    if (s) {
        q0 = q0 >> s | q1 << (64 - s);
        q1 = q1 >> s | q2 << (64 - s);
    }
    return make_uint4((unsigned)q0, (unsigned)(q0 >> 32), (unsigned)q1, (unsigned)(q1 >> 32));
}

// One CTA. The cell is read past the caches: the host rewrites it between runs.
__global__ void __launch_bounds__(kBeginThreads) k_begin(const RunCell* hcell, RunCell* __restrict__ cell,
                                                         Counters* __restrict__ ctr,
                                                         uint32_t* __restrict__ tiles, uint32_t n_tiles) {
    chain_wait();
    const int tid = threadIdx.x;
    constexpr int kWords = sizeof(RunCell) / 4;
    uint32_t v = 0;
    if (tid < kWords) v = __ldcv(reinterpret_cast<const uint32_t*>(hcell) + tid);
    for (uint32_t i = tid; i < sizeof(Counters) / 4; i += kBeginThreads) reinterpret_cast<uint32_t*>(ctr)[i] = 0u;
    // (an allocation of whole 16-byte words)
    for (uint32_t i = tid; i < (n_tiles + 3) / 4; i += kBeginThreads)
        reinterpret_cast<uint4*>(tiles)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (tid < kWords) reinterpret_cast<uint32_t*>(cell)[tid] = v;
}

// The image rows, 16 bytes per thread and step, to a device copy whose rows
// start on 128 bytes (the last word of a row may end in its padding).
__global__ void __launch_bounds__(kBeginThreads) k_fetch(const uint8_t* __restrict__ src, long long stride,
                                                         uint8_t* __restrict__ img, long long pitch, int W, int H) {
    chain_wait();
    const uint32_t cw = (uint32_t)(W + 15) / 16, total = cw * (uint32_t)H;
    const uint32_t step = gridDim.x * kBeginThreads;
    constexpr int kU = 4;
    for (uint32_t i0 = blockIdx.x * kBeginThreads + threadIdx.x; i0 < total; i0 += kU * step) {
        uint4 v[kU];
        uint32_t y[kU], x[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const uint32_t i = i0 + u * step;
            y[u] = i / cw;
            x[u] = 16u * (i - y[u] * cw);
            if (i < total) v[u] = load16(src + (long long)y[u] * stride + x[u], min(16, W - (int)x[u]));
        }
#pragma unroll
        for (int u = 0; u < kU; ++u)
            if (i0 + u * step < total) *reinterpret_cast<uint4*>(img + (long long)y[u] * pitch + x[u]) = v[u];
    }
}

__global__ void __launch_bounds__(256) k_export(const Counters* __restrict__ ctr, const Keypoint* __restrict__ kps,
                                                const RunCell* __restrict__ cell) {
    chain_wait();
    Counters* hctr = cell->ctr;
    Keypoint* hkps = cell->kps;
    const uint32_t n = min(ctr->n_oriented, cell->cap);
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    constexpr uint32_t kCtrWords = sizeof(Counters) / 4;
    if (tid < kCtrWords) reinterpret_cast<uint32_t*>(hctr)[tid] = reinterpret_cast<const uint32_t*>(ctr)[tid];
    const size_t kw = (size_t)n * (sizeof(Keypoint) / 4);
    for (size_t i = tid; i < kw; i += stride)
        reinterpret_cast<uint32_t*>(hkps)[i] = reinterpret_cast<const uint32_t*>(kps)[i];
}

}  // namespace

int launch_begin(const RunCell* hcell, RunCell* cell, Counters* ctr, uint32_t* tiles, size_t n_tiles, cudaStream_t st) {
    if (launch_chained(k_begin, 1, kBeginThreads, 0, st, hcell, cell, ctr, tiles, (uint32_t)n_tiles) != cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

int launch_fetch(const uint8_t* src, long long stride, uint8_t* img, long long pitch, int W, int H, cudaStream_t st) {
    // a thread's share is at least one 16-byte word; two CTAs per SM saturate the link
    const long long words = (long long)((W + 15) / 16) * H;
    if (words <= 0) return 0;
    const unsigned grid = (unsigned)std::min<long long>((words + kBeginThreads - 1) / kBeginThreads, 2 * 152);
    if (launch_chained(k_fetch, grid, kBeginThreads, 0, st, src, stride, img, pitch, W, H) != cudaSuccess) return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

int launch_export(const Counters* ctr, const Keypoint* kps, const RunCell* cell, cudaStream_t st) {
    if (launch_chained(k_export, 152, 256, 0, st, ctr, kps, cell) != cudaSuccess) return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace sift
