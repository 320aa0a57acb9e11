// pyramid.cu — Gaussian pyramid kernels (sm_103a).
//
// Stage (a) of the hot path: generate_gaussian_pyramid and
// generate_dog_pyramid (src/sift.rs:129-204), with the base blur of
// detect_and_compute_cpu (src/sift.rs:1200-1214). The levels are
// reference-compatible: each separable blur pass and the Lanczos3 resize end
// in u8 values exactly as the reference's GrayImage levels do, so every level
// is bit-identical to the CPU path, and so is every DoG value the detection
// forms from them. Products and sums are rounded one by one
// (__fmul_rn/__fadd_rn) in the reference's tap order.
//
// Every level is written as its u8 plane (1 byte/pixel, what the next level,
// the resize and every later stage read; DoG is formed from it where it is
// read, never stored) and, in the f32 and f16 storage modes, also in that
// type (f32 v/255 or f16 v, which only a copied level reads again); the
// default u8 storage writes the u8 plane alone.
//
// Kernels
//   k_blur_level   both separable passes of a level for r <= 28 on the tensor
//                  cores (level_tc.cuh), bit for bit the sequential sums.
//   k_blur_rows    horizontal pass for larger radii, one row per CTA. u8 out.
//   k_blur_cols    vertical pass for larger radii on a 32 x 64 tile.
//   k_lanczos_fused  the 2x Lanczos3 resize between octaves, both passes.
// The base level of a host call reads its image through an ImgRef cell (the
// engine's device copy, or the caller's pageable buffer in place).
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "level_tc.cuh"
#include "sift_internal.cuh"
#include "tables.h"

namespace sift {
namespace {

// v / 255 in f32, the IEEE quotient the reference computes (div255: a
// multiply and one fused correction, exact for every u8 value).
__device__ __forceinline__ float norm255(int v) { return div255((float)v); }

// Level storage: f32 holds v/255 (the reference's convert_u8_to_f32_gray
// value, src/sift.rs:92-101), f16 holds v (v/255 is not exact in f16), u8
// storage stores nothing beyond the u8 plane.
template <typename T>
__device__ __forceinline__ void store_level(T* p, int v, float vn);
template <>
__device__ __forceinline__ void store_level<float>(float* p, int v, float vn) {
    *p = vn;
}
template <>
__device__ __forceinline__ void store_level<__half>(__half* p, int v, float) {
    *p = __int2half_rn(v);
}
// u8 storage: the level is its u8 plane, which every kernel writes anyway
template <>
__device__ __forceinline__ void store_level<uint8_t>(uint8_t*, int, float) {}

__device__ __forceinline__ void unpack16(const uint4 b, float* v) {
    const unsigned w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        v[4 * e + 0] = float_of_byte<0>(w[e]);
        v[4 * e + 1] = float_of_byte<1>(w[e]);
        v[4 * e + 2] = float_of_byte<2>(w[e]);
        v[4 * e + 3] = float_of_byte<3>(w[e]);
    }
}

// imageproc's f32 -> u8 clamp (truncation) as an int
__device__ __forceinline__ int to_u8(float a) { return int_of(clamp_u8f(a)); }

constexpr int kRowThreads = 128;

// One row per CTA. Shared layout: weights[taps] (padded to a multiple of 4),
// then the row with r clamp-to-edge pixels on each side and 8 floats of slack.
__device__ __forceinline__ void blur_row(const uint8_t* __restrict__ in, int in_pitch, uint8_t* __restrict__ out,
                                         int out_pitch, int W, int r, const float* __restrict__ wts, int y, float* sm) {
    const int taps = 2 * r + 1;
    const int wpad = (taps + 3) & ~3;
    float* kw = sm;
    float* row = sm + wpad;
    const uint8_t* src = in + (long long)y * in_pitch;
    for (int i = threadIdx.x; i < wpad; i += blockDim.x) kw[i] = i < taps ? wts[i] : 0.0f;
    const int padded = W + 2 * r;
    // Interior as 4-byte words, consecutive lanes on consecutive words: the
    // four stores of a lane land 4 floats apart from its neighbour's (4-way
    // bank sharing; 16-byte words per lane would put a warp's stores in two
    // banks).
    const int nw4 = (in_pitch & 3) == 0 ? (W >> 2) : 0;
#pragma unroll 4
    for (int k = threadIdx.x; k < nw4; k += blockDim.x) {
        const unsigned b = *reinterpret_cast<const unsigned*>(src + 4 * k);
        float* d = row + r + 4 * k;
        d[0] = float_of_byte<0>(b);
        d[1] = float_of_byte<1>(b);
        d[2] = float_of_byte<2>(b);
        d[3] = float_of_byte<3>(b);
    }
    // clamp-to-edge borders, the tail after the whole words and the slack
    const int hi0 = r + 4 * nw4, nb = r + (padded + 8 - hi0);
    for (int j = threadIdx.x; j < nb; j += blockDim.x) {
        const int jj = j < r ? j : hi0 + (j - r);
        row[jj] = float_of_u8(src[clampi(jj - r, 0, W - 1)]);
    }
    __syncthreads();
    uint8_t* dst = out + (long long)y * out_pitch;
    // Short rows: a chain for each output, not four side by side in a quarter
    // of the threads (more instructions in all: rows of 200 pixels cost the
    // other octaves' kernels of a 1600 x 900 frame more than they save, 1 %).
    if (W <= kRowThreads) {
        if (threadIdx.x >= W) return;
        const float* p = row + threadIdx.x;
        float a = 0.0f;
#pragma unroll 8
        for (int i = 0; i < taps; ++i) a = __fadd_rn(a, __fmul_rn(p[i], kw[i]));
        dst[threadIdx.x] = (uint8_t)to_u8(a);
        return;
    }
    for (int x0 = threadIdx.x * 4; x0 < W; x0 += blockDim.x * 4) {
        float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
        const float* base = row + x0;  // x0 % 4 == 0 and wpad % 4 == 0: 16-byte aligned
        float4 A = *reinterpret_cast<const float4*>(base);
        int i = 0;
        for (; i + 4 <= taps; i += 4) {
            const float4 B = *reinterpret_cast<const float4*>(base + i + 4);
            const float4 K = *reinterpret_cast<const float4*>(kw + i);
            a0 = __fadd_rn(a0, __fmul_rn(A.x, K.x));
            a1 = __fadd_rn(a1, __fmul_rn(A.y, K.x));
            a2 = __fadd_rn(a2, __fmul_rn(A.z, K.x));
            a3 = __fadd_rn(a3, __fmul_rn(A.w, K.x));
            a0 = __fadd_rn(a0, __fmul_rn(A.y, K.y));
            a1 = __fadd_rn(a1, __fmul_rn(A.z, K.y));
            a2 = __fadd_rn(a2, __fmul_rn(A.w, K.y));
            a3 = __fadd_rn(a3, __fmul_rn(B.x, K.y));
            a0 = __fadd_rn(a0, __fmul_rn(A.z, K.z));
            a1 = __fadd_rn(a1, __fmul_rn(A.w, K.z));
            a2 = __fadd_rn(a2, __fmul_rn(B.x, K.z));
            a3 = __fadd_rn(a3, __fmul_rn(B.y, K.z));
            a0 = __fadd_rn(a0, __fmul_rn(A.w, K.w));
            a1 = __fadd_rn(a1, __fmul_rn(B.x, K.w));
            a2 = __fadd_rn(a2, __fmul_rn(B.y, K.w));
            a3 = __fadd_rn(a3, __fmul_rn(B.z, K.w));
            A = B;
        }
        for (; i < taps; ++i) {
            const float k = kw[i];
            a0 = __fadd_rn(a0, __fmul_rn(base[i + 0], k));
            a1 = __fadd_rn(a1, __fmul_rn(base[i + 1], k));
            a2 = __fadd_rn(a2, __fmul_rn(base[i + 2], k));
            a3 = __fadd_rn(a3, __fmul_rn(base[i + 3], k));
        }
        const int v0 = to_u8(a0), v1 = to_u8(a1), v2 = to_u8(a2), v3 = to_u8(a3);
        if (x0 + 3 < W) {  // out_pitch is a multiple of 32 and x0 of 4: one aligned word
            *reinterpret_cast<unsigned*>(dst + x0) =
                (unsigned)v0 | ((unsigned)v1 << 8) | ((unsigned)v2 << 16) | ((unsigned)v3 << 24);
        } else {
            dst[x0] = (uint8_t)v0;
            if (x0 + 1 < W) dst[x0 + 1] = (uint8_t)v1;
            if (x0 + 2 < W) dst[x0 + 2] = (uint8_t)v2;
        }
    }
}

__global__ void __launch_bounds__(kRowThreads) k_blur_rows(const uint8_t* __restrict__ in, int in_pitch,
                                                           uint8_t* __restrict__ out, int out_pitch, int W, int r,
                                                           const float* __restrict__ wts,
                                                           const ImgRef* __restrict__ ref) {
    chain_wait();
    if (ref) {  // a host call's base level: the image is wherever the cell says
        in = ref->ptr;
        in_pitch = (int)ref->pitch;
    }
    extern __shared__ __align__(16) float sm[];
    blur_row(in, in_pitch, out, out_pitch, W, r, wts, blockIdx.x, sm);
}

constexpr int kColTX = 32;                 // output columns per CTA
constexpr int kColRows = 64;               // output rows per CTA
constexpr int kColThreads = 256;           // 8 column groups of 4 x 32 row groups of 2
constexpr int kColRowsSmall = 8;           // of a small plane: an output per thread
constexpr int kColFew = 12;                // 64-row tiles of a small plane, at most

// Vertical pass over a 32 x 64 output tile. Shared layout: weights padded
// with zeros to a multiple of 8, lut[256] (v / 255 in f32), then
// (64 + taps8 - 1) rows x 32 floats of the u8 intermediate with
// clamp-to-edge rows. Each thread owns 4 columns x 2 rows and slides a
// two-row float4 window down the taps, in unrolled groups of 8; the zero taps
// at the end add +0 to a non-negative sum, which leaves it unchanged. Writes
// level s (TG and u8) as vector stores. No DoG plane is stored: the detection
// stages form DoG(s-1) = G_s/255 - G_{s-1}/255 (src/sift.rs:92-124) from the
// u8 planes through the v / 255 table where they read it.
__host__ __device__ constexpr int taps8(int r) { return ((2 * r + 1) + 7) & ~7; }

template <typename TG>
__device__ __forceinline__ void store_level4(TG* p, const int v[4], const float* lut);
template <>
__device__ __forceinline__ void store_level4<float>(float* p, const int v[4], const float* lut) {
    *reinterpret_cast<float4*>(p) = make_float4(lut[v[0]], lut[v[1]], lut[v[2]], lut[v[3]]);
}
template <>
__device__ __forceinline__ void store_level4<uint8_t>(uint8_t*, const int*, const float*) {}
template <>
__device__ __forceinline__ void store_level4<__half>(__half* p, const int v[4], const float*) {
    const __half2 a = __halves2half2(__int2half_rn(v[0]), __int2half_rn(v[1]));
    const __half2 b = __halves2half2(__int2half_rn(v[2]), __int2half_rn(v[3]));
    uint2 u;
    u.x = *reinterpret_cast<const unsigned*>(&a);
    u.y = *reinterpret_cast<const unsigned*>(&b);
    *reinterpret_cast<uint2*>(p) = u;
}

template <typename TG, int kRows>
__device__ __forceinline__ void blur_cols_tile(const uint8_t* __restrict__ tmp, int tmp_pitch, TG* __restrict__ out,
                                               uint8_t* __restrict__ out_u8, int pitch, int W, int H, int r,
                                               const float* __restrict__ wts, const float* __restrict__ lut255,
                                               int x0, int y0, float* sm) {
    const int taps = 2 * r + 1;
    const int tp = taps8(r);
    float* kw = sm;
    float* lut = sm + tp;
    float* tile = lut + 256;
    const int tid = threadIdx.x;
    for (int i = tid; i < tp; i += kColThreads) kw[i] = i < taps ? wts[i] : 0.0f;
    for (int i = tid; i < 256; i += kColThreads) lut[i] = lut255[i];
    const int rows = kRows + tp - 1;
    if (x0 + kColTX <= W && (tmp_pitch & 15) == 0) {
        // two 16-byte loads per row, all rows of the tile in flight
#pragma unroll 4
        for (int q = tid; q < rows * 2; q += kColThreads) {
            const int k = q >> 1, h = q & 1;
            const int ys = clampi(y0 - r + k, 0, H - 1);
            float v[16];
            unpack16(*reinterpret_cast<const uint4*>(tmp + (long long)ys * tmp_pitch + x0 + 16 * h), v);
            float* d = tile + k * kColTX + 16 * h;
#pragma unroll
            for (int e = 0; e < 16; ++e) d[e] = v[e];
        }
    } else {
        const int lx = tid & (kColTX - 1);
        const int xg = min(x0 + lx, W - 1);
        for (int k = tid / kColTX; k < rows; k += kColThreads / kColTX) {
            const int ys = clampi(y0 - r + k, 0, H - 1);
            tile[k * kColTX + lx] = float_of_u8(tmp[(long long)ys * tmp_pitch + xg]);
        }
    }
    __syncthreads();
    if constexpr (kRows == kColRowsSmall) {
        const int x = x0 + (tid & (kColTX - 1)), y = y0 + tid / kColTX;
        if (x >= W || y >= H) return;
        const float* p = tile + tid;
        float a = 0.0f;
#pragma unroll 8
        for (int i = 0; i < taps; ++i) a = __fadd_rn(a, __fmul_rn(p[i * kColTX], kw[i]));
        const int v = to_u8(a);
        const long long o = (long long)y * pitch + x;
        store_level(out + o, v, lut[v]);
        out_u8[o] = (uint8_t)v;
        return;
    }
    const int cg = tid & 7, rg = tid >> 3;
    const float4* col = reinterpret_cast<const float4*>(tile) + (2 * rg) * (kColTX / 4) + cg;
    float4 a0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), a1 = a0;
    float4 w0 = col[0];
    for (int i0 = 0; i0 < tp; i0 += 8) {
        const float4 ka = *reinterpret_cast<const float4*>(kw + i0);
        const float4 kb = *reinterpret_cast<const float4*>(kw + i0 + 4);
        const float k8[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float4 w1 = col[(i0 + q + 1) * (kColTX / 4)];
            const float k = k8[q];
            a0.x = __fadd_rn(a0.x, __fmul_rn(w0.x, k));
            a0.y = __fadd_rn(a0.y, __fmul_rn(w0.y, k));
            a0.z = __fadd_rn(a0.z, __fmul_rn(w0.z, k));
            a0.w = __fadd_rn(a0.w, __fmul_rn(w0.w, k));
            a1.x = __fadd_rn(a1.x, __fmul_rn(w1.x, k));
            a1.y = __fadd_rn(a1.y, __fmul_rn(w1.y, k));
            a1.z = __fadd_rn(a1.z, __fmul_rn(w1.z, k));
            a1.w = __fadd_rn(a1.w, __fmul_rn(w1.w, k));
            w0 = w1;
        }
    }
    const int xc = x0 + 4 * cg;
    if (xc >= W) return;
    const bool full = xc + 3 < W;
    const float4 acc[2] = {a0, a1};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int y = y0 + 2 * rg + j;
        if (y >= H) break;
        const int v[4] = {to_u8(acc[j].x), to_u8(acc[j].y), to_u8(acc[j].z), to_u8(acc[j].w)};
        const long long o = (long long)y * pitch + xc;
        if (full) {
            store_level4(out + o, v, lut);
            *reinterpret_cast<unsigned*>(out_u8 + o) =
                (unsigned)v[0] | ((unsigned)v[1] << 8) | ((unsigned)v[2] << 16) | ((unsigned)v[3] << 24);
        } else {
            for (int c = 0; c < 4 && xc + c < W; ++c) {
                store_level(out + o + c, v[c], lut[v[c]]);
                out_u8[o + c] = (uint8_t)v[c];
            }
        }
    }
}

template <typename TG, int kRows>
__global__ void __launch_bounds__(kColThreads) k_blur_cols(const uint8_t* __restrict__ tmp, int tmp_pitch,
                                                          TG* __restrict__ out, uint8_t* __restrict__ out_u8,
                                                          int pitch, int W, int H, int r,
                                                          const float* __restrict__ wts,
                                                          const float* __restrict__ lut255) {
    chain_wait();
    extern __shared__ __align__(16) float sm[];
    blur_cols_tile<TG, kRows>(tmp, tmp_pitch, out, out_u8, pitch, W, H, r, wts, lut255, blockIdx.x * kColTX,
                              blockIdx.y * kRows, sm);
}

// Fused level kernel: both passes of one level on the tensor cores
// (level_tc.cuh), a 64 x TY tile per CTA.
template <typename TG, int P, int PV, int TY, bool CLAMP>
__global__ void __launch_bounds__(tc::kThreads) k_blur_level(const uint8_t* __restrict__ in, int in_pitch,
                                                             TG* __restrict__ out, uint8_t* __restrict__ out_u8,
                                                             int pitch, int W, int H, TcParams tp,
                                                             const ImgRef* __restrict__ ref) {
    chain_wait();
    if (ref) {  // a host call's base level: the image is wherever the cell says
        in = ref->ptr;
        in_pitch = (int)ref->pitch;
    }
    extern __shared__ __align__(16) uint16_t smh[];
    tc::level_tile<TG, P, PV, TY, CLAMP>(in, in_pitch, out, out_u8, pitch, W, H, tp, blockIdx.x * tc::kTX,
                                         blockIdx.y * TY, smh);
}

// A level whose blur increment is below 1e-4 is a copy of the previous one
// (src/sift.rs:152-154).
template <typename TG>
__global__ void k_copy_level(const TG* __restrict__ prev, const uint8_t* __restrict__ prev_u8, TG* __restrict__ out,
                             uint8_t* __restrict__ out_u8, int pitch, int W, int H) {
    chain_wait();
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= W) return;
    long long o = (long long)y * pitch + x;
    if constexpr (!std::is_same<TG, uint8_t>::value) out[o] = prev[o];  // u8 storage: out is out_u8
    out_u8[o] = prev_u8[o];
}

// Base level without a blur (sigma <= assumed_blur, src/sift.rs:1204-1214).
template <typename TG>
__global__ void k_u8_to_level(const uint8_t* __restrict__ img, long long stride, TG* __restrict__ out,
                              uint8_t* __restrict__ out_u8, int pitch, int W, int H, const ImgRef* __restrict__ ref) {
    chain_wait();
    if (ref) {
        img = ref->ptr;
        stride = ref->pitch;
    }
    int x = blockIdx.x * blockDim.x + threadIdx.x;
    int y = blockIdx.y;
    if (x >= W) return;
    const int v = (int)img[(long long)y * stride + x];
    const long long o = (long long)y * pitch + x;
    store_level(out + o, v, norm255(v));
    out_u8[o] = (uint8_t)v;
}

// Both Lanczos3 passes of the 2x resize in one kernel (image 0.25.6
// vertical_sample then horizontal_sample): a 32 x 32 output tile stages its
// source window (at most kLzSpan x kLzSpan, checked on the host), runs the
// vertical pass for the columns the horizontal pass reads, then the
// horizontal pass; every value is formed exactly as in the two-kernel form.
// Tiles inside the uniform interior of a 2x resize (LanczosUniform) run both
// passes with the 12 taps as constants: each thread sums 4 outputs from 18
// shared loads, the tap loops unrolled; the sums are the same, in the same
// order. The other tiles (at the borders: all of a small plane's) stage their
// outputs' taps in shared memory beside the window; read from device memory
// tap by tap they took 10 us where this takes 5.5 (160 x 120; with them the
// pyramid 97 -> 85 us, at 640 x 480 121 -> 106, at 1080p 137 -> 124).
constexpr int kLzTaps = 14;  // of an output (a resize to half has 13 at most, of 15 pixels)
constexpr int kLzT = 32, kLzSpan = 80, kLzMid = 81;  // odd mid stride: lanes on rows hit 32 banks
constexpr int kLzIn = 96;  // staged row: 16-byte aligned x from x_lo & ~15, x_lo - (x_lo & ~15) + span <= 95

template <typename TG>
__device__ __forceinline__ void lanczos_tile(const uint8_t* __restrict__ src, int src_pitch, TG* __restrict__ dst,
                                             uint8_t* __restrict__ dst_u8, int dst_pitch, int nW, int nH,
                                             const int* __restrict__ vtab, const float* __restrict__ vw,
                                             const int* __restrict__ htab, const float* __restrict__ hw,
                                             const LanczosUniform& uni, int ox0, int oy0) {
    __shared__ __align__(16) float in_rows[kLzSpan][kLzIn];
    __shared__ float mid[kLzT][kLzMid];
    __shared__ float taps[2][kLzTaps][kLzT];       // vertical, horizontal
    __shared__ int first[2][kLzT], count[2][kLzT];  // of the taps, from y_lo and x_lo on
    const int* vleft = vtab;
    const int* vcount = vtab + nH;
    const int* voff = vtab + 2 * nH;
    const int* hleft = htab;
    const int* hcount = htab + nW;
    const int* hoff = htab + 2 * nW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ox1 = min(ox0 + kLzT, nW), oy1 = min(oy0 + kLzT, nH);
    const int x_lo = hleft[ox0], x_hi = hleft[ox1 - 1] + hcount[ox1 - 1];
    const int y_lo = vleft[oy0], y_hi = vleft[oy1 - 1] + vcount[oy1 - 1];
    const int sw = x_hi - x_lo, sh = y_hi - y_lo;
    const bool uniform = ox0 >= uni.x0 && ox0 + kLzT <= uni.x1 && oy0 >= uni.y0 && oy0 + kLzT <= uni.y1;
    if (!uniform) {
        // a thread stages four taps or so of output k of an axis, and lane 0 its place
        const int axis = warp >> 2, k = lane, i0 = warp & 3;
        const int out = min((axis ? ox0 : oy0) + k, (axis ? ox1 : oy1) - 1);
        const int* left = axis ? hleft : vleft;
        const int c = (axis ? hcount : vcount)[out], o = (axis ? hoff : voff)[out];
        const float* w = axis ? hw : vw;
        if (i0 == 0) {
            first[axis][k] = left[out] - (axis ? x_lo : y_lo);
            count[axis][k] = c;
        }
#pragma unroll
        for (int i = i0; i < kLzTaps; i += 4) taps[axis][i][k] = i < c ? w[o + i] : 0.0f;
    }
    // stage: 16-byte words from xa = x_lo & ~15 (staged column c holds x =
    // xa + c; the words end at align16(x_hi) <= the row pitch, a multiple of
    // 32), each byte to a float by one byte permute and one subtraction
    const int xa = x_lo & ~15, xo = x_lo - xa;
    const int nq = (x_hi - xa + 15) >> 4;
    if ((src_pitch & 15) == 0) {
        for (int q = tid; q < sh * nq; q += 256) {
            const int yy = q / nq, k = q - yy * nq;
            float v[16];
            unpack16(*reinterpret_cast<const uint4*>(src + (long long)(y_lo + yy) * src_pitch + xa + 16 * k), v);
            float4* d = reinterpret_cast<float4*>(&in_rows[yy][16 * k]);
#pragma unroll
            for (int e = 0; e < 4; ++e) d[e] = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
        }
    } else {
        for (int q = tid; q < sh * sw; q += 256) {
            const int yy = q / sw, xx = q - yy * sw;
            in_rows[yy][xo + xx] = float_of_u8(src[(long long)(y_lo + yy) * src_pitch + x_lo + xx]);
        }
    }
    __syncthreads();
    // in[y][x]: source (y_lo + y, x_lo + x)
    auto in = [&](int y, int x) -> float { return in_rows[y][xo + x]; };
    if (uniform) {
        // vertical pass: warp w makes mid rows 4w .. 4w+3 from source rows
        // 8w .. 8w+17 (output row r reads from 2r, tap i at j = 2r + i)
        for (int xx = lane; xx < sw; xx += 32) {
            float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int j = 0; j < 18; ++j) {
                const float v = in(8 * warp + j, xx);
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (j - 2 * r >= 0 && j - 2 * r < kLz2xTaps) a[r] = __fadd_rn(a[r], __fmul_rn(v, uni.wv[j - 2 * r]));
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) mid[4 * warp + r][xx] = a[r];
        }
        __syncthreads();
        // horizontal pass: lane = output row, warp w = outputs 4w .. 4w+3 of
        // it, from mid columns 8w .. 8w+17
        float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int j = 0; j < 18; ++j) {
            const float v = mid[lane][8 * warp + j];
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (j - 2 * r >= 0 && j - 2 * r < kLz2xTaps) b[r] = __fadd_rn(b[r], __fmul_rn(v, uni.wh[j - 2 * r]));
        }
        const long long od = (long long)(oy0 + lane) * dst_pitch + ox0 + 4 * warp;
        unsigned packed = 0u;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float t = b[r] < 0.0f ? 0.0f : (b[r] > 255.0f ? 255.0f : b[r]);
            const int v = (int)roundf(t);
            store_level(dst + od + r, v, norm255(v));
            packed |= (unsigned)v << (8 * r);
        }
        *reinterpret_cast<unsigned*>(dst_u8 + od) = packed;
        return;
    }
    // vertical pass: rows oy0..oy1-1 (one warp per row), columns x_lo..x_hi-1,
    // three to a lane (the last ones repeat column sw - 1)
    for (int oyl = warp; oyl < oy1 - oy0; oyl += 8) {
        const int l = first[0][oyl], c = count[0][oyl];
        const int x0 = min(lane, sw - 1), x1 = min(lane + 32, sw - 1), x2 = min(lane + 64, sw - 1);
        float t0 = 0.0f, t1 = 0.0f, t2 = 0.0f;
#pragma unroll
        for (int i = 0; i < kLzTaps; ++i) {
            if (i < c) {
                const float w = taps[0][i][oyl];
                t0 = __fadd_rn(t0, __fmul_rn(in(l + i, x0), w));
                t1 = __fadd_rn(t1, __fmul_rn(in(l + i, x1), w));
                t2 = __fadd_rn(t2, __fmul_rn(in(l + i, x2), w));
            }
        }
        mid[oyl][x0] = t0;
        if (lane + 32 < sw) mid[oyl][x1] = t1;
        if (lane + 64 < sw) mid[oyl][x2] = t2;
    }
    __syncthreads();
    // horizontal pass: lane = output column, warp w = rows w, w + 8, ..
    const int ox = ox0 + lane;
    if (ox >= ox1) return;
    const int l = first[1][lane], c = count[1][lane];
    float t[kLzT / 8] = {};
#pragma unroll
    for (int i = 0; i < kLzTaps; ++i) {
        if (i < c) {
            const float w = taps[1][i][lane];
#pragma unroll
            for (int r = 0; r < kLzT / 8; ++r) t[r] = __fadd_rn(t[r], __fmul_rn(mid[warp + 8 * r][l + i], w));
        }
    }
#pragma unroll
    for (int r = 0; r < kLzT / 8; ++r) {
        const int oy = oy0 + warp + 8 * r;
        if (oy >= oy1) return;
        const float s = t[r] < 0.0f ? 0.0f : (t[r] > 255.0f ? 255.0f : t[r]);
        const int v = (int)roundf(s);
        const long long od = (long long)oy * dst_pitch + ox;
        store_level(dst + od, v, norm255(v));
        dst_u8[od] = (uint8_t)v;
    }
}

template <typename TG>
__global__ void __launch_bounds__(256) k_lanczos_fused(const uint8_t* __restrict__ src, int src_pitch,
                                                       TG* __restrict__ dst, uint8_t* __restrict__ dst_u8,
                                                       int dst_pitch, int nW, int nH, const int* __restrict__ vtab,
                                                       const float* __restrict__ vw, const int* __restrict__ htab,
                                                       const float* __restrict__ hw, const LanczosUniform uni) {
    chain_wait();
    lanczos_tile<TG>(src, src_pitch, dst, dst_u8, dst_pitch, nW, nH, vtab, vw, htab, hw, uni, blockIdx.x * kLzT,
                     blockIdx.y * kLzT);
}

// Lanczos3 vertical pass (image 0.25.6 vertical_sample): tmp[oy][x] =
// sum_i G[left+i][x] * w_i, accumulated from 0 in tap order, kept in f32.
// Used when a tile's source window would not fit the fused kernel.
__global__ void k_lanczos_v(const uint8_t* __restrict__ src, int src_pitch, float* __restrict__ dst, int dst_pitch,
                            int W, int nH, const int* __restrict__ left, const int* __restrict__ count,
                            const int* __restrict__ woff, const float* __restrict__ w) {
    chain_wait();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int oy = blockIdx.y;
    if (x >= W || oy >= nH) return;
    const int l = left[oy], c = count[oy], o = woff[oy];
    float t = 0.0f;
    for (int i = 0; i < c; ++i)
        t = __fadd_rn(t, __fmul_rn(float_of_u8(src[(long long)(l + i) * src_pitch + x]), w[o + i]));
    dst[(long long)oy * dst_pitch + x] = t;
}

// Lanczos3 horizontal pass (image 0.25.6 horizontal_sample): clamp to
// [0, 255], round half away from zero, store as the next octave's base level.
template <typename TG>
__global__ void k_lanczos_h(const float* __restrict__ src, int src_pitch, TG* __restrict__ dst,
                            uint8_t* __restrict__ dst_u8, int dst_pitch, int nW, int nH, const int* __restrict__ left,
                            const int* __restrict__ count, const int* __restrict__ woff,
                            const float* __restrict__ w) {
    chain_wait();
    const int ox = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (ox >= nW || y >= nH) return;
    const int l = left[ox], c = count[ox], o = woff[ox];
    const float* row = src + (long long)y * src_pitch;
    float t = 0.0f;
    for (int i = 0; i < c; ++i) t = __fadd_rn(t, __fmul_rn(row[l + i], w[o + i]));
    t = t < 0.0f ? 0.0f : (t > 255.0f ? 255.0f : t);
    const int v = (int)roundf(t);
    const long long od = (long long)y * dst_pitch + ox;
    store_level(dst + od, v, norm255(v));
    dst_u8[od] = (uint8_t)v;
}

// ---------------------------------------------------------------------------
// Flattened batch launches. The entries of a batch are image-major (entry =
// image * O + octave); one launch covers octave o of every image. CTA b
// serves the image k with pref[k] <= b < pref[k + 1], where pref is the
// launch's prefix over the images' tile (or row) counts, and tile b - pref[k]
// of that image; the tile bodies are the single-image kernels' own.
constexpr int kBatchTY = 64;
__device__ __forceinline__ int find_image(const uint32_t* __restrict__ pref, int n, uint32_t b) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pref[mid] <= b) lo = mid; else hi = mid;
    }
    return lo;
}

// level s of octave o from level s - 1 (from the input image when s == 0)
__device__ __forceinline__ const uint8_t* level_src(const BatchPyr& bp, const OctaveDev& od, int k, int s,
                                                    int* pitch) {
    if (s == 0) {
        *pitch = bp.img_pitch[k];
        return reinterpret_cast<const uint8_t*>(bp.img_addr[k]);
    }
    *pitch = od.pitch;
    return bp.U + od.u_off + (long long)(s - 1) * od.plane;
}

template <int P, int PV, bool CLAMP>
__global__ void __launch_bounds__(tc::kThreads) kb_blur_level(BatchPyr bp, int o, int s, int n_img,
                                                              const uint32_t* __restrict__ pref, TcParams tp) {
    chain_wait();
    extern __shared__ __align__(16) uint16_t smh[];
    const int k = find_image(pref, n_img, blockIdx.x);
    const OctaveDev od = bp.ents[k * bp.O + o];
    const int t = (int)(blockIdx.x - pref[k]), tx = (od.W + tc::kTX - 1) / tc::kTX;
    int in_pitch = 0;
    const uint8_t* in = level_src(bp, od, k, s, &in_pitch);
    uint8_t* out = bp.U + od.u_off + (long long)s * od.plane;
    tc::level_tile<uint8_t, P, PV, kBatchTY, CLAMP>(in, in_pitch, out, out, od.pitch, od.W, od.H, tp, (t % tx) * tc::kTX,
                                                    (t / tx) * kBatchTY, smh);
}

__global__ void __launch_bounds__(kRowThreads) kb_blur_rows(BatchPyr bp, uint8_t* __restrict__ tmp, int o, int s,
                                                            int r, int n_img, const uint32_t* __restrict__ pref,
                                                            const float* __restrict__ wts) {
    chain_wait();
    extern __shared__ __align__(16) float sm[];
    const int k = find_image(pref, n_img, blockIdx.x);
    const OctaveDev od = bp.ents[k * bp.O + o];
    int in_pitch = 0;
    const uint8_t* in = level_src(bp, od, k, s, &in_pitch);
    blur_row(in, in_pitch, tmp + od.t_off, od.pitch, od.W, r, wts, (int)(blockIdx.x - pref[k]), sm);
}

__global__ void __launch_bounds__(kColThreads) kb_blur_cols(BatchPyr bp, const uint8_t* __restrict__ tmp, int o,
                                                            int s, int r, int n_img,
                                                            const uint32_t* __restrict__ pref,
                                                            const float* __restrict__ wts,
                                                            const float* __restrict__ lut255) {
    chain_wait();
    extern __shared__ __align__(16) float sm[];
    const int k = find_image(pref, n_img, blockIdx.x);
    const OctaveDev od = bp.ents[k * bp.O + o];
    const int t = (int)(blockIdx.x - pref[k]), tx = (od.W + kColTX - 1) / kColTX;
    uint8_t* out = bp.U + od.u_off + (long long)s * od.plane;
    blur_cols_tile<uint8_t, kColRows>(tmp + od.t_off, od.pitch, out, out, od.pitch, od.W, od.H, r, wts, lut255,
                            (t % tx) * kColTX, (t / tx) * kColRows, sm);
}

// Lanczos tables of one image's resize from octave o to o + 1 (offsets into
// the batch's integer and weight tables).
struct BatchLz {
    int vtab, vw, htab, hw;
    LanczosUniform uni;
};

__global__ void __launch_bounds__(256) kb_lanczos(BatchPyr bp, int o, int n_img, const uint32_t* __restrict__ pref,
                                                  const BatchLz* __restrict__ lz, const int* __restrict__ itab,
                                                  const float* __restrict__ ftab) {
    chain_wait();
    const int k = find_image(pref, n_img, blockIdx.x);
    const int e = k * bp.O + o;
    const OctaveDev od = bp.ents[e], nx = bp.ents[e + 1];
    const BatchLz& z = lz[e];
    const int t = (int)(blockIdx.x - pref[k]), tx = (nx.W + kLzT - 1) / kLzT;
    uint8_t* dst = bp.U + nx.u_off;
    lanczos_tile<uint8_t>(bp.U + od.u_off + (long long)bp.S * od.plane, od.pitch, dst, dst, nx.pitch, nx.W, nx.H,
                          itab + z.vtab, ftab + z.vw, itab + z.htab, ftab + z.hw, z.uni, (t % tx) * kLzT,
                          (t / tx) * kLzT);
}

}  // namespace

// ---- launchers ----------------------------------------------------------------

size_t blur_rows_smem(int W, int r) {
    int taps = 2 * r + 1;
    return sizeof(float) * ((size_t)((taps + 3) & ~3) + (size_t)W + 2 * (size_t)r + 8);
}
size_t blur_cols_smem(int r, int rows) {
    return sizeof(float) * ((size_t)taps8(r) + 256 + (size_t)(rows + taps8(r) - 1) * kColTX);
}

// 64-row tiles from this many on (two per multiprocessor): fewer leave
// multiprocessors idle or with one CTA, and 32-row tiles, which recompute
// more halo (48 against 80 rows per 64), still finish sooner.
constexpr long long kTallTiles = 2 * 152;

static int set_smem(const void* k, size_t smem) {
    if (smem <= 48 * 1024) return 0;
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess ? 0 : -1;
}

// The level kernel's shape for a radius: f(P, PV) with the smallest window
// and rows that hold it (tables.cpp: tc_blur lays the fragments out for them).
template <class F>
static int for_tc_shape(int r, F f) {
    if (r <= 4) return f(std::integral_constant<int, 4>{}, std::integral_constant<int, 8>{});
    if (r <= 8) return f(std::integral_constant<int, 12>{}, std::integral_constant<int, 8>{});
    if (r <= 12) return f(std::integral_constant<int, 12>{}, std::integral_constant<int, 16>{});
    if (r <= 16) return f(std::integral_constant<int, 20>{}, std::integral_constant<int, 16>{});
    if (r <= 20) return f(std::integral_constant<int, 20>{}, std::integral_constant<int, 24>{});
    if (r <= 24) return f(std::integral_constant<int, 28>{}, std::integral_constant<int, 24>{});
    return f(std::integral_constant<int, 28>{}, std::integral_constant<int, 32>{});
}

template <typename TG, int P, int PV, int TY, bool CLAMP>
int launch_blur_level_tc(const uint8_t* in, int in_pitch, TG* out, uint8_t* out_u8, int pitch, int W, int H,
                         const TcParams& tp, cudaStream_t st, const ImgRef* ref) {
    constexpr size_t smem = tc::Shape<P, PV, TY>::smem;
    const auto kern = k_blur_level<TG, P, PV, TY, CLAMP>;
    if (set_smem((const void*)kern, smem)) return -1;
    dim3 grid((W + tc::kTX - 1) / tc::kTX, (H + TY - 1) / TY);
    if (launch_chained(kern, grid, tc::kThreads, smem, st, in, in_pitch, out, out_u8, pitch, W, H, tp, ref) !=
        cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

// One level from the previous level's u8 plane: one launch on the tensor
// cores for the radii it takes (up to 28) unless the autotuner's radius limit
// (below 8) excludes them, else the two separable passes.
static bool level_fused(const TcBlur& b, int r, int fused_max_radius) {
    return b.ok && (fused_max_radius >= 8 || r <= fused_max_radius);
}

template <typename TG>
int launch_blur_level(const uint8_t* in, int in_pitch, uint8_t* tmp, TG* out, uint8_t* out_u8, int pitch, int W,
                      int H, int r, const float* wts, const TcBlur& b, const void* frags, const float* lut255,
                      cudaStream_t st, int* launches, int fused_max_radius, const ImgRef* ref, int tile_rows) {
    if (level_fused(b, r, fused_max_radius)) {
        const TcParams tp{static_cast<const uint4*>(frags), wts, r, b.init_a, b.init_b, b.scale_b, b.whole, b.near};
        // planes whose 64-row tiles would leave multiprocessors idle take 32-row tiles
        const bool tall = tile_rows == 64 ||
                          (tile_rows == 0 && (long long)((W + 63) / 64) * ((H + 63) / 64) >= kTallTiles);
        const int rc = for_tc_shape(r, [&](auto p, auto pv) {
            constexpr int P = decltype(p)::value, PV = decltype(pv)::value;
            if constexpr (P == 4) {  // only narrow kernels sum to 256
                if (b.clamp && tile_rows == 64)
                    return launch_blur_level_tc<TG, P, PV, 64, true>(in, in_pitch, out, out_u8, pitch, W, H, tp, st, ref);
                if (b.clamp)
                    return launch_blur_level_tc<TG, P, PV, 32, true>(in, in_pitch, out, out_u8, pitch, W, H, tp, st, ref);
            }
            return tall ? launch_blur_level_tc<TG, P, PV, 64, false>(in, in_pitch, out, out_u8, pitch, W, H, tp, st, ref)
                        : launch_blur_level_tc<TG, P, PV, 32, false>(in, in_pitch, out, out_u8, pitch, W, H, tp, st, ref);
        });
        if (rc) return rc;
        *launches += 1;
        return 0;
    }
    // Planes with few 64-row tiles take 8-row tiles: an output per thread ends
    // sooner than eight side by side (with the rows' form, 160 x 120 107 -> 101
    // us for the frame, 640 x 480 140 -> 137, 1280 x 720, ten tiles, 167 ->
    // 163). They stage r rows above and below each, so with more of them they
    // cost the other octaves' kernels more than they save (24, 1080p: 333 -> 335
    // us; 4096 x 4096 with 128 and 32: 2123 -> 2148, and with 8 of radii 79 to
    // 198, which stage 50 rows for one, 2120 -> 2128).
    const int cols = (W + kColTX - 1) / kColTX;
    const bool small = r <= kColRows && (long long)cols * ((H + kColRows - 1) / kColRows) <= kColFew;
    const int rows = small ? kColRowsSmall : kColRows;
    const auto k_cols = small ? k_blur_cols<TG, kColRowsSmall> : k_blur_cols<TG, kColRows>;
    const size_t rs = blur_rows_smem(W, r), cs = blur_cols_smem(r, rows);
    if (set_smem((const void*)k_blur_rows, rs) || set_smem((const void*)k_cols, cs)) return -1;
    if (launch_chained(k_blur_rows, H, kRowThreads, rs, st, in, in_pitch, tmp, pitch, W, r, wts, ref) !=
        cudaSuccess)
        return -1;
    dim3 grid(cols, (H + rows - 1) / rows);
    if (launch_chained(k_cols, grid, kColThreads, cs, st, tmp, pitch, out, out_u8, pitch, W, H, r, wts, lut255) !=
        cudaSuccess)
        return -1;
    *launches += 2;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

template <typename TG>
int launch_copy_level(const TG* prev, const uint8_t* prev_u8, TG* out, uint8_t* out_u8, int pitch, int W,
                      int H, cudaStream_t st) {
    dim3 grid((W + 255) / 256, H);
    if (launch_chained(k_copy_level<TG>, grid, 256, 0, st, prev, prev_u8, out, out_u8, pitch, W, H) != cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

template <typename TG>
int launch_u8_to_level(const uint8_t* img, long long stride, TG* out, uint8_t* out_u8, int pitch, int W, int H,
                       cudaStream_t st, const ImgRef* ref) {
    dim3 grid((W + 255) / 256, H);
    if (launch_chained(k_u8_to_level<TG>, grid, 256, 0, st, img, stride, out, out_u8, pitch, W, H, ref) !=
        cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

template <typename TG>
int launch_lanczos(const uint8_t* src, int src_pitch, int W, int H, float* tmp, int tmp_pitch, TG* dst,
                   uint8_t* dst_u8, int dst_pitch, int nW, int nH, const int* vtab, const float* vw, const int* htab,
                   const float* hw, const LanczosUniform& uni, cudaStream_t st, bool fused, int* launches) {
    if (fused) {
        dim3 g((nW + kLzT - 1) / kLzT, (nH + kLzT - 1) / kLzT);
        if (launch_chained(k_lanczos_fused<TG>, g, 256, 0, st, src, src_pitch, dst, dst_u8, dst_pitch, nW, nH, vtab,
                           vw, htab, hw, uni) != cudaSuccess)
            return -1;
        *launches += 1;
        return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
    }
    dim3 gv((W + 127) / 128, nH);
    if (launch_chained(k_lanczos_v, gv, 128, 0, st, src, src_pitch, tmp, tmp_pitch, W, nH, vtab, vtab + nH,
                       vtab + 2 * nH, vw) != cudaSuccess)
        return -1;
    dim3 gh((nW + 127) / 128, nH);
    if (launch_chained(k_lanczos_h<TG>, gh, 128, 0, st, tmp, tmp_pitch, dst, dst_u8, dst_pitch, nW, nH, htab,
                       htab + nW, htab + 2 * nW, hw) != cudaSuccess)
        return -1;
    (void)H;
    *launches += 2;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

// Whether an axis' windows and taps fit the fused kernel's tiles.
bool lanczos_fits(const AxisTaps& t) {
    const int n = (int)t.left.size();
    for (int a = 0; a < n; a += kLzT) {
        const int b = std::min(a + kLzT, n) - 1;
        if (t.left[b] + t.count[b] - t.left[a] > kLzSpan) return false;
    }
    return std::all_of(t.count.begin(), t.count.end(), [](int c) { return c <= kLzTaps; });
}

// ---- flattened batch launchers ------------------------------------------------

int blur_level_tiles(int W, int H) { return W > 0 && H > 0 ? ((W + tc::kTX - 1) / tc::kTX) * ((H + kBatchTY - 1) / kBatchTY) : 0; }
int blur_col_tiles(int W, int H) {
    return W > 0 && H > 0 ? ((W + kColTX - 1) / kColTX) * ((H + kColRows - 1) / kColRows) : 0;
}
int lanczos_tiles(int nW, int nH) { return nW > 0 && nH > 0 ? ((nW + kLzT - 1) / kLzT) * ((nH + kLzT - 1) / kLzT) : 0; }
size_t batch_lz_bytes() { return sizeof(BatchLz); }
void batch_lz_fill(void* out, int vtab, int vw, int htab, int hw, const LanczosUniform& uni) {
    BatchLz z{vtab, vw, htab, hw, uni};
    std::memcpy(out, &z, sizeof z);
}

// Level s of octave o of every image of a batch: the fused kernel (tiles
// prefixed by fused_pref) or the two passes (rows prefixed by
// rows_pref, column tiles by cols_pref; tmp holds each entry's
// horizontal-pass plane at its t_off).
int launch_blur_level_flat(const BatchPyr& bp, uint8_t* tmp, int o, int s, int r, int n_img,
                           const uint32_t* fused_pref, uint32_t n_fused, const uint32_t* rows_pref, uint32_t n_rows,
                           int max_w, const uint32_t* cols_pref, uint32_t n_cols, const float* wts, const TcBlur& b,
                           const void* frags, const float* lut255, cudaStream_t st, int* launches) {
    if (level_fused(b, r, 8)) {
        if (n_fused == 0) return 0;
        const TcParams tp{static_cast<const uint4*>(frags), wts, r, b.init_a, b.init_b, b.scale_b, b.whole, b.near};
        auto go = [&](auto kern, size_t smem) -> int {
            if (set_smem((const void*)kern, smem)) return -1;
            return launch_chained(kern, n_fused, tc::kThreads, smem, st, bp, o, s, n_img, fused_pref, tp) == cudaSuccess ? 0 : -1;
        };
        const int rc = for_tc_shape(r, [&](auto p, auto pv) {
            constexpr int P = decltype(p)::value, PV = decltype(pv)::value;
            constexpr size_t smem = tc::Shape<P, PV, kBatchTY>::smem;
            if constexpr (P == 4) {
                if (b.clamp) return go(kb_blur_level<P, PV, true>, smem);
            }
            return go(kb_blur_level<P, PV, false>, smem);
        });
        if (rc) return rc;
        *launches += 1;
        return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
    }
    if (n_rows == 0) return 0;
    const size_t rs = blur_rows_smem(max_w, r), cs = blur_cols_smem(r, kColRows);
    if (set_smem((const void*)kb_blur_rows, rs) || set_smem((const void*)kb_blur_cols, cs)) return -1;
    if (launch_chained(kb_blur_rows, n_rows, kRowThreads, rs, st, bp, tmp, o, s, r, n_img, rows_pref, wts) !=
        cudaSuccess)
        return -1;
    if (launch_chained(kb_blur_cols, n_cols, kColThreads, cs, st, bp, (const uint8_t*)tmp, o, s, r, n_img, cols_pref,
                       wts, lut255) != cudaSuccess)
        return -1;
    *launches += 2;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

// The 2x Lanczos3 resize of octave o to o + 1 of every image (every resize
// fits the fused kernel; the caller checks).
int launch_lanczos_flat(const BatchPyr& bp, int o, int n_img, const uint32_t* pref, uint32_t n_tiles,
                        const void* lz, const int* itab, const float* ftab, cudaStream_t st) {
    if (n_tiles == 0) return 0;
    if (launch_chained(kb_lanczos, n_tiles, 256, 0, st, bp, o, n_img, pref, (const BatchLz*)lz, itab, ftab) !=
        cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

#define SIFT_INST(TG)                                                                                              \
    template int launch_blur_level<TG>(const uint8_t*, int, uint8_t*, TG*, uint8_t*, int, int, int, int,           \
                                       const float*, const TcBlur&, const void*, const float*, cudaStream_t, int*, \
                                       int, const ImgRef*, int);                                                   \
    template int launch_copy_level<TG>(const TG*, const uint8_t*, TG*, uint8_t*, int, int, int,                    \
                                       cudaStream_t);                                                              \
    template int launch_u8_to_level<TG>(const uint8_t*, long long, TG*, uint8_t*, int, int, int, cudaStream_t,     \
                                        const ImgRef*);                                                            \
    template int launch_lanczos<TG>(const uint8_t*, int, int, int, float*, int, TG*, uint8_t*, int, int, int,      \
                                    const int*, const float*, const int*, const float*, const LanczosUniform&,      \
                                    cudaStream_t, bool, int*);
SIFT_INST(float)
SIFT_INST(__half)
SIFT_INST(uint8_t)
#undef SIFT_INST

}  // namespace sift
