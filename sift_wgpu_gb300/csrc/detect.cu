// detect.cu — 26-neighbour extrema, ordered candidates, subpixel refinement.
//
// Stages (b) and (c) of the hot path: find_scale_space_extrema
// (src/sift.rs:510-603) and refine_and_filter_extrema (src/sift.rs:299-474).
//
//   k_extrema_mask   the strict 26-neighbour test of a tile of pixels, one
//                    ballot word per 32 pixels of a row; the candidates are
//                    counted by tiles of words as they are found.
//   k_candidates     a CTA per tile of words: the counts of the tiles before
//                    it give every candidate its slot in (octave, layer, y,
//                    x) order, the order rayon's collect produces in the
//                    reference; then one thread per candidate, the Newton
//                    refinement, contrast and edge tests in the reference's
//                    f32 operation order; the result stays in the candidate's
//                    slot with a keep flag (the orientation stage reads the
//                    slots in order and skips the rejected ones, so no
//                    compaction pass is needed).
//
// All arithmetic is f32 with separately rounded operations (no FMA), so the
// candidates and refined keypoints are bit-identical to the CPU path; the one
// transcendental, 2^(octave + layer/S) for the keypoint size, is evaluated in
// f64 and rounded once.
#include <cuda_fp16.h>

#include <algorithm>

#include "tile_scan.cuh"

namespace sift {
namespace {

// DoG access for one octave (src/sift.rs:208-214 get_pixel_value, clamped).
// DoG of one octave recomputed from the u8 copies of its Gaussian levels:
// D_l = lut[G_{l+1}] - lut[G_l] with lut[v] = v/255 in f32 — the reference's
// f32 DoG bit for bit (src/sift.rs:92-124) in either storage mode, at one byte
// per level value instead of four (the refinement's scattered 3 x 3 x 3 reads
// then mostly hit L2).
struct DogFromU8 {
    const uint8_t* base;  // u8 level 0 of the octave
    const float* lut;     // v / 255, shared or global
    long long plane;
    int pitch, W, H;
    __device__ __forceinline__ float at(int l, int x, int y) const {
        x = clampi(x, 0, W - 1);
        y = clampi(y, 0, H - 1);
        const uint8_t* p = base + (long long)l * plane + (long long)y * pitch + x;
        return __fsub_rn(lut[p[plane]], lut[p[0]]);
    }
};

// ---------------------------------------------------------------------------
// Extrema of one octave, all layers s = 1..S at once:
//   strict max  <=>  v > max(M_{s-1}, M_{s+1}, ring8max_s)
//   strict min  <=>  v < min(m_{s-1}, m_{s+1}, ring8min_s)
// with M, m the 3 x 3 block's max and min, which is the reference's 26 strict
// comparisons (ties reject) of f32 DoG values.
//
// Only their order matters, and 16 bits hold it: two pixels go through every
// operation, three-way minima and maxima included, in one register. With h(v)
// the highest power of two in v (h(0) = 0), v / 255 in f32 is
//   (v * 0x808080 + h(v)) * 2^-31,
// (its binary digits repeat v's eight, and the bit after the 24th from the
// first one is always 1), so the DoG value of bytes a and b is the f32 rounding
// of (d * 0x808080 + h(a) - h(b)) * 2^-31, d = a - b. Where a <= 2 b and b <=
// 2 a the subtraction is exact and |h(a) - h(b)| <= 64: the key
//   128 d + h(a) - h(b) = T(a) - T(b),  T(v) = 128 v + h(v)
// orders the values, equal keys for equal values only. Elsewhere (a dark pixel
// beside a much brighter one in the next level) exact_key makes the key of the
// rounded difference; with it, the order of the keys of all 65 536 pairs is
// that of their f32 values.
//
// A CTA stages the keys of its 128 x 16 pixels and their neighbours for every
// DoG layer 0..S+1 in shared memory (clamped coordinates, as get_pixel_value
// clamps, at the image border), word i of a row the pixels x0 - 4 + i and
// x0 + 60 + i. Each thread owns one such pair of columns and 4 rows: per layer
// it forms the horizontal 3-max/3-min of 6 rows once and reuses them for the
// block max/min and the ring max/min of its 8 pixels; a ballot of either half
// is a word of the mask.
//
// The integer pipe bounds it (64 lanes per clock and SM for each of these
// operations, the three-way ones too). Octave 0 takes 79 us at 4096 x 4096 and
// 16 at 1080p; with f32 values, one pixel each, of a table in shared memory
// (64 x 16 tiles) it took 169 and 26. The stage: 351 -> 231 us and 91 -> 79.
// The rounded keys cost 4 us of the 79;
// 3 CTAs per SM, which spill nothing, take 9 % more than 4.
constexpr int kExTX = 128, kExTY = 16, kExRows = 4, kExMaxLayers = 18, kExThreads = 256;
constexpr int kExHalf = kExTX / 2;
constexpr int kExSW = kExHalf + 8;  // staged words of a row: pairs from x0 - 4 on
constexpr int kExSH = kExTY + 2;
constexpr uint32_t kExBias = 0x80008000u;

// The key of level bytes a (of the layer's upper level) and b, plus 0x8000, in
// the low 16 bits: v / 255 in units of 2^-31, its f32 difference, and what that
// has beyond d * 0x808080 (every step but the difference is exact).
__device__ __forceinline__ uint32_t exact_key(uint32_t a, uint32_t b) {
    constexpr float k255 = 8421504.0f;  // 0x808080
    const float af = (float)a, bf = (float)b;
    const float ha = __uint_as_float(__float_as_uint(af) & 0x7F800000u), hb = __uint_as_float(__float_as_uint(bf) & 0x7F800000u);
    const float diff = __fsub_rn(fmaf(af, k255, ha), fmaf(bf, k255, hb));
    const float d = af - bf;
    float e = fmaf(-d, k255, diff);
    if (fabsf(e) == 128.0f) e = copysignf(100.0f, e);  // (others are at most 64; the next d's key starts at 128)
    return __float_as_uint(fmaf(d, 128.0f, e) + (8388608.0f + 32768.0f));
}

// A pair of level bytes, in three forms: as f16 numbers, and their T up to a
// constant.
struct ExPair {
    __half2 v;
    uint32_t t;
};
// raw: the bytes below 0x64, i.e. 1024 + v as f16
__device__ __forceinline__ ExPair ex_pair(uint32_t raw) {
    const __half2 k1024 = __half2half2(__ushort_as_half(0x6400));
    ExPair p;
    p.v = __hsub2(*reinterpret_cast<const __half2*>(&raw), k1024);
    // the exponent bits alone are h(v)
    const uint32_t h = *reinterpret_cast<const uint32_t*>(&p.v) & 0x7C007C00u;
    const __half2 hk = __hadd2(*reinterpret_cast<const __half2*>(&h), k1024);
    p.t = raw * 128u + *reinterpret_cast<const uint32_t*>(&hk);
    return p;
}

// Four bytes of a row, from x on (clamped coordinates).
__device__ __forceinline__ uint32_t clamped_word(const uint8_t* row, int x, int W) {
    uint32_t w = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) w |= (uint32_t)row[clampi(x + k, 0, W - 1)] << (8 * k);
    return w;
}

// Stages layers 0 .. L - 1 of the tile: an item is four words of a row, all
// levels of it.
template <int NL>
__device__ __forceinline__ void stage_keys(uint32_t* tile, const uint8_t* base, long long plane, int pitch, int W,
                                           int H, int L, int x0, int y0) {
    constexpr int kChunks = kExSW / 4;
    for (int q = threadIdx.x; q < kExSH * kChunks; q += kExThreads) {
        const int yy = q / kChunks, c = q - yy * kChunks, x = x0 - 4 + 4 * c;
        const uint8_t* row = base + (long long)clampi(y0 - 1 + yy, 0, H - 1) * pitch;
        uint32_t* out = tile + yy * kExSW + 4 * c;
        const bool whole = x >= 0 && x + kExHalf + 4 <= W;
        auto word = [&](const uint8_t* r, int xx) {
            return whole ? *reinterpret_cast<const uint32_t*>(r + xx) : clamped_word(r, xx, W);
        };
        ExPair prev[4];
        uint32_t unsafe = 0;  // a bit for each layer
        auto level = [&](int l, uint32_t lo, uint32_t hi) {
            const uint32_t a = __byte_perm(lo, hi, 0x5140u), b = __byte_perm(lo, hi, 0x7362u);
            const ExPair p[4] = {ex_pair(__byte_perm(a, 0x64646464u, 0x4140u)), ex_pair(__byte_perm(a, 0x64646464u, 0x4342u)),
                                 ex_pair(__byte_perm(b, 0x64646464u, 0x4140u)), ex_pair(__byte_perm(b, 0x64646464u, 0x4342u))};
            if (l > 0) {
                const __half2 two = __half2half2(__ushort_as_half(0x4000));
                uint32_t key[4], bad = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    key[k] = p[k].t + kExBias - prev[k].t;
                    const __half2 s = __hfma2(two, p[k].v, __hneg2(prev[k].v)), t = __hfma2(two, prev[k].v, __hneg2(p[k].v));
                    bad |= *reinterpret_cast<const uint32_t*>(&s) | *reinterpret_cast<const uint32_t*>(&t);
                }
                if (bad & kExBias) unsafe |= 1u << (l - 1);
                *reinterpret_cast<uint4*>(out + (l - 1) * kExSH * kExSW) = make_uint4(key[0], key[1], key[2], key[3]);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) prev[k] = p[k];
        };
        if constexpr (NL > 0) {
            uint32_t lo[NL + 1], hi[NL + 1];  // all reads first
            if (whole) {
                const uint8_t* src = row + x;
#pragma unroll
                for (int l = 0; l <= NL; ++l, src += plane) {
                    lo[l] = *reinterpret_cast<const uint32_t*>(src);
                    hi[l] = *reinterpret_cast<const uint32_t*>(src + kExHalf);
                }
            } else {
                const uint8_t* src = row;
#pragma unroll
                for (int l = 0; l <= NL; ++l, src += plane) {
                    lo[l] = clamped_word(src, x, W);
                    hi[l] = clamped_word(src, x + kExHalf, W);
                }
            }
#pragma unroll
            for (int l = 0; l <= NL; ++l) level(l, lo[l], hi[l]);
        } else {
            const uint8_t* src = row;
#pragma unroll 1
            for (int l = 0; l <= L; ++l, src += plane) level(l, clamped_word(src, x, W), clamped_word(src, x + kExHalf, W));
        }
#pragma unroll 1
        for (; unsafe; unsafe &= unsafe - 1u) {
            const int l = __ffs(unsafe) - 1;
            const uint8_t *b = row + l * plane, *a = b + plane;
            const uint32_t al = word(a, x), ah = word(a, x + kExHalf), bl = word(b, x), bh = word(b, x + kExHalf);
            uint32_t key[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                key[k] = __byte_perm(exact_key(al >> (8 * k) & 255u, bl >> (8 * k) & 255u),
                                     exact_key(ah >> (8 * k) & 255u, bh >> (8 * k) & 255u), 0x5410u);
            *reinterpret_cast<uint4*>(out + l * kExSH * kExSW) = make_uint4(key[0], key[1], key[2], key[3]);
        }
    }
}

// NL > 0: the number of DoG layers (S + 2) is compiled in and the layer loop
// unrolls, so the sliding window renames registers instead of moving them;
// NL == 0: any S. The candidates are counted by tiles of kWordTile words, from
// word0 on.
template <int NL>
__device__ __forceinline__ void extrema_tile(const uint8_t* __restrict__ u8arena, const OctaveDev& od, int S,
                                             int border, uint32_t* __restrict__ words, long long word0,
                                             uint32_t* __restrict__ tiles, int x0, int y0, uint32_t* tile) {
    const int W = od.W, H = od.H, nw = od.nw, L = NL > 0 ? NL : S + 2;
    const int tid = threadIdx.x, lane = tid & 31;
    stage_keys<NL>(tile, u8arena + od.u_off, od.plane, od.pitch, W, H, L, x0, y0);
    __syncthreads();
    const int i = tid & (kExHalf - 1);                 // columns x0 + i and x0 + 64 + i
    const int r0 = (tid / kExHalf) * kExRows;          // 0, 4, 8, 12
    // lanes 0 .. 7 write: row r0 + lane / 2, the low halves' word (even) or the high halves'
    const int wrow = y0 + r0 + (lane >> 1 & 3), word = (x0 >> 5) + (i >> 5) + 2 * (lane & 1);
    const bool writes = lane < 2 * kExRows && wrow < H && word < nw;
    long long at = od.word_base + (long long)wrow * nw + word;
    auto in_x = [&](int x) { return x >= border && x < W - border; };
    const uint32_t columns = (in_x(x0 + i) ? 0x0000ffffu : 0u) | (in_x(x0 + kExHalf + i) ? 0xffff0000u : 0u);
    uint32_t rows = 0;  // a bit for each row that may hold candidates
#pragma unroll
    for (int j = 0; j < kExRows; ++j) rows |= (y0 + r0 + j >= border && y0 + r0 + j < H - border ? 1u : 0u) << j;
    // Sliding window over the layers: p = l-2, c = l-1, n = l.
    uint32_t BMp[kExRows], Bmp[kExRows], BMc[kExRows], Bmc[kExRows], RMc[kExRows], Rmc[kExRows], Vc[kExRows];
#pragma unroll
    for (int j = 0; j < kExRows; ++j) BMp[j] = Bmp[j] = BMc[j] = Bmc[j] = RMc[j] = Rmc[j] = Vc[j] = 0u;
#pragma unroll
    for (int l = 0; l < (NL > 0 ? NL : L); ++l) {
        const uint32_t* t = tile + (l * kExSH + r0) * kExSW + i + 4;  // staged row y0 + r0 - 1
        uint32_t mid[kExRows + 2], hM[kExRows + 2], hm[kExRows + 2], rM[kExRows + 2], rm[kExRows + 2];
#pragma unroll
        for (int j = 0; j < kExRows + 2; ++j) {
            const uint32_t left = t[j * kExSW - 1], right = t[j * kExSW + 1];
            mid[j] = t[j * kExSW];
            hM[j] = __vimax3_u16x2(left, mid[j], right);
            hm[j] = __vimin3_u16x2(left, mid[j], right);
            rM[j] = __vmaxu2(left, right);
            rm[j] = __vminu2(left, right);
        }
        uint32_t BMn[kExRows], Bmn[kExRows];
#pragma unroll
        for (int j = 0; j < kExRows; ++j) {
            BMn[j] = __vimax3_u16x2(hM[j], hM[j + 1], hM[j + 2]);
            Bmn[j] = __vimin3_u16x2(hm[j], hm[j + 1], hm[j + 2]);
        }
        if (l >= 2) {
            // centre layer l - 1
            uint32_t ext[kExRows], some = 0;
#pragma unroll
            for (int j = 0; j < kExRows; ++j) {
                const uint32_t nM = __vimax3_u16x2(BMp[j], BMn[j], RMc[j]), nm = __vimin3_u16x2(Bmp[j], Bmn[j], Rmc[j]);
                // a half other than zero: above all or below all
                ext[j] = (__vmaxu2(Vc[j], nM) ^ nM) | (__vminu2(Vc[j], nm) ^ nm);
                some |= ext[j];
            }
            uint32_t wv = 0;
            if (__any_sync(0xffffffffu, (some & columns) != 0u)) {
#pragma unroll
                for (int j = 0; j < kExRows; ++j) {
                    const uint32_t e = rows >> j & 1u ? ext[j] & columns : 0u;
                    const uint32_t lo = __ballot_sync(0xffffffffu, (e & 0xffffu) != 0u);
                    const uint32_t hi = __ballot_sync(0xffffffffu, e >> 16 != 0u);
                    if (lane >> 1 == j) wv = lane & 1 ? hi : lo;
                }
                if (writes && wv) atomicAdd(&tiles[(at - word0) / kWordTile], (uint32_t)__popc(wv));
            }
            if (writes) words[at] = wv;
            at += (long long)H * nw;
        }
#pragma unroll
        for (int j = 0; j < kExRows; ++j) {
            BMp[j] = BMc[j];
            Bmp[j] = Bmc[j];
            BMc[j] = BMn[j];
            Bmc[j] = Bmn[j];
            RMc[j] = __vimax3_u16x2(hM[j], hM[j + 2], rM[j + 1]);
            Rmc[j] = __vimin3_u16x2(hm[j], hm[j + 2], rm[j + 1]);
            Vc[j] = mid[j + 1];
        }
    }
}

// The extrema mask of entry e (one octave of one image), a tile per CTA.
template <int NL>
__global__ void __launch_bounds__(kExThreads, 4) k_extrema_mask(const uint8_t* __restrict__ u8arena, EntryTable tab, int e,
                                                      int border, uint32_t* __restrict__ words, long long word0,
                                                      uint32_t* __restrict__ tiles) {
    chain_wait();
    extern __shared__ __align__(16) uint32_t tile[];  // [layers][kExSH][kExSW]
    const OctaveDev od = tab.ents[e];
    extrema_tile<NL>(u8arena, od, tab.S, border, words, word0, tiles, blockIdx.x * kExTX, blockIdx.y * kExTY,
                     tile);
}

// The extrema masks of entries e0 .. e0 + n_e - 1 in one launch: CTA b takes
// tile b - tile_pref[k] of entry e0 + k, tile_pref[k] <= b < tile_pref[k + 1]
// (row-major tiles of kExTX x kExTY).
template <int NL>
__global__ void __launch_bounds__(kExThreads, 4) k_extrema_mask_flat(const uint8_t* __restrict__ u8arena, EntryTable tab, int e0,
                                                           int n_e, const uint32_t* __restrict__ tile_pref,
                                                           int border, uint32_t* __restrict__ words,
                                                           long long word0, uint32_t* __restrict__ tiles) {
    chain_wait();
    extern __shared__ __align__(16) uint32_t tile[];
    const uint32_t b = blockIdx.x;
    int lo = 0, hi = n_e;  // the last k with tile_pref[k] <= b
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (tile_pref[mid] <= b) lo = mid; else hi = mid;
    }
    const OctaveDev od = tab.ents[e0 + lo];
    const int tx = (od.W + kExTX - 1) / kExTX;
    const int t = (int)(b - tile_pref[lo]);
    extrema_tile<NL>(u8arena, od, tab.S, border, words, word0, tiles, (t % tx) * kExTX, (t / tx) * kExTY, tile);
}

// solve_linear_system (src/sift.rs:478-503), Cramer's rule in f32.
__device__ __forceinline__ bool solve3(const float a[3][3], const float b[3], float x[3]) {
#define M(p, q) __fmul_rn(p, q)
#define S(p, q) __fsub_rn(p, q)
#define A(p, q) __fadd_rn(p, q)
    const float det_a = A(S(M(a[0][0], S(M(a[1][1], a[2][2]), M(a[1][2], a[2][1]))),
                            M(a[0][1], S(M(a[1][0], a[2][2]), M(a[1][2], a[2][0])))),
                          M(a[0][2], S(M(a[1][0], a[2][1]), M(a[1][1], a[2][0]))));
    if (fabsf(det_a) < 1e-10f) return false;
    const float det_x = A(S(M(b[0], S(M(a[1][1], a[2][2]), M(a[1][2], a[2][1]))),
                            M(a[0][1], S(M(b[1], a[2][2]), M(a[1][2], b[2])))),
                          M(a[0][2], S(M(b[1], a[2][1]), M(a[1][1], b[2]))));
    const float det_y = A(S(M(a[0][0], S(M(b[1], a[2][2]), M(a[1][2], b[2]))),
                            M(b[0], S(M(a[1][0], a[2][2]), M(a[1][2], a[2][0])))),
                          M(a[0][2], S(M(a[1][0], b[2]), M(b[1], a[2][0]))));
    const float det_z = A(S(M(a[0][0], S(M(a[1][1], b[2]), M(b[1], a[2][1]))),
                            M(a[0][1], S(M(a[1][0], b[2]), M(b[1], a[2][0])))),
                          M(b[0], S(M(a[1][0], a[2][1]), M(a[1][1], a[2][0]))));
#undef M
#undef S
#undef A
    x[0] = __fdiv_rn(det_x, det_a);
    x[1] = __fdiv_rn(det_y, det_a);
    x[2] = __fdiv_rn(det_z, det_a);
    return true;
}

struct RefineParams {
    float sigma;
    float contrast_threshold;
    float edge_ratio;  // (edge threshold + 1)^2 / edge threshold
    int S;
    int levels_dog;  // S + 2
};

// One candidate through refine_and_filter_extrema (src/sift.rs:299-474).
template <class Dog>
__device__ __forceinline__ bool refine_one(const Dog& dog, int o, int entry, int x, int y, int s, const RefineParams& rp,
                           Keypoint* out) {
    int cx = x, cy = y, cl = s;
    const float scale = __int_as_float((127 + o) << 23);  // 2^o
    const int nl = rp.levels_dog;
    for (int step = 0; step < 5; ++step) {
        if (cl < 1 || cl >= nl - 1) return false;
        if (cx < 1 || cx >= dog.W - 1 || cy < 1 || cy >= dog.H - 1) return false;
        // the levels below, at and above the layer's two, rows cy - 1 .. cy + 1:
        // all inside, so each value is one read at a constant distance
        const uint8_t* g1 = dog.base + (long long)cl * dog.plane + (long long)cy * dog.pitch + cx;
        const uint8_t *g0 = g1 - dog.plane, *g2 = g1 + dog.plane, *g3 = g2 + dog.plane;
        const float* lut = dog.lut;
        const int up = -dog.pitch, down = dog.pitch;
        auto layer = [&](const uint8_t* lower, const uint8_t* upper, int at) {
            return __fsub_rn(lut[upper[at]], lut[lower[at]]);
        };
        const float c = layer(g1, g2, 0);
        const float cxp = layer(g1, g2, 1), cxm = layer(g1, g2, -1);
        const float cyp = layer(g1, g2, down), cym = layer(g1, g2, up);
        const float nc = layer(g2, g3, 0), pc = layer(g0, g1, 0);
        // (halves and quarters are exact)
        const float dx = __fmul_rn(__fsub_rn(cxp, cxm), 0.5f);
        const float dy = __fmul_rn(__fsub_rn(cyp, cym), 0.5f);
        const float ds = __fmul_rn(__fsub_rn(nc, pc), 0.5f);
        const float c2 = __fmul_rn(2.0f, c);
        const float dxx = __fsub_rn(__fadd_rn(cxp, cxm), c2);
        const float dyy = __fsub_rn(__fadd_rn(cyp, cym), c2);
        const float dss = __fsub_rn(__fadd_rn(nc, pc), c2);
        const float dxy = __fmul_rn(__fadd_rn(__fsub_rn(__fsub_rn(layer(g1, g2, down + 1), layer(g1, g2, down - 1)),
                                                        layer(g1, g2, up + 1)),
                                              layer(g1, g2, up - 1)),
                                    0.25f);
        const float dxs = __fmul_rn(__fsub_rn(__fsub_rn(layer(g2, g3, 1), layer(g2, g3, -1)),
                                              __fsub_rn(layer(g0, g1, 1), layer(g0, g1, -1))),
                                    0.25f);
        const float dys = __fmul_rn(__fsub_rn(__fsub_rn(layer(g2, g3, down), layer(g2, g3, up)),
                                              __fsub_rn(layer(g0, g1, down), layer(g0, g1, up))),
                                    0.25f);
        const float hm[3][3] = {{dxx, dxy, dxs}, {dxy, dyy, dys}, {dxs, dys, dss}};
        const float g[3] = {-dx, -dy, -ds};
        float off[3];
        if (!solve3(hm, g, off)) return false;
        if (fabsf(off[0]) < 0.5f && fabsf(off[1]) < 0.5f && fabsf(off[2]) < 0.5f) {
            const float lin = __fadd_rn(__fadd_rn(__fmul_rn(dx, off[0]), __fmul_rn(dy, off[1])), __fmul_rn(ds, off[2]));
            const float val = __fadd_rn(c, __fmul_rn(0.5f, lin));
            if (fabsf(val) < rp.contrast_threshold) return false;
            const float tr = __fadd_rn(dxx, dyy);
            const float trace_sq = __fmul_rn(tr, tr);
            const float det = __fsub_rn(__fmul_rn(dxx, dyy), __fmul_rn(dxy, dxy));
            if (det <= 0.0f) return false;
            const float ratio = __fdiv_rn(trace_sq, det);
            if (ratio >= rp.edge_ratio) return false;
            const float lf = __fadd_rn((float)cl, off[2]);
            const float e = __fadd_rn((float)o, __fdiv_rn(lf, (float)rp.S));
            const float p2 = (float)exp2((double)e);
            out->x = __fmul_rn(__fadd_rn((float)cx, off[0]), scale);
            out->y = __fmul_rn(__fadd_rn((float)cy, off[1]), scale);
            out->size = __fmul_rn(rp.sigma, p2);
            out->angle = 0.0f;
            out->response = val;
            out->octave = entry;
            out->layer = rust_as_i32(roundf(lf));
            return true;
        }
        cx = rust_as_i32(roundf(__fadd_rn((float)cx, off[0])));
        cy = rust_as_i32(roundf(__fadd_rn((float)cy, off[1])));
        cl = rust_as_i32(roundf(__fadd_rn((float)cl, off[2])));
        if (cl < 0 || cl >= nl) return false;
    }
    return false;
}

// The candidates of entries e0 .. e0 + n_e - 1 (whose mask words are
// consecutive; w counts from the first entry's first word) in (entry, layer, y,
// x) order, and their refinement. A CTA takes a tile of words: the counts of
// the tiles before it give its first slot, the words' bits go to a list in
// shared memory in order, then one thread per candidate writes its slot (a
// candidate's octave field holds its entry) and refines it. The survivors are
// counted per warp into oc->n_ref (a count, order-free).
//
// Latency bounds it (a chain of dependent scattered reads per candidate and
// step), so the tiles are small: 512 words, some 50 candidates of a dense
// frame, make 380 CTAs of a 1080p octave 0. A scan of the word counts with
// look-back, a kernel that emitted and one that refined took 12.7 + 5.9 + 20 us
// there and 30 + 17 + 60 us at 4096 x 4096, this one at first 20 and 54 us
// (cold caches; the stage with the mask 123 -> 91 us at 1080p, 410 -> 351 at
// 4096 x 4096; a 160 x 120 frame, end to end, 136 -> 122). Without the clamps of
// its 38 reads a step, and with 28 of them, the stage went from 79 to 71 and
// from 231 to 210 us.
constexpr int kCandThreads = 128, kCandWords = kWordTile / kCandThreads;
constexpr uint32_t kCandList = 1024;  // candidates at a time
static_assert(kWordTile * 32 <= 1 << 16, "a bit's index in its tile has 16 bits");
__global__ void __launch_bounds__(kCandThreads) k_candidates(
    const uint8_t* __restrict__ u8arena, const float* __restrict__ lut255, EntryTable tab, RefineParams rp, int e0,
    int n_e, long long n_words, const uint32_t* __restrict__ words, const uint32_t* __restrict__ tiles,
    uint32_t n_tiles, uint32_t* __restrict__ cand_off, Keypoint* __restrict__ cands,
    Keypoint* __restrict__ refined_at, uint32_t* __restrict__ keep, uint32_t cap, Counters* __restrict__ ctr,
    OctCounters* __restrict__ oc) {
    chain_wait();
    __shared__ float lut[256];
    __shared__ uint16_t list[kCandList];
    __shared__ uint32_t buf[kCandThreads / 32];
    const int tid = threadIdx.x;
    for (int v = tid; v < 256; v += kCandThreads) lut[v] = lut255[v];
    const long long base0 = tab.ents[e0].word_base;
    uint32_t base = 0, from = 0, kept = 0;
    for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        base += tiles_sum<kCandThreads>(tiles, from, t, buf);  // (and lut and list are free to use)
        from = t;
        const uint32_t count = tiles[t];
        if (t == n_tiles - 1 && tid == 0) oc->n_cand = base + count;
        if (count == 0 && !cand_off) continue;
        const long long w0 = (long long)t * kWordTile, mine = w0 + tid * kCandWords;
        uint32_t v[kCandWords], s = 0;
#pragma unroll
        for (int k = 0; k < kCandWords; ++k) {
            v[k] = mine + k < n_words ? words[mine + k] : 0u;
            s += __popc(v[k]);
        }
        const uint32_t ex = block_exclusive<kCandThreads>(s, buf);
        if (cand_off) {
            uint32_t at = base + ex;
#pragma unroll
            for (int k = 0; k < kCandWords; ++k) {
                if (mine + k < n_words) cand_off[mine + k] = at;
                at += __popc(v[k]);
            }
        }
        for (uint32_t first = 0; first < count; first += kCandList) {
            uint32_t at = ex - first;  // (wraps below first)
#pragma unroll
            for (int k = 0; k < kCandWords; ++k)
                for (uint32_t m = v[k]; m; m &= m - 1u, ++at)
                    if (at < kCandList) list[at] = (uint16_t)((tid * kCandWords + k) * 32 + __ffs(m) - 1);
            __syncthreads();
            const uint32_t n = min(count - first, kCandList);
            for (uint32_t j = tid; j < n; j += kCandThreads) {
                const uint32_t ci = base + first + j;
                if (ci >= cap) {
                    atomicOr(&ctr->overflow, 1u);
                    break;
                }
                const long long w = w0 + (list[j] >> 5);
                int lo = 0, hi = n_e;  // the last entry whose first word is <= w
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (tab.ents[e0 + mid].word_base - base0 <= w) lo = mid; else hi = mid;
                }
                const int e = e0 + lo;
                const OctaveDev od = tab.ents[e];
                const DogFromU8 dog{u8arena + od.u_off, lut, od.plane, od.pitch, od.W, od.H};
                const long long we = w - (od.word_base - base0);
                const uint32_t row = we >> 32 ? (uint32_t)(we / od.nw) : (uint32_t)we / (uint32_t)od.nw;
                const uint32_t layer = row / (uint32_t)od.H;
                const int x = (int)((uint32_t)we - row * (uint32_t)od.nw) * 32 + (list[j] & 31);
                const int y = (int)(row - layer * (uint32_t)od.H), sc = (int)layer + 1;
                const float scale = __int_as_float((127 + od.octave) << 23);
                Keypoint k;
                k.x = __fmul_rn(__fadd_rn((float)x, 0.5f), scale);
                k.y = __fmul_rn(__fadd_rn((float)y, 0.5f), scale);
                k.size = 0.0f;
                k.angle = 0.0f;
                k.response = dog.at(sc, x, y);
                k.octave = e;
                k.layer = sc;
                cands[ci] = k;
                Keypoint r;
                const bool ok = refine_one(dog, od.octave, e, x, y, sc, rp, &r);
                if (ok) refined_at[ci] = r;
                keep[ci] = ok ? 1u : 0u;
                kept += ok;
            }
            __syncthreads();
        }
    }
    kept = __reduce_add_sync(0xffffffffu, kept);
    if ((tid & 31) == 0 && kept) atomicAdd(&oc->n_ref, kept);
}

// Debug read-back of DoG layer l of octave o as a dense W x H f32 plane, each
// value formed by DogFromU8::at, the function the candidate emission and the
// refinement read DoG through (u8 planes and the v / 255 table in device
// memory). Not part of a run.
__global__ void k_dog_dense(const uint8_t* __restrict__ u8arena, const float* __restrict__ lut255, PyramidDev pyr,
                            int o, int l, float* __restrict__ out) {
    chain_wait();
    const OctaveDev& od = pyr.oct[o];
    const DogFromU8 dog{u8arena + od.u_off, lut255, od.plane, od.pitch, od.W, od.H};
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x < od.W && y < od.H) out[(long long)y * od.W + x] = dog.at(l, x, y);
}

}  // namespace

// ---- launchers -------------------------------------------------------------

int launch_dog_dense(const uint8_t* u8arena, const float* lut255, const PyramidDev& pyr, int o, int l, float* out,
                     cudaStream_t st) {
    const OctaveDev& od = pyr.oct[o];
    if (od.W <= 0 || od.H <= 0) return 0;
    dim3 grid((od.W + 127) / 128, od.H);
    if (launch_chained(k_dog_dense, grid, 128, 0, st, u8arena, lut255, pyr, o, l, out) != cudaSuccess) return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

static size_t extrema_smem(int S) { return sizeof(uint32_t) * (size_t)(S + 2) * kExSH * kExSW; }

int launch_extrema_mask(const uint8_t* u8arena, const EntryTable& tab, const OctaveDev& od,
                        int e, int border, uint32_t* words, uint32_t* tiles, cudaStream_t st) {
    if (od.W <= 0 || od.H <= 0) return 0;
    if (tab.S + 2 > kExMaxLayers) return -1;
    dim3 grid((od.W + kExTX - 1) / kExTX, (od.H + kExTY - 1) / kExTY);
    const size_t smem = extrema_smem(tab.S);
    void (*k)(const uint8_t*, EntryTable, int, int, uint32_t*, long long, uint32_t*) =
        tab.S == 3 ? k_extrema_mask<5> : (tab.S == 4 ? k_extrema_mask<6> : k_extrema_mask<0>);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return -1;
    if (launch_chained(k, grid, kExThreads, smem, st, u8arena, tab, e, border, words, od.word_base, tiles) !=
        cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

int extrema_tiles(int W, int H) {
    return W > 0 && H > 0 ? ((W + kExTX - 1) / kExTX) * ((H + kExTY - 1) / kExTY) : 0;
}

int launch_extrema_mask_flat(const uint8_t* u8arena, const EntryTable& tab, int e0, int n_e,
                             const uint32_t* tile_pref, uint32_t n_tiles, int border, uint32_t* words,
                             uint32_t* tiles, cudaStream_t st) {
    if (n_tiles == 0) return 0;
    if (tab.S + 2 > kExMaxLayers) return -1;
    const size_t smem = extrema_smem(tab.S);
    void (*k)(const uint8_t*, EntryTable, int, int, const uint32_t*, int, uint32_t*, long long, uint32_t*) =
        tab.S == 3 ? k_extrema_mask_flat<5> : (tab.S == 4 ? k_extrema_mask_flat<6> : k_extrema_mask_flat<0>);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return -1;
    if (launch_chained(k, n_tiles, kExThreads, smem, st, u8arena, tab, e0, n_e, tile_pref, border, words, 0ll, tiles) !=
        cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

int launch_candidates(const uint8_t* u8arena, const float* lut255, const EntryTable& tab, float sigma, float contrast,
                      float edge, int e0, int n_e, long long n_words, const uint32_t* words, const uint32_t* tiles,
                      uint32_t* cand_off, Keypoint* cands, Keypoint* refined_at, uint32_t* keep, uint32_t cap,
                      Counters* ctr, OctCounters* oc, cudaStream_t st) {
    if (n_words <= 0) return 0;
    const float e1 = edge + 1.0f;
    const RefineParams rp{sigma, contrast, e1 * e1 / edge, tab.S, tab.S + 2};
    const size_t n_tiles = word_tiles(n_words);
    // a CTA per tile; of a very long list several, so that the sums over the
    // tiles before stay a small part of the reads
    const unsigned grid = (unsigned)std::min<size_t>(n_tiles, 8192);
    if (launch_chained(k_candidates, grid, kCandThreads, 0, st, u8arena, lut255, tab, rp, e0, n_e, n_words, words,
                       tiles, (uint32_t)n_tiles, cand_off, cands, refined_at, keep, cap, ctr, oc) != cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace sift
