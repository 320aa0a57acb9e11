// level_tc.cuh — one Gaussian level on the tensor cores, bit for bit the
// reference's (radii up to 28).
//
// The reference truncates an f32 sum of rounded products to u8 after each of
// the two passes. Only that integer is kept, so it is enough to know the sum
// to within its distance from the next integer: both passes are contractions
// of u8 pixels with a band of whole-number weights (two limbs, tables.cpp:
// tc_blur), which mma.sync sums exactly in its f32 accumulators; the pixels
// whose exact sum lies within the reference's own rounding error of an
// integer (a few in 10^4) are summed again in the reference's order. No
// rounding of the tensor core enters: every partial sum is a whole number
// below 2^24 (in units of 2^-24, see below).
//
// Why mma.sync and not tcgen05: the band is 7 to 57 taps wide, so a 16 x 8
// tile needs a 16 to 64-deep contraction, while a 128-row tcgen05 tile would
// contract 128 + 2 r deep for the same taps, five to ten times the work, and
// return its sums through tensor memory. Measured: 8.7 cycles per
// m16n8k16 and scheduler, 593 TFLOP/s.
//
// A CTA makes a 64 x TY tile: the clamp-to-edge window of the previous
// level's bytes goes to shared memory zero-extended to 16 bits, which read as
// f16 are the subnormals v 2^-24, so no conversion is needed (products and
// sums keep the factor exactly); the horizontal pass reads it with ldmatrix
// as the A operand (rows x window) against the band as B, and writes its u8
// results in the same 16-bit form; the vertical pass has the band as A and
// reads the horizontal result transposed by ldmatrix as B. The accumulators'
// start value puts the sum into the mantissa as fixed point, so the integer
// and the fraction are bit fields of the result.
//
// Bound: instruction issue and the latency around its two barriers (45 % of
// issue slots, 20 % of the tensor cycles at 4096 x 4096), which a sum in the
// reference's order lengthens: with none at all a 1080p frame's levels would
// take 119 us instead of 139. So the error bound is kept tight (half an ulp of
// each partial sum, tables.cpp; relative to 255 and rounded up to a power of
// two, three times as many sums were near, 157 us with the next) and the taps
// are in shared memory (read from the L2 cache at the first such sum, 150 us).
// Measured against
// the scalar kernel it replaced (one rounded multiply and add per tap):
// a 4096 x 4096 level of radius 4, 48.1 -> 34.0 us (40 -> 18.5 M warp
// instructions); radius 13 on 2048 x 2048 (two passes before), 36 -> 18 us;
// radius 20 on 480 x 270, 10.3 -> 9 us; a 160 x 120 frame's pyramid,
// 153 -> 97 us.
#pragma once

#include "sift_internal.cuh"

namespace sift {

// The taps of one blur (tables.h: TcBlur) as the kernel takes them.
struct TcParams {
    const uint4* frags;  // kh x 32 lanes, then kv x 32 lanes x 2
    const float* wts;    // the f32 taps
    int r;
    float init_a, init_b, scale_b, whole;
    uint32_t near;
};

namespace tc {

constexpr int kTX = 64;
constexpr int kThreads = 256;
constexpr int kTaps = 64;  // (57 at most)
constexpr int kHS = 72;  // row stride of the horizontal result (halves): 9 x 16 bytes, ldmatrix rows in distinct banks

// P: columns staged left and right of the tile; PV: rows above and below.
template <int P, int PV, int TY>
struct Shape {
    static constexpr int KH = (8 + 2 * P) / 16, KV = (16 + 2 * PV) / 16;
    static constexpr int RH = TY + 2 * PV;   // rows of the horizontal pass
    static constexpr int SW = kTX + 2 * P;   // staged row (halves), an odd multiple of 8
    static constexpr size_t smem = sizeof(uint16_t) * ((size_t)RH * SW + (size_t)RH * kHS) + sizeof(float) * kTaps;
    static_assert((8 + 2 * P) % 16 == 0 && (16 + 2 * PV) % 16 == 0 && RH % 16 == 0 && (SW / 8) % 2 == 1, "tile shape");
};

// d = a b + c
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1,
                                         const float* c) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

// The reference's sum of one output over `taps` staged values `step` halves
// apart: products and sums rounded one by one in tap order, truncated to u8.
__device__ __noinline__ uint32_t exact_tap_sum(const uint16_t* p, int step, const float* wts, int taps) {
    float s = 0.0f;
    for (int i = 0; i < taps; ++i, p += step) s = __fadd_rn(s, __fmul_rn((float)*p, wts[i]));
    return (uint32_t)clamp_u8(s);
}

// Four sums of a lane (accumulators of the two limbs) to whole numbers: byte 0
// of v[j] (byte 1 is 0). True if a lane of the warp has a sum that the fixed
// point does not decide; m is this lane's mask of them. A sum below 1 is
// always 0: the reference's sums are not negative (black areas stay on the
// fast path).
template <bool CLAMP>
__device__ __forceinline__ bool to_bytes(const float (&ca)[4], const float (&cb)[4], const TcParams& tp,
                                         uint32_t (&v)[4], uint32_t& m) {
    constexpr int kWhole = CLAMP ? 18 : 17;  // bits above the fraction
    uint32_t b[4], frac[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float s = __fmaf_rn(cb[j], tp.scale_b, ca[j]);
        b[j] = __float_as_uint(s);
        frac[j] = b[j] << kWhole;
        // the whole part to the low mantissa bits by an addition that truncates
        v[j] = __float_as_uint(__fadd_rz(s, tp.whole));
        if (CLAMP) v[j] = min(v[j] & 0x1ffu, 255u);
    }
    if (!__any_sync(0xffffffffu, min(min(frac[0], frac[1]), min(frac[2], frac[3])) < tp.near)) return false;
    const uint32_t one = __float_as_uint(tp.init_a) + (1u << (32 - kWhole));
    m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (frac[j] < tp.near && b[j] >= one) m |= 1u << j;
    return true;
}

// Four pixels of a level, from their bytes, in the level's own storage.
__device__ __forceinline__ void store_level_word(uint8_t*, uint32_t) {}  // u8 storage: the level is its u8 plane
__device__ __forceinline__ void store_level_word(float* p, uint32_t w) {
    *reinterpret_cast<float4*>(p) = make_float4(div255(float_of_byte<0>(w)), div255(float_of_byte<1>(w)),
                                                div255(float_of_byte<2>(w)), div255(float_of_byte<3>(w)));
}
__device__ __forceinline__ void store_level_word(__half* p, uint32_t w) {
    // v as f16: the bits 0x6400 + v are 1024 + v
    const __half2 k = __halves2half2(__ushort_as_half(0x6400), __ushort_as_half(0x6400));
    const uint32_t a = __byte_perm(w, 0x64u, 0x4140u), b = __byte_perm(w, 0x64u, 0x4342u);
    const __half2 lo = __hsub2(*reinterpret_cast<const __half2*>(&a), k), hi = __hsub2(*reinterpret_cast<const __half2*>(&b), k);
    *reinterpret_cast<uint2*>(p) =
        make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// The tile at (x0, y0) of a W x H level; in and out rows start on 4 bytes.
template <typename TG, int P, int PV, int TY, bool CLAMP>
__device__ __forceinline__ void level_tile(const uint8_t* __restrict__ in, int in_pitch, TG* __restrict__ out,
                                           uint8_t* __restrict__ out_u8, int pitch, int W, int H, const TcParams& tp,
                                           int x0, int y0, uint16_t* sm) {
    using S = Shape<P, PV, TY>;
    uint16_t* src = sm;
    uint16_t* hs = sm + S::RH * S::SW;
    float* wts = reinterpret_cast<float*>(hs + S::RH * kHS);  // the taps
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    if (tid < 2 * tp.r + 1) wts[tid] = tp.wts[tid];
    // Stage: a row is SW / 4 words of 4 pixels, one per lane; warp w takes
    // rows w, w + 8, .. with all their loads in flight. Words outside the row
    // repeat its first or last pixel (a byte permute with the lane's
    // selector); the last word may read up to 3 bytes past the row's end,
    // inside the aligned word that holds its last pixel.
    {
        constexpr int kWords = S::SW / 4, kRows = S::RH / 8;
        static_assert(kWords <= 32, "one word per lane");
        if (lane < kWords) {
            const int x = x0 - P + 4 * lane;
            uint32_t w[kRows];
            if (x0 >= P && x0 + kTX + P <= W && y0 >= PV && y0 + TY + PV <= H) {
                const uint8_t* p = in + (long long)(y0 - PV + warp) * in_pitch + x;
                const long long step = 8ll * in_pitch;
#pragma unroll
                for (int i = 0; i < kRows; ++i, p += step) w[i] = *reinterpret_cast<const uint32_t*>(p);
            } else {
                const int xw = clampi(x, 0, (W - 1) & ~3);
                uint32_t sel = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) sel |= (uint32_t)(clampi(x + k, 0, W - 1) - xw) << (4 * k);
#pragma unroll
                for (int i = 0; i < kRows; ++i) {
                    const int y = clampi(y0 - PV + warp + 8 * i, 0, H - 1);
                    w[i] = *reinterpret_cast<const uint32_t*>(in + (long long)y * in_pitch + xw);
                }
#pragma unroll
                for (int i = 0; i < kRows; ++i) w[i] = __byte_perm(w[i], 0u, sel);
            }
            uint16_t* d = src + warp * S::SW + 4 * lane;
#pragma unroll
            for (int i = 0; i < kRows; ++i)
                *reinterpret_cast<uint2*>(d + i * 8 * S::SW) =
                    make_uint2(__byte_perm(w[i], 0u, 0x4140u), __byte_perm(w[i], 0u, 0x4342u));
        }
    }
    const float ia[4] = {tp.init_a, tp.init_a, tp.init_a, tp.init_a}, ib[4] = {tp.init_b, tp.init_b, tp.init_b, tp.init_b};
    // horizontal pass: warp w makes columns 8 w .. 8 w + 7 of every row
    {
        uint4 bf[S::KH];
#pragma unroll
        for (int k = 0; k < S::KH; ++k) bf[k] = tp.frags[k * 32 + lane];
        __syncthreads();
        // lane l addresses row l & 15, half l >> 4 of a 16 x 16 block
        const uint32_t a0 = (uint32_t)__cvta_generic_to_shared(src + (lane & 15) * S::SW + 8 * warp + 8 * (lane >> 4));
        uint16_t* h = hs + g * kHS + 8 * warp + 2 * t;
#pragma unroll
        for (int mb = 0; mb < S::RH / 16; ++mb, h += 16 * kHS) {
            float ca[4], cb[4];
#pragma unroll
            for (int k = 0; k < S::KH; ++k) {
                uint32_t a[4];
                ldsm4(a, a0 + (uint32_t)(mb * 16 * S::SW + 16 * k) * 2u);
                mma16816(ca, a, bf[k].x, bf[k].y, k ? ca : ia);
                mma16816(cb, a, bf[k].z, bf[k].w, k ? cb : ib);
            }
            uint32_t v[4], m;
            const bool some = to_bytes<CLAMP>(ca, cb, tp, v, m);
            // (row g, columns 2t, 2t+1) and (row g + 8, the same)
            *reinterpret_cast<uint32_t*>(h) = __byte_perm(v[0], v[1], 0x5410u);
            *reinterpret_cast<uint32_t*>(h + 8 * kHS) = __byte_perm(v[2], v[3], 0x5410u);
            if (some) {
                while (m) {
                    const int j = __ffs(m) - 1;
                    m &= m - 1u;
                    const int dy = 8 * (j >> 1), dx = j & 1;
                    h[dy * kHS + dx] = (uint16_t)exact_tap_sum(
                        src + (mb * 16 + g + dy) * S::SW + 8 * warp + 2 * t + dx + P - tp.r, 1, wts, 2 * tp.r + 1);
                }
                __syncwarp();
            }
        }
    }
    // vertical pass: a warp makes 16 rows of NB blocks of 8 columns
    constexpr int kMB = TY / 16, NB = TY / 16;  // 8 warps: kMB row blocks x 8 / kMB column groups
    static_assert(NB == 2 || NB == 4, "tile height");
    const int mb = warp % kMB, c0 = 8 * NB * (warp / kMB);
    float ca[NB][4], cb[NB][4];
    // lane l addresses row l & 15 of columns 8 (l >> 4) .. of a 16 x 16 block
    const uint32_t b0 = (uint32_t)__cvta_generic_to_shared(hs + (mb * 16 + (lane & 15)) * kHS + c0 + 8 * (lane >> 4));
    {
        const uint4* vf = tp.frags + S::KH * 32 + 2 * lane;
        uint4 fa = vf[0], fb = vf[1];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < S::KV; ++k) {
            const uint32_t wa[4] = {fa.x, fa.y, fa.z, fa.w}, wb[4] = {fb.x, fb.y, fb.z, fb.w};
            if (k + 1 < S::KV) {
                fa = vf[(k + 1) * 64];
                fb = vf[(k + 1) * 64 + 1];
            }
#pragma unroll
            for (int nb = 0; nb < NB; nb += 2) {
                uint32_t r[4];
                ldsm4t(r, b0 + (uint32_t)(k * 16 * kHS + 8 * nb) * 2u);
                mma16816(ca[nb], wa, r[0], r[1], k ? ca[nb] : ia);
                mma16816(cb[nb], wb, r[0], r[1], k ? cb[nb] : ib);
                mma16816(ca[nb + 1], wa, r[2], r[3], k ? ca[nb + 1] : ia);
                mma16816(cb[nb + 1], wb, r[2], r[3], k ? cb[nb + 1] : ib);
            }
        }
    }
    // Block nb of a lane: rows g and g + 8, columns 2t, 2t + 1. Neighbouring
    // lanes exchange so that even lanes hold 4 columns of row g and odd lanes
    // of row g + 8, then the quad's halves so that a lane holds 4 NB
    // neighbouring columns.
    const int odd = t & 1, high = t >> 1;
    uint32_t w[NB];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
        uint32_t v[4], m;
        const bool some = to_bytes<CLAMP>(ca[nb], cb[nb], tp, v, m);
        uint32_t p = __byte_perm(__byte_perm(v[0], v[1], 0x0040u), __byte_perm(v[2], v[3], 0x0040u), 0x5410u);
        if (some) {
            while (m) {
                const int j = __ffs(m) - 1;
                m &= m - 1u;
                const int dy = 8 * (j >> 1), dx = j & 1;
                const uint32_t e = exact_tap_sum(
                    hs + (mb * 16 + g + dy + PV - tp.r) * kHS + c0 + 8 * nb + 2 * t + dx, kHS, wts, 2 * tp.r + 1);
                p = (p & ~(0xffu << (8 * j))) | e << (8 * j);
            }
            __syncwarp();
        }
        const uint32_t q = __shfl_xor_sync(0xffffffffu, p, 1);
        w[nb] = __byte_perm(p, q, odd ? 0x3276u : 0x5410u);  // columns 4 high .. of block nb
    }
    uint32_t row[NB];
#pragma unroll
    for (int i = 0; i < NB / 2; ++i) {
        // lanes of the low half keep blocks 0 .. NB/2 - 1, of the high half the others
        const uint32_t keep = high ? w[NB / 2 + i] : w[i], give = high ? w[i] : w[NB / 2 + i];
        const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 2);
        row[2 * i] = high ? got : keep;
        row[2 * i + 1] = high ? keep : got;
    }
    const int y = y0 + mb * 16 + g + 8 * odd, x = x0 + c0 + 4 * NB * high;
    if (y >= H || x >= W) return;
    const long long o = (long long)y * pitch + x;
    // the last columns may end in the row's padding (the pitch is a multiple of 32)
    if constexpr (NB == 4)
        *reinterpret_cast<uint4*>(out_u8 + o) = make_uint4(row[0], row[1], row[2], row[3]);
    else
        *reinterpret_cast<uint2*>(out_u8 + o) = make_uint2(row[0], row[1]);
#pragma unroll
    for (int i = 0; i < NB; ++i) store_level_word(out + o + 4 * i, row[i]);
}

}  // namespace tc
}  // namespace sift
