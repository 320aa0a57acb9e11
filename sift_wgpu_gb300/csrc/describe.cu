// describe.cu — orientation assignment and 4x4x8 descriptors (sm_103a).
//
// Stages (d) and (e) of the hot path: assign_orientations
// (src/sift.rs:605-726) and compute (src/sift.rs:917-1060) with
// normalize_and_clip_descriptor (src/sift.rs:889-913).
//
//   k_orientation   one warp per refined keypoint (orient_one): the (2r+1)^2
//                   window is split over the lanes, each lane takes its samples
//                   four at a time and adds them into its own column of a
//                   bin-major shared histogram (conflict-free, no atomics),
//                   columns are summed in a fixed order, then the two [1,1,1]/3
//                   smoothing passes and the peak test run one bin per lane;
//                   peaks come out in bin order through a ballot.
//   k_descriptor    one CTA per oriented keypoint (describe_one): the bilinear
//                   samples of the window are computed once into a shared grid,
//                   pairs of window samples are split over the threads and
//                   evaluated on packed f32x2 arithmetic, trilinear
//                   contributions are added into 128 shared bins as u32 fixed
//                   point (integer addition is associative, so the result does
//                   not depend on scheduling), then L2 normalise, clip at 0.2,
//                   renormalise.
// Both queues run from the last item of an octave's list (the largest
// windows first).
//
// The orientation histogram follows the reference's f32 operation order
// without FMA, except the Gaussian weight (hardware exponential of a
// reciprocal product); every bin index is exact (a table over the byte
// differences);
// its column sums are in a fixed order. The descriptor loop trades exactness
// for speed within the descriptor tolerance (see describe_one). Orientations
// and descriptors therefore agree with the reference within rounding, not bit
// for bit.
#include <algorithm>
#include <type_traits>

#include "sift_internal.cuh"

namespace sift {
namespace {

constexpr int kOriWarps = 8;  // orientation: one keypoint per warp

// Work-queue kernels launch more CTAs than fit on the device. A CTA (or an
// orientation warp) below persist_from takes at most kBudget items and
// retires, which frees its slot for kernels of more urgent streams (the
// smaller octaves' chains) instead of holding it until the queue drains; the
// CTAs from persist_from on, the last wave, loop until the queue is empty,
// so every item is taken whatever the grid.
constexpr int kOriBudget = 4;   // keypoints per warp
constexpr int kDescBudget = 2;  // keypoints per CTA

// One level of the u8 arena. Every storage mode keeps it, and both stages here
// read it whatever else is stored: it is the smallest and the fastest to read,
// and v / 255 (div255, the IEEE quotient) is the f32 mode's stored value.
struct GaussPlane {
    const uint8_t* base;
    int pitch, W, H;
    // get_gauss_pixel_value (src/sift.rs:218-223)
    __device__ __forceinline__ uint32_t at(int x, int y) const {
        return base[(long long)clampi(y, 0, H - 1) * pitch + clampi(x, 0, W - 1)];
    }
    __device__ __forceinline__ float px(int x, int y) const { return div255((float)at(x, y)); }
    // the same as v itself (0..255): the descriptor's histogram is
    // L2-normalised, so the factor 255 cancels
    __device__ __forceinline__ float px_raw(int x, int y) const { return (float)at(x, y); }
    // get_gauss_pixel_bilinear (src/sift.rs:238-266)
    __device__ __forceinline__ float bilinear(float x, float y) const {
        const float xf = floorf(x), yf = floorf(y);
        const float xc = __fadd_rn(xf, 1.0f), yc = __fadd_rn(yf, 1.0f);
        const float dx = __fsub_rn(x, xf), dy = __fsub_rn(y, yf);
        const int x0 = rust_as_i32(xf), y0 = rust_as_i32(yf), x1 = rust_as_i32(xc), y1 = rust_as_i32(yc);
        const float q11 = px(x0, y0), q21 = px(x1, y0), q12 = px(x0, y1), q22 = px(x1, y1);
        const float omx = __fsub_rn(1.0f, dx), omy = __fsub_rn(1.0f, dy);
        float v = __fmul_rn(__fmul_rn(q11, omx), omy);
        v = __fadd_rn(v, __fmul_rn(__fmul_rn(q21, dx), omy));
        v = __fadd_rn(v, __fmul_rn(__fmul_rn(q12, omx), dy));
        v = __fadd_rn(v, __fmul_rn(__fmul_rn(q22, dx), dy));
        return v;
    }
};

__device__ __forceinline__ GaussPlane plane_for(const uint8_t* u8arena, const OctaveDev& od, int S, int layer) {
    return GaussPlane{u8arena + od.u_off + (long long)clampi(layer, 0, S + 2) * od.plane, od.pitch, od.W, od.H};
}

// ---------------------------------------------------------------------------
// Orientation. Every storage mode keeps the levels as u8 planes, which this
// stage reads: a gradient is a pair of differences of bytes, and its bin of
// the 36 (src/sift.rs:652-656) depends on that pair alone. kBinSide^2 bins,
// one for each pair, are made once (k_ori_bins): off the axes every
// difference pair's angle is at least 6.4e-5 bins from a bin edge, above the
// f32 rounding of the reference's sequence (the differences of the two
// v / 255, atan2f, the wrap and the division: below 2e-5 bins), so the f64
// angle decides; on the axes the f32 sequence gives the bins 0, 9, 18 and 26
// (3/2 pi times 36 over 2 pi rounds below 27). A lookup replaces the
// arctangent polynomial, the edge test and its exact path; with it, the
// window's integer addressing, four samples in flight per lane, the row
// prefetch and the smoothing in registers took the octave-0 launch from 50 to
// 40 us at 1080p (43 -> 24 M warp instructions) and from 380 to 256 us at
// 4096 x 4096, where it issues 2.4 instructions a cycle and SM, bound by
// issue and the latency of the byte loads together.
constexpr int kBinSide = 512;  // differences -256 .. 255
// The table in tiles of 16 x 8 differences, a cache line each: most pairs of a
// warp's samples are small, and fall into a few lines instead of one for each
// vertical difference: the octave-0 launch 40 -> 37.4 us at 1080p, the stage
// 358 -> 337 us at 4096 x 4096. (Making v / 255 in registers instead of reading
// it from shared memory halves that pipe's work and takes 347.) (x, y) =
// differences + 256.
__device__ __forceinline__ uint32_t bin_at(uint32_t x, uint32_t y) {
    return x + (x >> 4) * 112u + y * 16u + (y >> 3) * (8u * kBinSide - 128u);
}

__global__ void __launch_bounds__(kBinSide) k_ori_bins(uint8_t* __restrict__ bins) {
    chain_wait();
    const int dx = (int)threadIdx.x - kBinSide / 2, dy = (int)blockIdx.x - kBinSide / 2;
    int b;
    if (dy == 0) {
        b = dx < 0 ? 18 : 0;
    } else if (dx == 0) {
        b = dy > 0 ? 9 : 26;
    } else {
        const double two_pi = 6.283185307179586476925;
        const double a = atan2((double)dy, (double)dx);
        b = (int)((a < 0.0 ? a + two_pi : a) * (double)kOriBins / two_pi);
    }
    bins[bin_at(threadIdx.x, blockIdx.x)] = (uint8_t)b;
}

// The tables of the orientation stage: v / 255 (shared memory) and the bins.
struct OriTables {
    const float* lut;
    const uint8_t* bins;
};

// The four neighbours of a sample's pixel, as bytes.
struct OriBytes {
    uint32_t right, left, below, above;
};

// One sample (src/sift.rs:640-662): its bin and its share, the magnitude
// times the Gaussian weight at window offset (fdx, fdy).
struct OriSample {
    uint32_t bin;
    float v;
};
__device__ __forceinline__ OriSample ori_sample(const OriBytes& p, float fdx, float fdy, float inv_wd,
                                                const OriTables& tb) {
    OriSample s;
    s.bin = tb.bins[bin_at(p.right - p.left + kBinSide / 2, p.below - p.above + kBinSide / 2)];
    const float gx = __fsub_rn(tb.lut[p.right], tb.lut[p.left]), gy = __fsub_rn(tb.lut[p.below], tb.lut[p.above]);
    // the hardware square root (within an ulp; the bins are sums whose
    // order differs from the reference's anyway)
    const float mag = sqrt_approx(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)));
    // exp(-(dx^2 + dy^2) / wd) with the quotient as a product by 1 / wd and
    // the hardware exponential: a few ulp from expf of the IEEE quotient,
    // the same order as expf's own distance from the host libm
    const float ex = __fmul_rn(-__fadd_rn(__fmul_rn(fdx, fdx), __fmul_rn(fdy, fdy)), inv_wd);
    const float wgt = ex2_approx(__fmul_rn(ex, 1.4426950408889634f));  // in [e^-10, 1]
    s.v = __fmul_rn(mag, wgt);
    return s;
}

// Two samples, in this order, into the lane's column of the bin-major
// histogram hist[bin][32]: both bins are read at once, the first sum is
// forwarded where they are the same.
__device__ __forceinline__ void ori_add2(const OriSample& a, const OriSample& b, float* hist_lane) {
    float* ha = hist_lane + a.bin * 32;
    float* hb = hist_lane + b.bin * 32;
    const float va = *ha, vb = *hb;
    const float na = __fadd_rn(va, a.v);
    const float nb = __fadd_rn(a.bin == b.bin ? na : vb, b.v);
    *ha = na;
    *hb = nb;
}

// The orientation window of one keypoint (src/sift.rs:640-662), lane-strided:
// sample k = lane + 32 j of the (2r+1)^2 window, row-major, read from the u8
// level. A lane takes its samples kOriStep at a time (k, k + 32, ..: their
// loads in flight together) and adds them to its histogram column in window
// order, as one at a time would; samples past the window or outside the level
// add +0.0, which leaves a bin bit-identical.
// PLAIN: the window is inside the level and every position rounds to the
// keypoint's rounded position plus its offset, so a sample is one offset into
// the plane; else each position is rounded (f32::round of the f32 sum) and
// clamped by itself.
constexpr int kOriStep = 4;
template <bool PLAIN>
__device__ __forceinline__ void ori_window(const uint8_t* __restrict__ u8arena, long long level, int pitch, int W, int H,
                                           float xo, float yo, int r, float wd, float* hist_lane, int lane,
                                           const OriTables& tb) {
    const float inv_wd = __frcp_rn(wd);
    const int side = 2 * r + 1;
    const float side_f = (float)side, r_f = (float)r;
    // Sample k = lane + 32 j is (x, y) = (k % side - r, k / side - r): exact
    // small integers in f32 that advance by fixed amounts per step, with one
    // row wrap (as selects) at most; `off` is its byte offset.
    const float inv_side = rcp_approx(side_f);
    const int q0 = floor_i(((float)lane + 0.5f) * inv_side), dq = floor_i(32.5f * inv_side), dr = 32 - dq * side;
    const float dr_f = (float)dr, dq_f = (float)dq;
    const int doff = dq * pitch + dr, woff = pitch - side;
    float x = (float)(lane - q0 * side) - r_f, y = (float)q0 - r_f;
    // (32-bit offsets from the arena, which PLAIN levels lie within)
    const uint32_t org = (uint32_t)level + (uint32_t)((round_away_i(yo) - r) * pitch + (round_away_i(xo) - r));
    uint32_t off = org + (uint32_t)(q0 * pitch + lane - q0 * side);
    while (y <= r_f) {
        float sx[kOriStep], sy[kOriStep];
        bool in[kOriStep];
        OriBytes p[kOriStep];
#pragma unroll
        for (int u = 0; u < kOriStep; ++u) {
            sx[u] = x;
            sy[u] = y;
            in[u] = y <= r_f;
            if (PLAIN) {
                const uint32_t at = in[u] ? off : org, below = at + (uint32_t)pitch, above = at - (uint32_t)pitch;
                p[u] = OriBytes{(u8arena + 1)[at], (u8arena - 1)[at], u8arena[below], u8arena[above]};
            } else {
                int xi = round_away_i(__fadd_rn(xo, x)), yi = round_away_i(__fadd_rn(yo, y));
                in[u] = in[u] && !(xi < 1 || xi >= W - 1 || yi < 1 || yi >= H - 1);
                xi = clampi(xi, 1, W - 2);
                yi = clampi(yi, 1, H - 2);
                const uint8_t* at = u8arena + level + (long long)yi * pitch + xi;
                p[u] = OriBytes{at[1], at[-1], at[pitch], at[-pitch]};
            }
            // the next sample
            x += dr_f;
            y += dq_f;
            off += (uint32_t)doff;
            const bool w = x > r_f;
            x = w ? x - side_f : x;
            y = w ? y + 1.0f : y;
            off = w ? off + (uint32_t)woff : off;
        }
        OriSample s[kOriStep];
#pragma unroll
        for (int u = 0; u < kOriStep; ++u) {
            s[u] = ori_sample(p[u], sx[u], sy[u], inv_wd, tb);
            s[u].v = in[u] ? s[u].v : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < kOriStep; u += 2) ori_add2(s[u], s[u + 1], hist_lane);
    }
}

// The orientation peaks of one refined keypoint (src/sift.rs:605-726),
// computed by one warp: the window into the warp's bin-major histogram
// hist[36][32], the column sums and the two smoothing passes in registers, the
// peaks in bin order written to angles[0 .. count). Returns the count (the
// same in every lane).
__device__ __forceinline__ uint32_t orient_one(const uint8_t* __restrict__ u8arena, const EntryTable& tab,
                                               const Keypoint& kp, float* hist, int lane,
                                               float* __restrict__ angles, const OriTables& tb) {
    const float two_pi = 2.0f * kPi;
    const float bin_w = 2.0f * kPi / (float)kOriBins;
    const int e = kp.octave;  // entry
    if (!(e >= 0 && e < tab.n)) return 0;
    const OctaveDev od = tab.ents[e];
    const int o = od.octave;
    const long long level = od.u_off + (long long)clampi(kp.layer, 0, tab.S + 2) * od.plane;
    // division by 2^o is the multiplication by 2^-o, exactly
    const float inv_scale = __int_as_float((127 - o) << 23);
    const float xo = __fmul_rn(kp.x, inv_scale), yo = __fmul_rn(kp.y, inv_scale);
    const float so = __fmul_rn(kp.size, inv_scale);
    if (!(so > 0.0f)) return 0;
    const int r = rust_as_i32(roundf(__fmul_rn(4.5f, so)));
    const float ws = __fmul_rn(1.5f, so);
    const float wd = __fmul_rn(__fmul_rn(2.0f, ws), ws);
#pragma unroll
    for (int b = 0; b < kOriBins / 4; ++b)
        reinterpret_cast<float4*>(hist)[b * 32 + lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncwarp();

    // Windows entirely inside the level (most keypoints) take the loop
    // without bounds checks; the others add +0.0 for samples outside, which
    // leaves a bin bit-identical. The plain loop also wants positions well
    // off the rounding edge: an f32 sum xo + dx below 2^16 is within 2^-9 of
    // the exact one, so it rounds to round(xo) + dx.
    const bool interior = xo - (float)r >= 2.5f && xo + (float)r <= (float)(od.W - 3) - 0.5f &&
                          yo - (float)r >= 2.5f && yo + (float)r <= (float)(od.H - 3) - 0.5f;
    const bool plain = interior && level + od.plane < (1ll << 32) && fabsf(xo - floorf(xo) - 0.5f) > 0.0078125f && fabsf(yo - floorf(yo) - 0.5f) > 0.0078125f;
    if (plain) {
        // every row's first and last sector on the way before the first is needed
        const uint8_t* row = u8arena + level + (long long)(round_away_i(yo) - r - 1 + lane) * od.pitch + (round_away_i(xo) - r - 1);
        for (int q = lane; q < 2 * r + 3; q += 32, row += 32ll * od.pitch) {
            asm volatile("prefetch.global.L1 [%0];" ::"l"(row));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(row + 2 * r + 2));
        }
    }
    if (plain)
        ori_window<true>(u8arena, level, od.pitch, od.W, od.H, xo, yo, r, wd, hist + lane, lane, tb);
    else
        ori_window<false>(u8arena, level, od.pitch, od.W, od.H, xo, yo, r, wd, hist + lane, lane, tb);
    __syncwarp();
    // Column sums: bin `lane` in four interleaved partial sums (the column
    // index rotated by the bin keeps the 32 lanes in 32 banks), bins 32..35
    // by eight lanes each and a shuffle tree.
    float h0, h1;
    {
        const float* hb = hist + lane * 32;
        float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll
        for (int l = 0; l < 32; l += 4) {
            s0 = __fadd_rn(s0, hb[(l + lane) & 31]);
            s1 = __fadd_rn(s1, hb[(l + 1 + lane) & 31]);
            s2 = __fadd_rn(s2, hb[(l + 2 + lane) & 31]);
            s3 = __fadd_rn(s3, hb[(l + 3 + lane) & 31]);
        }
        h0 = __fadd_rn(__fadd_rn(s0, s1), __fadd_rn(s2, s3));
        const int bb = 32 + (lane >> 3), c0 = (lane & 7) * 4;
        const float* ht = hist + bb * 32;
        float t = __fadd_rn(__fadd_rn(ht[(c0 + bb) & 31], ht[(c0 + 1 + bb) & 31]),
                            __fadd_rn(ht[(c0 + 2 + bb) & 31], ht[(c0 + 3 + bb) & 31]));
        t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, 1));
        t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, 2));
        t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, 4));
        h1 = __shfl_sync(0xffffffffu, t, 8 * (lane & 3));
    }
    // Bin `lane` is h0, bin 32 + lane of lanes 0..3 is h1; the neighbours on
    // the circle of 36 come by shuffles.
    float p0, n0, p1, n1;
    auto neighbours = [&]() {
        p0 = __shfl_up_sync(0xffffffffu, h0, 1);
        n0 = __shfl_down_sync(0xffffffffu, h0, 1);
        p1 = __shfl_up_sync(0xffffffffu, h1, 1);
        n1 = __shfl_down_sync(0xffffffffu, h1, 1);
        const float last = __shfl_sync(0xffffffffu, h1, kOriBins - 33), mid = __shfl_sync(0xffffffffu, h1, 0);
        const float b31 = __shfl_sync(0xffffffffu, h0, 31), b0 = __shfl_sync(0xffffffffu, h0, 0);
        p0 = lane == 0 ? last : p0;
        n0 = lane == 31 ? mid : n0;
        p1 = lane == 0 ? b31 : p1;
        n1 = lane == kOriBins - 33 ? b0 : n1;
    };
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        neighbours();
        h0 = div3(__fadd_rn(__fadd_rn(p0, h0), n0));
        h1 = div3(__fadd_rn(__fadd_rn(p1, h1), n1));
    }
    neighbours();
    const bool tail = lane < kOriBins - 32;
    // the sums are not negative, so their bits order them
    const float mx = __uint_as_float(
        __reduce_max_sync(0xffffffffu, max(__float_as_uint(h0), tail ? __float_as_uint(h1) : 0u)));
    const float thr = __fmul_rn(mx, 0.8f);
    bool pk[2] = {false, false};
    float pa[2] = {0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float cv = q ? h1 : h0, pv = q ? p1 : p0, nv = q ? n1 : n0;
        pk[q] = (q == 0 || tail) && cv >= thr && cv > pv && cv > nv;
        if (pk[q]) {
            const float den = __fadd_rn(__fsub_rn(pv, __fmul_rn(2.0f, cv)), nv);
            const float off = fabsf(den) > 1e-5f ? __fdiv_rn(__fmul_rn(0.5f, __fsub_rn(pv, nv)), den) : 0.0f;
            const float center = __fmul_rn(__fadd_rn((float)(lane + 32 * q), 0.5f), bin_w);
            const float a = __fadd_rn(center, __fmul_rn(off, bin_w));
            float fa = rem_euclid_2b(a, two_pi);  // a in (0, 2 pi + pi/36)
            if (fa > kPi) fa = __fsub_rn(fa, two_pi);
            pa[q] = fa;
        }
    }
    const uint32_t m0 = __ballot_sync(0xffffffffu, pk[0]);
    const uint32_t m1 = __ballot_sync(0xffffffffu, pk[1]);
    const uint32_t lt = (1u << lane) - 1u;
    if (pk[0]) angles[__popc(m0 & lt)] = pa[0];
    if (pk[1]) angles[__popc(m0) + __popc(m1 & lt)] = pa[1];
    __syncwarp();
    return (uint32_t)(__popc(m0) + __popc(m1));
}

__global__ void __launch_bounds__(32 * kOriWarps, 5) k_orientation(const uint8_t* __restrict__ u8arena, EntryTable tab,
                                                                const float* __restrict__ lut255,
                                                                const uint8_t* __restrict__ bins,
                                                                const Keypoint* __restrict__ refined_at,
                                                                const uint32_t* __restrict__ keep, uint32_t ncap,
                                                                OctCounters* __restrict__ oc,
                                                                float* __restrict__ ori_angle,
                                                                uint32_t* __restrict__ ori_count,
                                                                uint32_t* __restrict__ tiles, int persist_from) {
    chain_wait();
    __shared__ __align__(16) float hist[kOriWarps][kOriBins][32];
    __shared__ float slut[256];
    const int lane = threadIdx.x, wid = threadIdx.y;
    for (int v = wid * 32 + lane; v < 256; v += 32 * kOriWarps) slut[v] = lut255[v];
    __syncthreads();
    const OriTables tb{slut, bins};
    const uint32_t n = min(oc->n_cand, ncap);  // candidate slots; rejected ones get 0 peaks
    const bool persist = (int)blockIdx.x >= persist_from;
    // A warp claims several slots at once where the list gives every resident
    // warp at least four such claims (fewer leave warps idle at the end: 1080p
    // 3 slots a claim 58 us, 1 slot 41 us); it skips the rejected ones (two
    // in five) without a claim each.
    const uint32_t claim = min(max(n / (4u * 152u * 5u * kOriWarps), 1u), (uint32_t)kOriBudget);
    for (uint32_t taken = 0; persist || taken < (uint32_t)kOriBudget; taken += claim) {
        uint32_t i0 = 0;
        if (lane == 0) i0 = atomicAdd(&oc->next_ori, claim);
        i0 = __shfl_sync(0xffffffffu, i0, 0);
        if (i0 >= n) break;
        // from the last slot: the largest windows first
        const uint32_t mine = n - 1 - min(i0 + lane, n - 1);
        const bool valid = lane < (int)claim && i0 + lane < n;
        const bool kept = valid && keep[mine] != 0u;
        if (valid && !kept) ori_count[mine] = 0u;
        for (uint32_t m = __ballot_sync(0xffffffffu, kept); m; m &= m - 1u) {
            const uint32_t i = n - 1 - (i0 + (uint32_t)__ffs(m) - 1u);
            const uint32_t cnt = orient_one(u8arena, tab, refined_at[i], &hist[wid][0][0], lane,
                                            ori_angle + (size_t)i * kOriMaxPeaks, tb);
            if (lane == 0) {
                ori_count[i] = cnt;
                if (cnt) atomicAdd(&tiles[i / kSlotTile], cnt);
            }
        }
    }
}

constexpr int kDescThreads = 128;
static_assert(kDescThreads == kDescLen && kDescThreads == 128, "one descriptor bin per thread, four warps");
// The histogram: 8 angle bins and a 9th (the share of bin 0 that wrapped from
// bin 7) of cells -1..4 per axis (the 4 x 4 window and a border that takes the
// trilinear spill, so no sample needs a clamp or a validity test), in 8 copies.
// A row of cells is 5 apart from the next: cell 4 of one and cell -1 of the
// next, whose sums nobody reads, are the same.
// Word (bin, cell, copy) = bin * kHistBin + cell * 8 + copy: a bin's word lies
// in a bank of its cell and copy alone, so that the lanes of a warp, most of
// them in a few cells but in any bin, collide only by cell; the bank of a
// layout with the bins innermost also depends on each lane's bin.
constexpr int kHistSide = 5;
constexpr int kHistCopies = 8;
constexpr int kHistBin = 32 * kHistCopies;  // cells -1 .. 4 by -1 .. 4: 31, and one unused
constexpr int kHistWords = 9 * kHistBin;
static_assert(5 * kHistSide + 6 <= 32 && kHistBin % 32 == 0, "a word's bank is its cell's and copy's");
constexpr int kDescRadGrid = 31;                      // largest radius served from the grid
constexpr int kDescGridSide = 2 * kDescRadGrid + 3;   // offsets -(rad+1) .. rad+1

// A row of the window and its sample pairs that can be inside the rotated
// square, as a warp enumerates them: pair m of the warp, if it lies in this
// row, is at window offset (px + 2 m, py), grid index c + 2 m; k holds the
// parity of the grid row (times 2) and 16 times the histogram copy of m = 0.
// The copy is (i + q) & 7 of pair i of row q: neighbours in a row and pairs
// above each other, which mostly share cells, use different copies (2.35
// wavefronts per atomic by a CPU model of the bank conflicts; by i & 7, 2.6;
// with rows of cells 6 apart 2.5 and 2.8; a layout with the bins innermost
// by lane & 7, 3.2).
struct __align__(16) PairRow {
    float px, py;
    int c, k;
};
constexpr int kWarpRows = 16;                                  // a warp takes the rows q with q % 4 = warp
constexpr int kWarpWords = kWarpRows * (kDescRadGrid + 1) / 32;  // a bit for each of its pairs
struct WarpPairs {
    PairRow row[kWarpRows];      // the rows that have pairs
    uint32_t start[kWarpWords];  // the pairs that start a row
};
static_assert(kWarpRows * 4 >= 2 * kDescRadGrid + 1, "every row has a warp");

// Fills in the warp's rows; returns the count of its pairs. (Row q, py = q -
// rad, has pairs at px = 2 i - rad - p, i = 0 .. rad, p the parity of its grid
// row q + 1.) The two strips |ca px + sa py| < lim and |ca py - sa px| < lim
// cut an interval out of each row; near-zero ca, sa are widened to 1e-4, which
// with the margins (0.01 on lim, a quarter pixel on x) only adds pairs. A
// third of the window's pairs are outside; whether a sample is inside is
// decided by itself.
__device__ __forceinline__ int warp_pairs(WarpPairs* w, float ca, float sa, float lim, int rad, int gst, int warp,
                                          int lane) {
    const float ic = rcp_approx(copysignf(fmaxf(fabsf(ca), 1e-4f), ca)), is = rcp_approx(copysignf(fmaxf(fabsf(sa), 1e-4f), sa));
    const float hx = (lim + 0.01f) * fabsf(ic), hy = (lim + 0.01f) * fabsf(is);
    const float rad_f = (float)rad;
    if (lane < kWarpWords) w->start[lane] = 0u;
    __syncwarp();  // the zeroes before any lane's atomicOr (shuffles and ballots do not order memory)
    // lane l: row 4 (l % 16) + warp (the lanes above 15 repeat them)
    const int q = 4 * (lane & (kWarpRows - 1)) + warp, p = (q + 1) & 1;
    const float py = (float)q - rad_f, shift = rad_f + (float)p, end = rad_f + 1.0f;
    // both within [-rad - 1, rad + 1]
    const float lo = fminf(fmaxf(fmaxf(-sa * ic * py - hx, ca * is * py - hy) - 0.25f, -end), end);
    const float hi = fmaxf(fminf(fminf(-sa * ic * py + hx, ca * is * py + hy) + 0.25f, end), -end);
    // px + 1 >= lo and px <= hi
    const int first = max(-floor_i(-0.5f * (lo + shift - 1.0f)), 0);
    const int last = min(floor_i(0.5f * (hi + shift)), rad);
    const int count = q < 2 * rad + 1 ? max(last - first + 1, 0) : 0;
    int at = count;
#pragma unroll
    for (int d = 1; d < kWarpRows; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, at, d, kWarpRows);
        if ((lane & (kWarpRows - 1)) >= d) at += y;
    }
    const int total = __shfl_sync(0xffffffffu, at, kWarpRows - 1);
    const bool some = count > 0 && lane < kWarpRows;
    const uint32_t rows = __ballot_sync(0xffffffffu, some);
    if (some) {
        at -= count;  // the row's first pair
        const int i0 = first - at;
        w->row[__popc(rows & ((1u << lane) - 1u))] =
            PairRow{(float)(2 * i0) - shift, py, (q + 1) * gst + 2 * i0 + 1, 16 * (i0 + q) + 2 * p};
        atomicOr(&w->start[at >> 5], 1u << (at & 31));
    }
    __syncwarp();
    return total;
}

// The eight shares of a sample, added to the histogram word by word: four
// cells (the next in x, in y, in both; byte distances kX, kY), two bins (kA)
// each.
template <int kA, int kX, int kY>
__device__ __forceinline__ void add_shares(uint32_t at, const uint32_t (&v)[8]) {
    asm volatile(
        "red.shared.add.u32 [%0], %1;\n red.shared.add.u32 [%0 + %15], %2;\n"
        "red.shared.add.u32 [%0 + %9], %3;\n red.shared.add.u32 [%0 + %10], %4;\n"
        "red.shared.add.u32 [%0 + %11], %5;\n red.shared.add.u32 [%0 + %12], %6;\n"
        "red.shared.add.u32 [%0 + %13], %7;\n red.shared.add.u32 [%0 + %14], %8;" ::"r"(at),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "n"(kX), "n"(kX + kA),
        "n"(kY), "n"(kY + kA), "n"(kX + kY), "n"(kX + kY + kA), "n"(kA)
        : "memory");
}

// The descriptor of one oriented keypoint (src/sift.rs:917-1060 and
// normalize_and_clip_descriptor, src/sift.rs:889-913), computed by the whole
// CTA (kDescThreads threads; it synchronises the CTA) into dst()[0 .. 128):
//  1. The bilinear samples the gradients need, bilinear(xo + i, yo + j) for
//     integer offsets i, j in [-(rad+1), rad+1], go to a shared grid once
//     (the reference re-evaluates four bilinears per window sample).
//  2. Each thread takes pairs of neighbouring window samples and evaluates
//     both at once with Blackwell's packed f32x2 multiply/add/FMA; the eight
//     trilinear contributions of
//     each are added to 128 shared bins as u32 fixed point (2^-f units, f
//     chosen so no bin can overflow): integer addition is associative, so the
//     descriptor is the same on every run.
//  3. The four warps normalise, clip at 0.2, renormalise.
// Radii above the grid (not reachable with the default sigma) fall back to
// per-sample bilinears from the level itself.
template <class Dst>
__device__ __forceinline__ void describe_one(const uint8_t* __restrict__ u8arena, const EntryTable& tab,
                                             const Keypoint& kp,
                                             float* grid, unsigned int* hist, WarpPairs* pairs_of, float* red_lo,
                                             float* red_hi,
                                             const Dst& dst) {
    const int tid = threadIdx.x;
    const float sqrt2 = __fsqrt_rn(2.0f);
    const int e = kp.octave;  // entry
    for (int w = tid; w < kHistWords / 4; w += kDescThreads)
        reinterpret_cast<uint4*>(hist)[w] = make_uint4(0u, 0u, 0u, 0u);
    const bool valid_oct = e >= 0 && e < tab.n;
    OctaveDev od{};
    if (valid_oct) od = tab.ents[e];
    const int o = od.octave;
    // division by 2^o is the multiplication by 2^-o, exactly
    const float inv_scale = valid_oct ? __int_as_float((127 - o) << 23) : 1.0f;
    const float so = valid_oct ? __fmul_rn(kp.size, inv_scale) : 0.0f;
    const bool valid = valid_oct && so > 0.0f;
    float inv_fix = 0.0f;
    if (valid) {
        const GaussPlane g = plane_for(u8arena, od, tab.S, kp.layer);
        const float xo = __fmul_rn(kp.x, inv_scale), yo = __fmul_rn(kp.y, inv_scale);
        const float ang = kp.angle;
        // the hardware sine and cosine (|ang| <= pi; absolute error ~4e-7,
        // a shift of ~1e-5 px at the window's edge)
        float sa, ca;
        __sincosf(ang, &sa, &ca);
        const float bw = __fmul_rn(3.0f, so);
        const float ww = __fmul_rn(bw, 4.0f);
        const float wsig = __fmul_rn(0.5f, ww);
        const float wd = __fmul_rn(__fmul_rn(2.0f, wsig), wsig);
        const int rad = rust_as_i32(ceilf(__fmul_rn(__fmul_rn(ww, sqrt2), 0.5f)));
        const float wm1 = (float)(g.W - 1), hm1 = (float)(g.H - 1);
        const int side = 2 * rad + 1;
        const int total = side * side;
        const bool use_grid = rad <= kDescRadGrid;
        const int gs = side + 2;
        // Grid layout: row gr (0 .. gs - 1) at gr * gst + (gr & 1), row
        // stride gst = gs + 1 (even), one spare slot per row (the last of
        // an even row, the first of an odd row). With the pair loop's
        // phase (the pairs of odd rows start one sample to the left), all
        // four float pairs a pair of samples reads are 8-byte aligned.
        const int gst = gs + 1;
        // |rx|, |ry| below lim keep xb, yb inside (-1, 4) after rounding, so
        // every cell index lies in the padded grid (samples within 1e-6
        // of the window edge, whose shares there are ~0, are left out)
        const float lim = __fmul_rn(2.5f, bw) * 0.99999905f;
        int n_pairs = 0;
        float lo = 3.0e38f, hi = 0.0f;
        if (use_grid) {
            n_pairs = warp_pairs(pairs_of + (tid >> 5), ca, sa, lim, rad, gst, tid >> 5, tid & 31);
            // the spare slots, read only for the phantom element of a
            // row's end pair, hold 0
            if (tid < gs) grid[tid * gst + ((tid & 1) ? 0 : gs)] = 0.0f;
            // Bilinear samples at the window's integer offsets, in v units
            // (px_raw), straight from the level (the patch stays in L1). All
            // of them share the
            // fraction of (xo, yo): the reference's sample positions xo + i
            // differ from it only by the rounding of that sum. Clamped
            // reads (get_gauss_pixel_value) only for windows at the border.
            const float xf = floorf(xo), yf = floorf(yo);
            const float fdx = xo - xf, fdy = yo - yf;
            const int px0 = (int)xf - (rad + 1), py0 = (int)yf - (rad + 1);
            const bool inner = px0 >= 0 && py0 >= 0 && px0 + gs < g.W && py0 + gs < g.H;
            const float inv_gs = 1.0f / (float)gs;
            if (inner) {
                // A thread makes a block of 4 x 4 grid points from 5 rows of
                // 5 pixels, two aligned words a row (the shift is the same
                // for every block; the second word may end past the row, in
                // its padding or the next, never past the arena): each
                // row's horizontal lerps serve the points above and below
                // it, two columns at once on f32x2 pairs. The same two
                // lerps per point as below, so the same values.
                const int blocks = (gs + 3) >> 2;
                const float inv_blocks = 1.0f / (float)blocks;
                const int pitch4 = g.pitch >> 2, shift = 8 * (px0 & 3);
                const uint32_t* org = reinterpret_cast<const uint32_t*>(g.base + (long long)py0 * g.pitch + (px0 & ~3));
                const float2 fdx2 = make_float2(fdx, fdx), fdy2 = make_float2(fdy, fdy);
                const float2 neg1 = make_float2(-1.0f, -1.0f);
                float tf = (float)tid;
                for (int t = tid; t < blocks * blocks; t += kDescThreads, tf += (float)kDescThreads) {
                    const int by = floor_i((tf + 0.5f) * inv_blocks), bx = t - by * blocks;
                    const int nr = min(4, gs - 4 * by), nc = min(4, gs - 4 * bx);
                    // all words first (rows past the block's last repeat it)
                    const uint32_t* pp = org + 4 * by * pitch4 + bx;
                    uint32_t w[5][2];
#pragma unroll
                    for (int j = 0; j < 5; ++j) {
                        const uint32_t* pr = pp + min(j, nr) * pitch4;
                        w[j][0] = pr[0];
                        w[j][1] = pr[1];
                    }
                    float* gp = grid + 4 * by * gst + 4 * bx;  // (gst is even: pairs of even rows are aligned)
                    float2 up0, up1;
#pragma unroll
                    for (int j = 0; j < 5; ++j) {
                        const uint32_t b4 = __funnelshift_r(w[j][0], w[j][1], shift);
                        const float a0 = float_of_byte<0>(b4), a1 = float_of_byte<1>(b4), a2 = float_of_byte<2>(b4),
                                    a3 = float_of_byte<3>(b4), a4 = float_of_byte<0>(w[j][1] >> shift);
                        const float2 l0 = make_float2(a0, a1), l1 = make_float2(a2, a3);
                        const float2 r0 = __ffma2_rn(fdx2, __ffma2_rn(l0, neg1, make_float2(a1, a2)), l0);
                        const float2 r1 = __ffma2_rn(fdx2, __ffma2_rn(l1, neg1, make_float2(a3, a4)), l1);
                        if (j > 0 && j <= nr) {
                            const float2 b0 = __ffma2_rn(fdy2, __ffma2_rn(up0, neg1, r0), up0);
                            const float2 b1 = __ffma2_rn(fdy2, __ffma2_rn(up1, neg1, r1), up1);
                            float* d = gp + (j - 1) * gst + ((j - 1) & 1);
                            if (nc == 4) {
                                if ((j - 1) & 1) {  // (odd rows sit one slot on: their middle pair is aligned)
                                    d[0] = b0.x;
                                    *reinterpret_cast<float2*>(d + 1) = make_float2(b0.y, b1.x);
                                    d[3] = b1.y;
                                } else {
                                    *reinterpret_cast<float2*>(d) = b0;
                                    *reinterpret_cast<float2*>(d + 2) = b1;
                                }
                                lo = fminf(lo, fminf(fminf(b0.x, b0.y), fminf(b1.x, b1.y)));
                                hi = fmaxf(hi, fmaxf(fmaxf(b0.x, b0.y), fmaxf(b1.x, b1.y)));
                            } else {
                                const float v[3] = {b0.x, b0.y, b1.x};
#pragma unroll
                                for (int k = 0; k < 3; ++k)
                                    if (k < nc) {
                                        d[k] = v[k];
                                        lo = fminf(lo, v[k]);
                                        hi = fmaxf(hi, v[k]);
                                    }
                            }
                        }
                        up0 = r0;
                        up1 = r1;
                    }
                }
            } else {
                float qf = (float)tid;
                for (int q = tid; q < gs * gs; q += kDescThreads, qf += (float)kDescThreads) {
                    const int qy = floor_i((qf + 0.5f) * inv_gs);
                    const int qx = q - qy * gs;
                    const float q11 = g.px_raw(px0 + qx, py0 + qy), q21 = g.px_raw(px0 + qx + 1, py0 + qy);
                    const float q12 = g.px_raw(px0 + qx, py0 + qy + 1), q22 = g.px_raw(px0 + qx + 1, py0 + qy + 1);
                    // the reference's bilinear blend as two lerps (within the
                    // descriptor tolerance)
                    const float r0 = fmaf(fdx, q21 - q11, q11), r1 = fmaf(fdx, q22 - q12, q12);
                    const float b = fmaf(fdy, r1 - r0, r0);
                    grid[qy * gst + (qy & 1) + qx] = b;
                    lo = fminf(lo, b);
                    hi = fmaxf(hi, b);
                }
            }
        } else {
            lo = 0.0f;
            hi = 1.0f;
        }
        // Fixed point: |gx|, |gy| <= range of the sampled values, so every
        // bin is below sqrt(2) * range * total (Gaussian and trilinear
        // weights <= 1 with unit sum); the scale is the largest power of
        // two that keeps that bound under 2^32.
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, m));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, m));
        }
        if ((tid & 31) == 0) {
            red_lo[tid >> 5] = lo;
            red_hi[tid >> 5] = hi;
        }
        __syncthreads();
        lo = fminf(fminf(red_lo[0], red_lo[1]), fminf(red_lo[2], red_lo[3]));
        hi = fmaxf(fmaxf(red_hi[0], red_hi[1]), fmaxf(red_hi[2], red_hi[3]));
        const float range = fmaxf(hi - lo, 1.0f / 65536.0f);
        // and every single contribution (<= sqrt(2) * range) below 2^23,
        // where its rounding to an integer is exact (the subnormal grid of
        // the pair loop, the 2^23 rounding add of the per-sample loop)
        const float per = 1.4143f * range;
        // floor(log2 q) of a positive normal float is its exponent field
        const int fbits = max(0, min(40, min((__float_as_int(4.0e9f / (per * (float)total)) >> 23) - 127,
                                             (__float_as_int(8.0e6f / per) >> 23) - 127)));
        const float to_fix = __int_as_float((127 + fbits) << 23);
        inv_fix = __int_as_float((127 - fbits) << 23);
        // Descriptor samples are interpolated linearly into their bins, so
        // the sample loops are written for speed within the descriptor
        // tolerance: fused multiply-adds, reciprocal products instead of
        // divisions, the hardware's approximate square root and exp2
        // (scale folded in), an arctangent polynomial in units of angle
        // bins (error 1.5e-5 bin) from which the relative angle is binned
        // directly (floor and & 7 give the rem_euclid bins), and the
        // fixed-point rounding fused into the weight product. Each changes a
        // descriptor value by ~1e-5 or less.
        const float inv_bw = 1.0f / bw;
        const float angb = ang * (4.0f / kPi);  // keypoint angle in 45-degree bins
        const float wexp = -1.4426950408889634f / wd;  // exp(-d2/wd) = exp2(d2 * wexp)
        const uint32_t hist_at = (uint32_t)__cvta_generic_to_shared(hist);
        const float rad_f = (float)rad;
        // windows that stay inside the level need no per-sample border test
        const bool edge = !(__fadd_rn(xo, -rad_f) >= 0.0f && __fadd_rn(xo, rad_f) < wm1 &&
                            __fadd_rn(yo, -rad_f) >= 0.0f && __fadd_rn(yo, rad_f) < hm1);
        if (use_grid) {
            // Sample pairs: a thread takes the window samples (px, py) and
            // (px + 1, py) and evaluates both with packed f32x2 arithmetic,
            // the same operations per element as one sample alone. A row
            // has rad + 1 pairs: from px = -rad in rows of even grid index
            // (the last pair's second element, px = rad + 1, is outside the
            // window), from px = -rad - 1 in rows of odd grid index (the
            // first pair's first element is outside), so the float pairs
            // of the gradients' grid reads are 8-byte aligned (one 64-bit
            // load each). A warp enumerates the pairs of its rows that can be
            // inside the rotated square (warp_pairs).
            // Fixed point on the subnormal grid: a float below 2^-125 is
            // k * 2^-149 and its bit pattern is k, so a contribution scaled
            // by 2^(fbits - 149) and rounded once to the nearest float (the
            // last multiply) has the fixed-point integer as its bits (k <
            // 2^23 by the scale choice): no conversion and no offset to
            // subtract before the atomic. The scale is split so every factor
            // stays a normal float: 2^(fbits - 49) rides in the exponent,
            // exp2(d2 * wexp + fbits - 49) = 2^(fbits - 49) exp(-d2 / wd),
            // and 2^-100 in the two angle weights. (The library is built
            // without flush-to-zero, and mul.rn.f32x2 keeps subnormals.)
            const float fb = (float)(fbits - 49);
            const float2 ca2 = make_float2(ca, ca), sa2 = make_float2(sa, sa), nsa2 = make_float2(-sa, -sa);
            const float2 ib2 = make_float2(inv_bw, inv_bw), half3 = make_float2(1.5f, 1.5f);
            const float2 wexp2 = make_float2(wexp, wexp), fb2 = make_float2(fb, fb);
            const float2 m15 = make_float2(kMagic15, kMagic15), nm15 = make_float2(-kMagic15, -kMagic15);
            const float2 neg1 = make_float2(-1.0f, -1.0f), one2 = make_float2(1.0f, 1.0f);
            constexpr float kAngScale = 7.888609052210118e-31f;  // 2^-100
            const float2 as2 = make_float2(kAngScale, kAngScale), nas2 = make_float2(-kAngScale, -kAngScale);
            const float2 angb2 = make_float2(angb, angb);
            const WarpPairs* mine = pairs_of + (tid >> 5);
            const uint32_t to_me = 0xffffffffu >> (31 - (tid & 31));
            auto pairs = [&](auto edge_tag) {
                constexpr bool kEdge = decltype(edge_tag)::value;
#pragma unroll 1
                for (int m = tid & 31, before = -1; m < n_pairs; m += 32) {
                    // the row: as many as have started up to this pair
                    const uint32_t starts = mine->start[m >> 5];
                    const PairRow row = mine->row[before + __popc(starts & to_me)];
                    before += __popc(starts);
                    const float px = fmaf(2.0f, (float)m, row.px), py = row.py;
                    const bool v0 = px >= -rad_f, v1 = px < rad_f;
                    const int c = row.c + 2 * m;
                    // rows gr - 1 and gr + 1 sit one slot the other way
                    const int cv = c + 1 - (row.k & 2);
                    const float2 P = make_float2(px, px + 1.0f), Q = make_float2(py, py);
                    const float2 rx = __ffma2_rn(P, ca2, __fmul2_rn(Q, sa2));
                    const float2 ry = __ffma2_rn(P, nsa2, __fmul2_rn(Q, ca2));
                    bool in0 = v0 && fabsf(rx.x) < lim && fabsf(ry.x) < lim;
                    bool in1 = v1 && fabsf(rx.y) < lim && fabsf(ry.y) < lim;
                    if constexpr (kEdge) {
                        const float xs0 = xo + px, ys0 = yo + py, xs1 = xo + P.y;
                        const bool rowin = !(ys0 < 0.0f || ys0 >= hm1);
                        in0 = in0 && rowin && !(xs0 < 0.0f || xs0 >= wm1);
                        in1 = in1 && rowin && !(xs1 < 0.0f || xs1 >= wm1);
                    }
                    // (left, right) and (above, below) of both elements
                    const float2 gl = *reinterpret_cast<const float2*>(grid + c - 1);
                    const float2 gr = *reinterpret_cast<const float2*>(grid + c + 1);
                    const float2 gu = *reinterpret_cast<const float2*>(grid + cv - gst);
                    const float2 gd = *reinterpret_cast<const float2*>(grid + cv + gst);
                    const float2 gx = __ffma2_rn(gl, neg1, gr);
                    const float2 gy = __ffma2_rn(gu, neg1, gd);
                    const float2 m2 = __ffma2_rn(gx, gx, __fmul2_rn(gy, gy));
                    const float2 ea = __ffma2_rn(__ffma2_rn(P, P, __fmul2_rn(Q, Q)), wexp2, fb2);
                    const float2 wm = __fmul2_rn(make_float2(sqrt_approx(m2.x), sqrt_approx(m2.y)),
                                           make_float2(ex2_approx(ea.x), ex2_approx(ea.y)));
                    const float2 ab = __fadd2_rn(atan2_bins2(gy, gx), make_float2(-angb, -angb));
                    const float2 xb = __ffma2_rn(rx, ib2, half3), yb = __ffma2_rn(ry, ib2, half3);
                    // floors by the 1.5 * 2^23 rounding-down add: the low
                    // bits of tx, ty, ta are the integers
                    const float2 tx = __fadd2_rd(xb, m15), ty = __fadd2_rd(yb, m15), ta = __fadd2_rd(ab, m15);
                    const float2 fx = __ffma2_rn(__fadd2_rn(tx, nm15), neg1, xb);
                    const float2 fy = __ffma2_rn(__fadd2_rn(ty, nm15), neg1, yb);
                    const float2 fa = __ffma2_rn(__fadd2_rn(ta, nm15), neg1, ab);
                    // histogram byte of cell (xbi, ybi), bin abi & 7 and the
                    // pair's copy, from the float bits (the 0x4B400000
                    // offsets cancel mod 2^32, 0x4B400000 & 7 == 0)
                    constexpr uint32_t kA = 4 * kHistBin, kX = 4 * kHistCopies, kY = kX * kHistSide;
                    constexpr uint32_t kCellOff = (kX + kY) - (kX + kY) * 0x4B400000u;
                    const uint32_t at = hist_at + kCellOff + (uint32_t)((row.k >> 2) + 4 * m & 28);
                    const uint32_t at0 = __float_as_uint(ty.x) * kY + __float_as_uint(tx.x) * kX +
                                         (__float_as_uint(ta.x) & 7u) * kA + at;
                    const uint32_t at1 = __float_as_uint(ty.y) * kY + __float_as_uint(tx.y) * kX +
                                         (__float_as_uint(ta.y) & 7u) * kA + at;
                    const float2 wy0 = __fmul2_rn(wm, __ffma2_rn(fy, neg1, one2)), wy1 = __fmul2_rn(wm, fy);
                    const float2 wx0 = __ffma2_rn(fx, neg1, one2);
                    // (1 - fa) * 2^-100 and fa * 2^-100 (exact scalings)
                    const float2 wa0 = __ffma2_rn(fa, nas2, as2), wa1 = __fmul2_rn(fa, as2);
                    uint32_t s0[8], s1[8];
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) {
                        const float2 wxy = __fmul2_rn((cc & 1) ? fx : wx0, (cc & 2) ? wy1 : wy0);
                        // the products, rounded to the nearest fixed-point
                        // integer on the subnormal grid, are their own bits
                        const float2 n0 = __fmul2_rn(wxy, wa0), n1 = __fmul2_rn(wxy, wa1);
                        s0[2 * cc] = __float_as_uint(n0.x);
                        s0[2 * cc + 1] = __float_as_uint(n1.x);
                        s1[2 * cc] = __float_as_uint(n0.y);
                        s1[2 * cc + 1] = __float_as_uint(n1.y);
                    }
                    if (in0) add_shares<kA, kX, kY>(at0, s0);
                    if (in1) add_shares<kA, kX, kY>(at1, s1);
                }
            };
            if (edge)
                pairs(std::true_type{});
            else
                pairs(std::false_type{});
        } else {
            // Radii above the grid: one sample per thread, four bilinears
            // from the level per sample (the reference's own evaluation).
            for (int k = tid; k < total; k += kDescThreads) {
                const int qy = k / side;
                const float px = (float)(k - qy * side) - rad_f, py = (float)qy - rad_f;
                const float rx = fmaf(ca, px, sa * py);
                const float ry = fmaf(-sa, px, ca * py);
                if (!(fabsf(rx) < lim && fabsf(ry) < lim)) continue;
                const float xs = xo + px, ys = yo + py;
                if (xs < 0.0f || xs >= wm1 || ys < 0.0f || ys >= hm1) continue;
                const float gx =
                    __fsub_rn(g.bilinear(__fadd_rn(xs, 1.0f), ys), g.bilinear(__fsub_rn(xs, 1.0f), ys));
                const float gy =
                    __fsub_rn(g.bilinear(xs, __fadd_rn(ys, 1.0f)), g.bilinear(xs, __fsub_rn(ys, 1.0f)));
                const float mag = sqrt_approx(fmaf(gx, gx, gy * gy));
                const float wm = mag * ex2_approx(fmaf(px, px, py * py) * wexp);
                const float ab = atan2_bins(gy, gx) - angb;  // in [-12, 4]
                const float xb = fmaf(rx, inv_bw, 1.5f), yb = fmaf(ry, inv_bw, 1.5f);
                int xbi, ybi, abi;
                const float xbf = floor_fi(xb, &xbi), ybf = floor_fi(yb, &ybi), abf = floor_fi(ab, &abi);
                const float fx = xb - xbf, fy = yb - ybf, fa = ab - abf;
                const float wa1 = fa * to_fix, wa0 = to_fix - wa1;
                const float wx0 = 1.0f - fx, wx1 = fx;
                const float wy0 = wm * (1.0f - fy), wy1 = wm * fy;
                unsigned int* h0 =
                    hist + (abi & 7) * kHistBin + ((ybi + 1) * kHistSide + (xbi + 1)) * kHistCopies + (tid & 7);
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    const float wxy = ((cc & 1) ? wx1 : wx0) * ((cc & 2) ? wy1 : wy0);
                    unsigned int* hc = h0 + ((cc & 2) ? kHistSide * kHistCopies : 0) + ((cc & 1) ? kHistCopies : 0);
                    atomicAdd(hc, __float_as_uint(__fmaf_rn(wxy, wa0, kMagic)) - 0x4B000000u);
                    atomicAdd(hc + kHistBin, __float_as_uint(__fmaf_rn(wxy, wa1, kMagic)) - 0x4B000000u);
                }
            }
        }
    }
    __syncthreads();  // the histogram is complete
    // normalize_and_clip_descriptor (src/sift.rs:889-913), one bin per
    // thread; the sums of squares over the four warps in a fixed order
    {
        // the copies' sums, lanes over the cells (two 16-byte reads a bin),
        // then handed to the bins' own threads (through the grid's memory)
        uint32_t* sums = reinterpret_cast<uint32_t*>(grid);
        {
            const int ia = tid >> 4, cell = tid & 15;
            const unsigned int* h = hist + ia * kHistBin + (((cell >> 2) + 1) * kHistSide + (cell & 3) + 1) * kHistCopies;
            // odd rows of cells read their halves in the other order: no bank conflicts
            const int turn = cell & 4;
            uint4 x = *reinterpret_cast<const uint4*>(h + turn), y = *reinterpret_cast<const uint4*>(h + (turn ^ 4));
            unsigned v = x.x + x.y + x.z + x.w + y.x + y.y + y.z + y.w;
            if (ia == 0) {
                x = *reinterpret_cast<const uint4*>(h + 8 * kHistBin + turn);
                y = *reinterpret_cast<const uint4*>(h + 8 * kHistBin + (turn ^ 4));
                v += x.x + x.y + x.z + x.w + y.x + y.y + y.z + y.w;
            }
            sums[cell * 9 + ia] = v;
        }
        __syncthreads();
        const int bin = tid;  // (iy * 4 + ix) * 8 + ia
        const unsigned v = sums[(bin >> 3) * 9 + (bin & 7)];
        float d = __fmul_rn((float)v, inv_fix);
        float ss = __fmul_rn(d, d);
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, m));
        if ((tid & 31) == 0) red_lo[tid >> 5] = ss;
        __syncthreads();
        const float norm = __fsqrt_rn(__fadd_rn(__fadd_rn(red_lo[0], red_lo[1]), __fadd_rn(red_lo[2], red_lo[3])));
        if (!(norm < 1e-8f)) {  // the same for every thread
            d = fminf(__fmul_rn(d, __fdiv_rn(1.0f, norm)), 0.2f);
            float s2 = __fmul_rn(d, d);
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) s2 = __fadd_rn(s2, __shfl_xor_sync(0xffffffffu, s2, m));
            if ((tid & 31) == 0) red_hi[tid >> 5] = s2;
            __syncthreads();
            const float n2 =
                __fsqrt_rn(__fadd_rn(__fadd_rn(red_hi[0], red_hi[1]), __fadd_rn(red_hi[2], red_hi[3])));
            if (!(n2 < 1e-8f)) d = __fmul_rn(d, __fdiv_rn(1.0f, n2));
        }
        dst()[bin] = d;
    }
}

// One CTA per oriented keypoint (persistent over the list), describe_one on
// each. The shared-memory pipe bounds it: 80 % of its wavefronts at octave 0
// of a 1080p frame (12 857 keypoints, 146 us; half of them the atomics, 2.46 a
// warp instruction), with 69 % of the issue slots. What it was before, with a
// histogram of bins innermost and pairs listed one by one in shared memory:
// 167 us, the stage 223 us at 1080p and 1406 us at 4096 x 4096, now 199 and
// 1261. Of that, the bank layout, the warps' own enumeration of their pairs
// and the sums over copies gave 1406 -> 1298 us, the grid fill by words 1276,
// rows of cells 5 apart 1261. Adding the shares of a pair's two samples at
// once where they have the same cells and bin made 7 % more instructions and
// no difference in time; 16 copies (2.1 wavefronts) leave room for 6 CTAs per
// SM, and 6 took 2.5 % more than 7, which take 1.5 % more than 8 (64 registers,
// 1232 us at 4096 x 4096). Rows of cells mirrored where that spreads a window
// row over more banks and 16-byte stores of the grid leave out 7 % of the
// wavefronts, and change the time by less than 1 %: with 8 CTAs the kernel is
// as near to the issue slots as to the shared-memory pipe.
__global__ void __launch_bounds__(kDescThreads, 8) k_descriptor(const uint8_t* __restrict__ u8arena, EntryTable tab,
                                                              const Keypoint* __restrict__ oriented,
                                                              OctCounters* __restrict__ oc,
                                                              float* __restrict__ desc, uint32_t cap,
                                                              const RunCell* __restrict__ cell,
                                                              int persist_from) {
    chain_wait();
    __shared__ __align__(16) float grid[kDescGridSide * (kDescGridSide + 1)];
    __shared__ __align__(16) unsigned int hist[kHistWords];
    __shared__ WarpPairs pairs_of[kDescThreads / 32];
    __shared__ float red_lo[kDescThreads / 32], red_hi[kDescThreads / 32];
    const int tid = threadIdx.x;
    const uint32_t base = oc->out_base;
    uint32_t n = oc->n_ori;
    if (base >= cap) n = 0;
    else if (n > cap - base) n = cap - base;
    // Keypoints differ ~4x in window area: they come from a queue. Thread 0
    // claims the next item while the CTA works on the current one (slot
    // next[p ^ 1]), unless the CTA retires after the current one.
    __shared__ uint32_t next[2];
    // a host call's result buffer, by the run's cell
    __shared__ float* hdesc;
    __shared__ uint32_t hcap;
    const bool persist = (int)blockIdx.x >= persist_from;
    if (tid == 0) {
        next[0] = atomicAdd(&oc->next_desc, 1u);
        hdesc = cell ? cell->desc : nullptr;
        hcap = cell ? cell->cap : 0u;
    }
    for (int taken = 0, p = 0;; ++taken, p ^= 1) {
        __syncthreads();  // next[p] is visible, the grid and histogram are free
        const uint32_t cur = next[p];
        if (cur >= n) break;
        const bool more = persist || taken + 1 < kDescBudget;
        uint32_t claim = n;
        if (tid == 0 && more) claim = atomicAdd(&oc->next_desc, 1u);
        // the queue runs from the last keypoint: an octave's list is in layer
        // order, so the largest windows go first and the smallest make the
        // tail of the stage
        const uint32_t i = base + (n - 1 - cur);
        const Keypoint kp = oriented[i];
        // keypoints below hcap straight into the host call's buffer
        describe_one(u8arena, tab, kp, grid, hist, pairs_of, red_lo, red_hi,
                         [&] { return (i < hcap ? hdesc : desc) + (size_t)i * kDescLen; });
        if (tid == 0) next[p ^ 1] = claim;
    }
}

}  // namespace

size_t ori_bins_bytes() { return (size_t)kBinSide * kBinSide; }
int launch_ori_bins(uint8_t* bins, cudaStream_t st) {
    if (launch_chained(k_ori_bins, kBinSide, kBinSide, 0, st, bins) != cudaSuccess) return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

int launch_orientation(const uint8_t* u8arena, const EntryTable& tab, const float* lut255, const uint8_t* bins,
                       const Keypoint* refined_at, const uint32_t* keep, uint32_t ncap, OctCounters* oc,
                       float* ori_angle, uint32_t* ori_count, uint32_t* tiles, int grid, int persist_ctas,
                       cudaStream_t st) {
    if (launch_chained(k_orientation, grid, dim3(32, kOriWarps), 0, st, u8arena, tab, lut255, bins, refined_at, keep,
                       ncap, oc, ori_angle, ori_count, tiles, std::max(grid - persist_ctas, 0)) != cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

int launch_descriptor(const uint8_t* u8arena, const EntryTable& tab, const Keypoint* oriented, OctCounters* oc,
                      float* desc, uint32_t cap, const RunCell* cell, int grid, int persist_ctas, cudaStream_t st) {
    if (launch_chained(k_descriptor, grid, kDescThreads, 0, st, u8arena, tab, oriented, oc, desc, cap, cell,
                       std::max(grid - persist_ctas, 0)) != cudaSuccess)
        return -1;
    return cudaPeekAtLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace sift
