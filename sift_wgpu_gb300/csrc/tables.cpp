// tables.cpp — host-side filter tables of the pyramid.
//
// The blur kernels and the Lanczos3 resampling taps depend only on the
// parameters and the image size, so they are built once on the host (in f32,
// the way the reference builds them) and uploaded; every GPU thread then uses
// the identical weights. Compiled with -ffp-contract=off so that each product
// and sum is rounded separately, as in Rust.
//
//  * gaussian_kernel: imageproc 0.25.0 gaussian_blur_f32's kernel (the crate
//    is a dependency of the reference, Cargo.lock:648-650, not vendored):
//    radius ceil(2 sigma), taps (sqrt(2 pi) sigma)^-1 exp(-x^2 / (2 sigma^2)).
//  * lanczos_axis: image 0.25.6 resize's per-axis taps (Cargo.lock:634-636):
//    centre (i + 0.5) * ratio, support 3 * max(ratio, 1), window clamped to
//    the source, lanczos3((j - centre + 0.5) / max(ratio, 1)) normalised by
//    the window's sum.
//  * blur_sigmas: the increments of generate_gaussian_pyramid
//    (src/sift.rs:129-177) and the base blur (src/sift.rs:1204-1214).
#include "tables.h"

#include <algorithm>
#include <cmath>

namespace sift {

namespace {
constexpr float kPiF = 3.14159265358979323846f;

// f32::powi with a run-time exponent (repeated squaring, as compiler
// builtins evaluate it).
float powi(float a, int b) {
    bool recip = b < 0;
    unsigned n = recip ? 0u - (unsigned)b : (unsigned)b;
    float r = 1.0f;
    for (;;) {
        if (n & 1u) r *= a;
        n >>= 1;
        if (n == 0) break;
        a *= a;
    }
    return recip ? 1.0f / r : r;
}

float sinc(float t) {
    float a = t * kPiF;
    if (t == 0.0f) return 1.0f;
    return std::sin(a) / a;
}

float lanczos3(float x) {
    if (std::fabs(x) < 3.0f) return sinc(x) * sinc(x / 3.0f);
    return 0.0f;
}
}  // namespace

std::vector<float> gaussian_kernel(float sigma) {
    float fr = std::ceil(2.0f * sigma);
    int radius = fr > 0.0f ? (int)fr : 0;
    std::vector<float> k((size_t)(2 * radius + 1), 0.0f);
    float c = 1.0f / (std::sqrt(2.0f * kPiF) * sigma);
    for (int i = 0; i <= radius; ++i) {
        float x = (float)i;
        float v = c * std::exp(-(x * x) / (2.0f * (sigma * sigma)));
        k[(size_t)(radius + i)] = v;
        k[(size_t)(radius - i)] = v;
    }
    return k;
}

namespace {
// The f16 bits of a whole number of at most 11 significant bits.
uint32_t half_of_int(int v) {
    const uint32_t s = v < 0 ? 0x8000u : 0u;
    uint32_t m = (uint32_t)(v < 0 ? -v : v);
    if (m == 0) return 0;
    int e = 0;
    while (m >> (e + 1)) ++e;
    m = e <= 10 ? m << (10 - e) : m >> (e - 10);
    return s | (uint32_t)(e + 15) << 10 | (m & 0x3ffu);
}
}  // namespace

// Weights W = round(w 2^q) as a 2^shift + b with whole limbs that f16 holds
// (a <= 2048) and whose sums over 255-valued pixels stay below 2^24, so the
// tensor core's f32 accumulators hold both sums exactly whatever its order of
// addition. The level value s = sum(W p) / 2^q is then known to within
//   quantisation   255 max(sum of the positive, sum of the negative w - W/2^q)
//   the reference's rounding: one per product, one per partial sum of the
//                  sequential f32 sum, each at most 2^-24 of its value, the
//                  partial sum after tap k being at most 255 (w_0 + .. + w_k)
//   the kernel's   2^-16 (2^-15 with 9 whole bits), rounding the two limbs'
//                  sum to 15 (14) fraction bits
// The kernel adds that bound e to s and takes floor(s + e) where its fraction
// is at least 2 e (there the reference truncates to the same integer); the
// other pixels, a few in 10^4, are summed again in the reference's order.
TcBlur tc_blur(const std::vector<float>& w) {
    TcBlur t;
    const int n = (int)w.size(), r = n / 2;
    if (n < 1 || r > 28) return t;
    double wmax = 0.0, wsum = 0.0;
    for (float v : w) {
        if (!(v >= 0.0f)) return t;
        wmax = std::max(wmax, (double)v);
        wsum += v;
    }
    if (!(wmax > 0.0)) return t;
    // a = w 2^qa <= 2047, sums of a below 2^24 / 2 with the start value
    int qa = 15;
    while (qa > 4 && wmax * std::ldexp(1.0, qa) > 2040.0) --qa;
    std::vector<long long> a(n), b(n);
    int shift = 12;
    double quant = 0.0;
    for (;; --shift) {
        if (shift < 4) return t;
        long long sb = 0;
        double up = 0.0, down = 0.0;
        const double scale = std::ldexp(1.0, qa + shift), unit = std::ldexp(1.0, -(qa + shift));
        for (int i = 0; i < n; ++i) {
            const long long W = std::llrint((double)w[i] * scale);
            a[i] = (W + (1ll << (shift - 1))) >> shift;
            b[i] = W - a[i] * (1ll << shift);
            sb += b[i] < 0 ? -b[i] : b[i];
            const double d = (double)w[i] - (double)W * unit;
            (d > 0 ? up : down) += std::fabs(d);
        }
        quant = 255.0 * std::max(up, down);
        if (sb * 255 < (1ll << 23)) break;
    }
    for (int i = 0; i < n; ++i)
        if (a[i] > 2047) return t;
    // The reference's rounding error: half an ulp of each product and of each
    // partial sum, which are largest where every pixel is 255 (half an ulp
    // does not fall as the value rises).
    double cum = 0.0, ref = 0.0;
    auto half_ulp = [](double x) { return x > 0.0 ? std::ldexp(1.0, std::ilogb(x) - 24) : 0.0; };
    for (int i = 0; i < n; ++i) {
        cum += w[i];
        ref += half_ulp(255.0 * w[i]) + half_ulp(255.0 * cum * (1.0 + 4.0 * n * std::ldexp(1.0, -24)));
    }
    t.clamp = 255.0 * wsum + 1.0 >= 256.0;
    const int frac = t.clamp ? 14 : 15;
    if (255.0 * wsum + 1.0 >= std::ldexp(1.0, 23 - frac) || qa + 24 - frac > 24) return t;
    const double e = quant + ref + std::ldexp(0.5, -frac);  // (the last: the rounding to `frac` bits)
    // s in units of 1 is 2^(qa - 24) in the accumulators (pixels enter as
    // f16 subnormals, v 2^-24); the start value puts s in the mantissa with
    // `frac` fraction bits
    t.init_a = (float)std::ldexp(1.0, qa + (23 - frac) - 24);
    const double be = std::ceil(std::ldexp(e, qa + shift));  // whole b units
    if (be * 2 >= std::ldexp(1.0, 24)) return t;
    t.init_b = (float)std::ldexp(be, -24);
    t.scale_b = (float)std::ldexp(1.0, -shift);
    t.whole = (float)(std::ldexp(1.0, qa - 24 + 23) - t.init_a);
    // s enlarged by e: the reference's sum lies in [s - 2 e, s]
    const uint32_t thr = (uint32_t)std::ceil(2.0 * std::ldexp(be, frac - qa - shift));
    if (thr >> (frac - 2)) return t;
    t.near = thr << (32 - frac);
    // fragments (m16n8k16): lane = 4 g + t holds k = 2t, 2t+1 (+8)
    const int P = r <= 4 ? 4 : (r + 3) / 8 * 8 + 4, PV = (r + 7) / 8 * 8;
    t.kh = (8 + 2 * P) / 16;
    t.kv = (16 + 2 * PV) / 16;
    // (each limb's halves once: a layout for a new image size makes some 18 000
    // fragment words, 420 us of conversions tap by tap, 70 us so)
    std::vector<uint32_t> ha(n), hb(n);
    for (int i = 0; i < n; ++i) {
        ha[i] = half_of_int((int)a[i]);
        hb[i] = half_of_int((int)b[i]);
    }
    t.frags.resize((size_t)(t.kh * 4 + t.kv * 8) * 32);
    uint32_t* f = t.frags.data();
    auto pair = [n](const std::vector<uint32_t>& h, int i) -> uint32_t {  // taps i, i + 1
        return ((unsigned)i < (unsigned)n ? h[i] : 0u) | ((unsigned)(i + 1) < (unsigned)n ? h[i + 1] << 16 : 0u);
    };
    for (int ks = 0; ks < t.kh; ++ks)
        for (int lane = 0; lane < 32; ++lane) {
            const int g = lane >> 2, k = 16 * ks + 2 * (lane & 3), i = k - g - (P - r);  // column n = g
            for (const auto* h : {&ha, &hb})
                for (int d : {0, 8}) *f++ = pair(*h, i + d);
        }
    for (int ks = 0; ks < t.kv; ++ks)
        for (int lane = 0; lane < 32; ++lane) {
            const int g = lane >> 2, k = 16 * ks + 2 * (lane & 3), i = k - g - (PV - r);  // row m = g, g + 8
            for (const auto* h : {&ha, &hb})
                for (int d : {0, -8, 8, 0}) *f++ = pair(*h, i + d);
        }
    t.ok = true;
    return t;
}

AxisTaps lanczos_axis(uint32_t src, uint32_t dst) {
    AxisTaps t;
    float ratio = (float)src / (float)dst;
    float sratio = ratio < 1.0f ? 1.0f : ratio;
    float support = 3.0f * sratio;
    for (uint32_t o = 0; o < dst; ++o) {
        float input = ((float)o + 0.5f) * ratio;
        long long left = (long long)std::floor(input - support);
        left = std::max<long long>(0, std::min<long long>(left, (long long)src - 1));
        long long right = (long long)std::ceil(input + support);
        right = std::max<long long>(left + 1, std::min<long long>(right, (long long)src));
        input = input - 0.5f;
        t.left.push_back((int)left);
        t.count.push_back((int)(right - left));
        t.woff.push_back((int)t.w.size());
        size_t base = t.w.size();
        float sum = 0.0f;
        for (long long i = left; i < right; ++i) {
            float wv = lanczos3(((float)i - input) / sratio);
            t.w.push_back(wv);
            sum += wv;
        }
        for (size_t j = base; j < t.w.size(); ++j) t.w[j] /= sum;
    }
    return t;
}

BlurPlan blur_plan(const SiftCudaParams& p) {
    BlurPlan b;
    b.base = p.sigma > p.assumed_blur ? std::sqrt(p.sigma * p.sigma - p.assumed_blur * p.assumed_blur) : 0.0f;
    if (!(b.base > 1e-4f)) b.base = 0.0f;
    float k = std::pow(2.0f, 1.0f / (float)p.num_intervals);
    std::vector<float> target;
    for (uint32_t s = 0; s < p.num_intervals + 3; ++s) target.push_back(p.sigma * powi(k, (int)s));
    for (uint32_t o = 0; o < p.num_octaves; ++o) {
        float scale = std::ldexp(1.0f, (int)o);
        float prev = p.sigma * scale;
        std::vector<float> row;
        for (uint32_t s = 1; s < p.num_intervals + 3; ++s) {
            float t = target[s] * scale;
            float blur = std::sqrt(t * t - prev * prev);
            row.push_back(blur < 1e-4f ? 0.0f : blur);
            prev = t;
        }
        b.level.push_back(row);
    }
    return b;
}

}  // namespace sift
