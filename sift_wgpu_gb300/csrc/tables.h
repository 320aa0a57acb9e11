// tables.h — host-side filter tables (tables.cpp).
#pragma once

#include <stdint.h>

#include <vector>

#include "../../include/sift_cuda.h"

namespace sift {

struct AxisTaps {
    std::vector<int> left, count, woff;
    std::vector<float> w;
};

struct BlurPlan {
    float base;                             // base blur sigma, 0 = none
    std::vector<std::vector<float>> level;  // [octave][s-1], 0 = copy level
};

// The taps of a blur as the tensor-core level kernel takes them (level_tc.cuh):
// whole-number weights in two limbs, W_i = a_i 2^shift + b_i ~ w_i 2^q, laid
// out as the operand fragments of both passes, and the interval in which the
// reference's rounded sum can lie around the exact one.
struct TcBlur {
    bool ok = false;      // false: a radius or taps the kernel does not take
    int kh = 0, kv = 0;   // 16-wide k-steps of the horizontal and vertical pass
    bool clamp = false;   // sums can reach 256: 9 whole bits and a clamp
    float init_a = 0, init_b = 0, scale_b = 0;  // accumulator start values, 2^-shift
    float whole = 0;      // added with truncation: the whole part to the low mantissa bits
    uint32_t near = 0;    // the exact sum decides below it (the fraction in the top bits)
    std::vector<uint32_t> frags;  // kh x 32 lanes x 4, then kv x 32 lanes x 8
};
TcBlur tc_blur(const std::vector<float>& taps);

std::vector<float> gaussian_kernel(float sigma);
AxisTaps lanczos_axis(uint32_t src, uint32_t dst);
BlurPlan blur_plan(const SiftCudaParams& p);

}  // namespace sift
