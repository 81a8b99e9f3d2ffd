// FP32 functions of the precession and excitation kernels (explicit fused
// multiply-adds: the same results with and without contraction).
#pragma once

#include <cuda_runtime.h>

namespace homs {

// cos and sin on [-pi/4, pi/4]: sin r = r + r^3 P(r^2), cos r = 1 + r^2 Q(r^2), P and Q
// interpolants at the Chebyshev nodes of the interval (errors 1e-8 and 1e-10).
__device__ __forceinline__ void cis32_eighth(float r, float &cs, float &sn) {
    const float z = r * r;
    float p = -0.00019587890880412386f, c = 2.4463788293265746e-05f;
    p = __fmaf_rn(p, z, 0.008332748270629749f);
    c = __fmaf_rn(c, z, -0.0013887589155600576f);
    p = __fmaf_rn(p, z, -0.1666666466231438f);
    c = __fmaf_rn(c, z, 0.04166665064451703f);
    sn = __fmaf_rn(r * z, p, r);
    c = __fmaf_rn(c, z, -0.49999999969119313f);
    cs = __fmaf_rn(c, z, 1.0f);
}

// cos and sin of an angle in FP32.  Two-constant Cody-Waite reduction to the
// nearest multiple of pi/2 by fused multiply-adds (below 2^15 the dropped third
// constant is under 4e-11); within an ulp of sincosf.
constexpr float CIS32_RANGE = 32768.0f;  // |x| below this
__device__ __forceinline__ void cis32(float x, float &cs, float &sn) {
    constexpr float MAGIC = 12582912.0f;  // 1.5 * 2^23: adds round to an integer
    const float t = __fmaf_rn(x, 0.636619772f, MAGIC);
    const int quad = __float_as_int(t);
    const float k = t - MAGIC;
    float r = __fmaf_rn(k, -1.57079637f, x);
    r = __fmaf_rn(k, 4.37113883e-8f, r);
    float s, c;
    cis32_eighth(r, c, s);
    // a quarter turn swaps the two and a half turn flips both signs
    const float a = (quad & 1) ? s : c, b = (quad & 1) ? c : s;
    const unsigned turn = (unsigned)quad << 30;
    cs = __uint_as_float(__float_as_uint(a) ^ ((turn + 0x40000000u) & 0x80000000u));
    sn = __uint_as_float(__float_as_uint(b) ^ (turn & 0x80000000u));
}

}  // namespace homs
