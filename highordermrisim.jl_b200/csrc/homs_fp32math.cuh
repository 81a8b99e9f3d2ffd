// FP32 functions of the coil kernel (homs_precess32.cu), on two spins at a time
// (explicit fused multiply-adds: the same results with and without contraction).
#pragma once

#include <cuda_runtime.h>

namespace homs {

// Two FP32 values in one register pair, for packed operations (a product that
// feeds a sum may be contracted into a multiply-add).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
}
__device__ __forceinline__ f32x2 pair(float c) { return pack2(c, c); }
__device__ __forceinline__ f32x2 pfma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 pmul(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 padd(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 pneg(f32x2 a) { return a ^ 0x8000000080000000ull; }

// cos and sin of two angles.  Two-constant Cody-Waite reduction to the nearest
// multiple of pi/2 by fused multiply-adds (below 2^15 the dropped third constant is
// under 4e-11); on [-pi/4, pi/4] sin r = r + r^3 P(r^2), cos r = 1 + r^2 Q(r^2), P and Q
// interpolants at the Chebyshev nodes of the interval (errors 1e-8 and 1e-10); a
// quarter turn swaps the two and a half turn flips both signs.  Within an ulp of
// sincosf.
constexpr float CIS32_RANGE = 32768.0f;  // |x| below this
__device__ __forceinline__ void cis32_pair(f32x2 x, f32x2 &cs, f32x2 &sn) {
    const f32x2 magic = pair(12582912.0f);
    const f32x2 t = pfma(x, pair(0.636619772f), magic);
    const f32x2 k = padd(t, pneg(magic));
    f32x2 r = pfma(k, pair(-1.57079637f), x);
    r = pfma(k, pair(4.37113883e-8f), r);
    const f32x2 z = pmul(r, r);
    f32x2 p = pfma(pair(-0.00019587890880412386f), z, pair(0.008332748270629749f));
    f32x2 c = pfma(pair(2.4463788293265746e-05f), z, pair(-0.0013887589155600576f));
    p = pfma(p, z, pair(-0.1666666466231438f));
    c = pfma(c, z, pair(0.04166665064451703f));
    p = pfma(pmul(r, z), p, r);
    c = pfma(c, z, pair(-0.49999999969119313f));
    c = pfma(c, z, pair(1.0f));
    const float2 s2 = unpack2(p), c2 = unpack2(c), t2 = unpack2(t);
    float co[2], so[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int quad = __float_as_int(e ? t2.y : t2.x);
        const float s = e ? s2.y : s2.x, o = e ? c2.y : c2.x;
        const float a = (quad & 1) ? s : o, b = (quad & 1) ? o : s;
        const unsigned turn = (unsigned)quad << 30;
        co[e] = __uint_as_float(__float_as_uint(a) ^ ((turn + 0x40000000u) & 0x80000000u));
        so[e] = __uint_as_float(__float_as_uint(b) ^ (turn & 0x80000000u));
    }
    cs = pack2(co[0], co[1]);
    sn = pack2(so[0], so[1]);
}

}  // namespace homs
