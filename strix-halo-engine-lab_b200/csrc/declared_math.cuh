// Device forms of the reference's declared scalar math. Each function is the published operation sequence of the
// cited host function, written with explicit round-to-nearest intrinsics so the bits do not depend on compiler flags.
#pragma once
#include "common.cuh"

namespace b200moe {

__device__ __forceinline__ float pow2i(int k) { return __uint_as_float(static_cast<u32>(k + 127) << 23); }

// exp(x) from basic IEEE operations (include/strix/ds41_moe.hpp:38-54): Cody-Waite reduction by ln 2, degree-7 Taylor
// polynomial in Horner form with separate multiply and add, two-step power-of-two scaling.
__device__ __forceinline__ float declared_exp(float x) {
    const float c = fminf(fmaxf(x, -104.0f), 89.0f);  // selects at the end replace the cases, so that several evaluations overlap
    const float n = rintf(__fmul_rn(c, 1.44269504f));
    const float r = __fsub_rn(__fsub_rn(c, __fmul_rn(n, 0.693359375f)), __fmul_rn(n, -2.12194440e-4f));
    float p = 1.98412698e-4f;
    p = __fadd_rn(__fmul_rn(p, r), 1.38888889e-3f);
    p = __fadd_rn(__fmul_rn(p, r), 8.33333333e-3f);
    p = __fadd_rn(__fmul_rn(p, r), 4.16666667e-2f);
    p = __fadd_rn(__fmul_rn(p, r), 1.66666667e-1f);
    p = __fadd_rn(__fmul_rn(p, r), 0.5f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f);
    const int k = static_cast<int>(n), k1 = k / 2, k2 = k - k1;
    float f = __fmul_rn(__fmul_rn(p, pow2i(k1)), pow2i(k2));
    if (x > 88.0f) f = __uint_as_float(0x7f800000u);
    if (x < -103.0f) f = 0.0f;
    return x == x ? f : x;
}
// ln of a positive normal float (include/strix/ds41_moe.hpp:65-79).
__device__ __forceinline__ float declared_log(float y) {
    const u32 bits = __float_as_uint(y);
    int k = static_cast<int>((bits >> 23) & 0xffu) - 127;
    float m = __uint_as_float((bits & 0x7fffffu) | 0x3f800000u);
    if (m > 1.41421356f) { m = __fmul_rn(m, 0.5f); k = k + 1; }
    const float s = __fdiv_rn(__fsub_rn(m, 1.0f), __fadd_rn(m, 1.0f)), s2 = __fmul_rn(s, s);
    float p = 0.111111111f;
    p = __fadd_rn(__fmul_rn(p, s2), 0.142857143f);
    p = __fadd_rn(__fmul_rn(p, s2), 0.2f);
    p = __fadd_rn(__fmul_rn(p, s2), 0.333333333f);
    p = __fadd_rn(__fmul_rn(p, s2), 1.0f);
    const float kf = static_cast<float>(k);
    return __fadd_rn(__fmul_rn(kf, 0.693359375f), __fadd_rn(__fmul_rn(kf, -2.12194440e-4f), __fmul_rn(__fmul_rn(2.0f, s), p)));
}
__device__ __forceinline__ float declared_log1p(float e) {  // ds41_moe.hpp:81-85
    const float u = __fadd_rn(1.0f, e);
    if (u == 1.0f) return e;
    return __fmul_rn(declared_log(u), __fdiv_rn(e, __fsub_rn(u, 1.0f)));
}
__device__ __forceinline__ float sqrt_softplus_score(float z) {  // ds41_moe.hpp:98-100, route_policy.hpp:78-81
    return __fsqrt_rn(z > 20.0f ? z : declared_log1p(declared_exp(z)));
}
__device__ __forceinline__ float sigmoid_score(float z) {  // route_policy.hpp:74-77
    return __fdiv_rn(1.0f, __fadd_rn(1.0f, declared_exp(-z)));
}
// SwiGLU with the shared clamp trait (ds41_moe.hpp:57-60; moe/activation_policy.hpp:22-24). limit = +inf: no clamp.
__device__ __forceinline__ float swiglu_ds41(float gate, float up, float limit) {
    const float g = gate > limit ? limit : gate;
    const float u = up < -limit ? -limit : (up > limit ? limit : up);
    return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, declared_exp(-g))), u);
}

// gfx1151 expf twin at zero correction tables (src/cpu/core/routed_expert.cpp:208-261): Cody-Waite split of
// x * log2(e) with two fused steps, v_exp(a) = float(exp2(double(a))) for |a| < 1, scaled by 2^e.
// The host evaluates exp2 in double with the C library; a double within an ulp or two of it changes the rounded float only when it lands
// within 2^-29 of a float rounding boundary. 2^a = 1 + a P(a), P the series of (2^a - 1) / a (degree 12: the remainder for |a| <= 0.51 is
// 2^-57): the one addition of 1 comes last, so that the sum is off by little more than its own rounding. (With the 1 inside the first pair of
// terms one float came out wrong, 0x1.0dcadep-9, whose double lies 0.44 ulp from the middle of two floats.) 2^e comes in two steps, as a
// subnormal result is then rounded once. Selects replace the cases: outside the two limits e and a are not meaningful and not used, a NaN
// passes through. The result is the host form's for every float, and that of CUDA's exp2(double), scalbnf and branches, whose calls kept
// several evaluations of a warp from overlapping: 551 clocks each where this one takes a third of the instructions.
__device__ __forceinline__ float gfx1151_expf(float x) {
    const float kLog2e = __uint_as_float(0x3fb8aa3bu), kLog2eLo = __uint_as_float(0x32a5705fu);
    const float ph = __fmul_rn(x, kLog2e);
    const float big = __fadd_rn(ph, 12582912.0f), e = __fsub_rn(big, 12582912.0f);  // rint for |ph| < 2^22, its integer in big's low bits
    float pl = __fmaf_rn(x, kLog2e, -ph);
    pl = __fmaf_rn(x, kLog2eLo, pl);
    const double a = static_cast<double>(__fadd_rn(__fsub_rn(ph, e), pl));
    // P = sum of ln(2)^k / k! a^(k - 1), pairwise (Estrin): six dependent steps with the last one instead of thirteen
    const double a2 = __dmul_rn(a, a), a4 = __dmul_rn(a2, a2), a8 = __dmul_rn(a4, a4);
    const double c1 = __fma_rn(0x1.ebfbdff82c58fp-3, a, 0x1.62e42fefa39efp-1), c3 = __fma_rn(0x1.3b2ab6fba4e77p-7, a, 0x1.c6b08d704a0cp-5), c5 = __fma_rn(0x1.430912f86c787p-13, a, 0x1.5d87fe78a6731p-10);
    const double c7 = __fma_rn(0x1.62c0223a5c824p-20, a, 0x1.ffcbfc588b0c7p-17), c9 = __fma_rn(0x1.e4cf5158b8ecap-28, a, 0x1.b5253d395e7c4p-24), c11 = __fma_rn(0x1.c3bd650fc2986p-36, a, 0x1.e8cac7351bb25p-32);
    const double low = __fma_rn(c3, a2, c1), mid = __fma_rn(c7, a2, c5), high = __fma_rn(0x1.816193166d0f9p-40, a4, __fma_rn(c11, a2, c9));
    const double y = __fma_rn(__fma_rn(high, a8, __fma_rn(mid, a4, low)), a, 1.0);
    const int k = min(max(static_cast<int>(__float_as_uint(big) - 0x4b400000u), -160), 160), k1 = k >> 1, k2 = k - k1;
    float f = __fmul_rn(__fmul_rn(static_cast<float>(y), pow2i(k1)), pow2i(k2));
    if (__uint_as_float(0xc2ce8ed0u) > x) f = 0.0f;
    if (__uint_as_float(0x42b17218u) < x) f = __uint_as_float(0x7f800000u);
    return f;
}
__device__ __forceinline__ float swiglu_qwen(float g, float u) {  // routed_expert.cpp:151-153
    return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, gfx1151_expf(-g))), u);
}

}  // namespace b200moe
