// dfloat.cuh - double-float arithmetic on FP32 pairs and the FP64 -> FP32-pair split.
//
// Compiled into translation units built with -fmad=false: the error-free transforms below rely on
// every sum and product being rounded as written.
#pragma once

#include <cuda_runtime.h>

namespace vedo {
namespace {   // internal linkage: the header is compiled into each engine's translation unit

// Double-float (hi + lo, ~48 bits) arithmetic from error-free FP32 transforms (Knuth's two-sum,
// the FMA two-product).  Both spheres' positions are split into hi/lo FP32 pairs (split32 below),
// then the relative displacement, |d|^2 and the overlap numerator R^2 - |d|^2 need no FP64 work.
// Splits stored once and splits formed when a pair needs them come from the same function on the
// same FP64 positions, so the two ways give identical bits.
struct dfl { float hi, lo; };
__device__ __forceinline__ dfl two_sum(float a, float b) {
    const float s = a + b, bb = s - a;
    return dfl{s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ dfl df_add(dfl a, dfl b) {
    const dfl s = two_sum(a.hi, b.hi);
    return two_sum(s.hi, s.lo + (a.lo + b.lo));
}
// (hm + lm) - (hs + ls)
__device__ __forceinline__ dfl df_diff(float hm, float lm, float hs, float ls) {
    const dfl d = two_sum(hm, -hs);
    return two_sum(d.hi, d.lo + (lm - ls));
}
__device__ __forceinline__ dfl df_sq(dfl a) {
    const float p = a.hi * a.hi;
    return two_sum(p, fmaf(a.hi, a.hi, -p) + 2.0f * a.hi * a.lo);
}
// x = hi + lo with hi = x rounded to FP32 (nearest, ties to even) and lo = (x - hi) rounded to
// FP32, from the bits of x with integer operations (GB300's FP64 pipe is its scarcest): for
// 2^-70 <= |x| < 2^101; zero, tiny and huge values take the FP64 conversions.
// The FP64 conversions of the rare exponents, out of line: GB300 issues FP64 conversions on its
// FP64 pipe (2 lanes per cycle per SM), and a short branch kept inline is predicated rather than
// jumped over, so its FP64 instructions would be issued on every call.
__device__ __noinline__ void split32_wide(double x, float& hi, float& lo) {
    hi = (float)x;
    lo = (float)(x - (double)hi);
}
__device__ __forceinline__ void split32(double x, float& hi, float& lo) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int e = (int)((u >> 52) & 0x7ff) - 1023;           // unbiased exponent
    if (e < -70 || e > 100) {                                  // 2^(e-52) below stays a normal FP32
        split32_wide(x, hi, lo);
        return;
    }
    const unsigned long long mant = u & 0xfffffffffffffull;   // 52 bits
    const unsigned sign = (unsigned)(u >> 63) << 31;
    const unsigned m23 = (unsigned)(mant >> 29);
    const unsigned rem = (unsigned)(mant & 0x1fffffffu);      // 29 bits below FP32's mantissa
    const bool up = rem > 0x10000000u || (rem == 0x10000000u && (m23 & 1u));
    // exponent and mantissa as one integer: a carry out of the mantissa bumps the exponent
    const unsigned body = (((unsigned)(e + 127)) << 23) + m23 + (up ? 1u : 0u);
    hi = __uint_as_float(sign | body);
    // x - hi = (rem or rem - 2^29) units of 2^(e - 52), exactly; its FP32 rounding
    const int r = up ? (int)rem - (int)0x20000000 : (int)rem;
    const float unit = __uint_as_float((unsigned)(e - 52 + 127) << 23);   // 2^(e-52)
    const float lr = __int2float_rn(r) * unit;
    lo = r == 0 ? 0.0f : (sign ? -lr : lr);                     // x - hi = +0 when exact
}

}  // namespace
}  // namespace vedo
