// FP64 helpers built for this GPU's FP64 pipe.  Measured on a GB300 (one dependent chain
// per warp, clock64): every FP64-pipe warp instruction - DFMA, DADD, DMUL, and also DSETP
// and DMNMX - holds its SM sub-partition for 64 cycles, whatever the number of active
// lanes and independent chains; so does every FP64 <-> FP32 or integer conversion (56 to
// 64 cycles).  An integer or FP32 instruction takes 1 or 2.  So comparisons, signs,
// minima and conversions are done on the bit patterns here, and reciprocals, quotients
// and square roots start from an FP32 seed and take 3, 5 and 4 or 5 FP64 instructions
// (the operators: about 5.5, 8.8 and 9.5 by the same measurement).
//
// Reciprocal: Householder's iteration of third order, r = r0 (1 + e + e^2), e = 1 - x r0,
// from an FP32 seed with |e| <= 2^-21: the remainder e^3 is below 2^-63.  Square root: the
// binomial series of (1 - e)^(-1/2) to second order at y0 ~ x^(-1/2), e = 1 - x y0^2.
// Arguments outside the seed's range go to the operators.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hf {

// Bit patterns are taken by __double2hiint / __double2loint throughout: tests on a
// reinterpreted 64-bit integer are recognised by the compiler and turned back into FP64
// comparisons.
__device__ __forceinline__ unsigned fp_abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
__device__ __forceinline__ unsigned long long fp_abs_bits(double x) {
    return (unsigned long long)fp_abs_hi(x) << 32 | (unsigned)__double2loint(x);
}
__device__ __forceinline__ bool fp_zero(double x) { return (fp_abs_hi(x) | (unsigned)__double2loint(x)) == 0; }
__device__ __forceinline__ double fp_bits(unsigned long long b) {
    return __hiloint2double((int)(b >> 32), (int)(unsigned)b);
}
__device__ __forceinline__ bool fp_finite(double x) { return fp_abs_hi(x) < 0x7ff00000u; }
__device__ __forceinline__ bool fp_nan(double x) { return fp_abs_bits(x) > 0x7ff0000000000000ull; }
// x < 0.0 and x >= 0.0, both false for a NaN (its sign bit may be set, and the NaN of an
// invalid operation has it set); -0.0 is not negative
__device__ __forceinline__ bool fp_neg(double x) {
    return __double2hiint(x) < 0 && fp_abs_bits(x) - 1 < 0x7ff0000000000000ull;
}
// x < 0.0 or a NaN with its sign bit set: shorter, for states that are refused for either
__device__ __forceinline__ bool fp_neg_or_nan(double x) { return __double2hiint(x) < 0 && !fp_zero(x); }
__device__ __forceinline__ bool fp_ge0(double x) {
    return __double2hiint(x) >= 0 ? fp_abs_bits(x) <= 0x7ff0000000000000ull : fp_zero(x);
}
// x > 0.0 (false for a NaN)
__device__ __forceinline__ bool fp_pos(double x) { return __double2hiint(x) >= 0 && !fp_zero(x) && !fp_nan(x); }
// order of the bit patterns as integers = order of the numbers (no NaN; -0.0 < +0.0)
__device__ __forceinline__ long long fp_order(double x) {
    const int hi = __double2hiint(x), s = hi >> 31;
    return (long long)(hi ^ (s & 0x7fffffff)) << 32 | (unsigned)(__double2loint(x) ^ s);
}
__device__ __forceinline__ bool fp_lt(double a, double b) { return fp_order(a) < fp_order(b); }
__device__ __forceinline__ double fp_min(double a, double b) { return fp_lt(b, a) ? b : a; }
__device__ __forceinline__ double fp_max(double a, double b) { return fp_lt(a, b) ? b : a; }
__device__ __forceinline__ double fp_abs_max(double a, double b) {  // max(|a|, |b|) as a magnitude
    const unsigned long long x = fp_abs_bits(a), y = fp_abs_bits(b);
    return fp_bits(x > y ? x : y);
}

// The FP64 forms of the rare cases, out of line: inlined, the compiler would execute them
// ahead of the test that avoids them.
static __device__ __noinline__ double fp_half_lib(double x) { return 0.5 * x; }
static __device__ __noinline__ bool fp_prod_pos_lib(double x, double y) { return x * y > 0.0; }

// x/2 (exponent decrement; denormal results by the product)
__device__ __forceinline__ double fp_half(double x) {
    if (fp_abs_hi(x) - 0x00200000u < 0x7fd00000u) return __hiloint2double(__double2hiint(x) - 0x00100000, __double2loint(x));
    return fp_zero(x) ? x : fp_half_lib(x);
}

// x rounded toward zero to FP32; 0 below the FP32 normal range, infinity above it
__device__ __forceinline__ float fp_to_f32(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned mag = hi & 0x7fffffffu;
    unsigned b = __funnelshift_l(lo, mag - 0x38000000u, 3);
    b = mag < 0x38100000u ? 0u : b;
    b = mag >= 0x47f00000u ? 0x7f800000u : b;
    return __uint_as_float(b | (hi & 0x80000000u));
}
// FP64 value of a finite FP32 number; 0 below the FP32 normal range
__device__ __forceinline__ double fp_from_f32(float f) {
    const unsigned b = __float_as_uint(f), m = b & 0x7fffffffu;
    const double d = __hiloint2double((int)(((m >> 3) + 0x38000000u) | (b & 0x80000000u)), (int)(b << 29));
    return m < 0x00800000u ? 0.0 : d;
}

__device__ __forceinline__ float fp_rcp_seed(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float fp_rsqrt_seed(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// 2^-100 <= |x| < 2^100: the seed and the products of the iterations stay normal
__device__ __forceinline__ bool fp_seedable(double x) { return fp_abs_hi(x) - 0x39b00000u < 0x0c800000u; }

static __device__ __noinline__ double fp_rcp_lib(double x) { return 1.0 / x; }
static __device__ __noinline__ double fp_div_lib(double a, double b) { return a / b; }
static __device__ __noinline__ double fp_sqrt_lib(double x) { return sqrt(x); }

// 1/x within 1 ulp
__device__ __forceinline__ double fp_rcp(double x) {
    if (!fp_seedable(x)) return fp_rcp_lib(x);
    const double r = fp_from_f32(fp_rcp_seed(fp_to_f32(x)));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
// a/b within 1 ulp (a: any finite number whose quotient is normal, or 0)
__device__ __forceinline__ double fp_div(double a, double b) {
    if (!fp_seedable(b) || !(fp_zero(a) || fp_seedable(a))) return fp_div_lib(a, b);
    const double r0 = fp_from_f32(fp_rcp_seed(fp_to_f32(b)));
    const double r = fma(r0, fma(-b, r0, 1.0), r0);  // 42 bits
    const double q = a * r;
    return fma(fma(-b, q, a), r, q);
}
// sqrt(x) within 1 ulp (norms and step sizes)
__device__ __forceinline__ double fp_sqrt(double x) {
    if (__double2hiint(x) < 0 || !fp_seedable(x)) return fp_sqrt_lib(x);
    const double y = fp_from_f32(fp_rsqrt_seed(fp_to_f32(x)));
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    const float f = fp_to_f32(e);
    return fma(t, fma(0.5, e, fp_from_f32(0.375f * f * f)), t);
}
// sqrt(x): h = x y rounds, and its own remainder x - h^2 (exact) corrects it, so the result is off
// by half a unit and 2^-10 of one; one instruction more
__device__ __forceinline__ double fp_sqrt_near(double x) {
    if (__double2hiint(x) < 0 || !fp_seedable(x)) return fp_sqrt_lib(x);
    const double y = fp_from_f32(fp_rsqrt_seed(fp_to_f32(x)));
    const double h = x * y, t = fma(-h, h, x) * y;  // sqrt(x) = h + t (1/2 + 3/8 e + ...), e = t / sqrt(x)
    return fma(t, 0.5 + fp_from_f32(0.375f * fp_to_f32(t) * fp_to_f32(y)), h);
}

}  // namespace hf
