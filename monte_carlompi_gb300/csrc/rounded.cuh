// FP64 square roots and quotients from the hardware's approximations: a Newton step, then the
// residual's correction (Markstein, IBM J. Res. Dev. 34, 1990), and what shows that the result is the
// correctly rounded one, as sqrt() and / give it.  The correction misses it only where the exact value
// lies within 2^-28 ulp of the middle between two doubles, which the residual of the result tells:
// about one result in 500,000 is uncertain, and then taken from sqrt() or /.
// (Compiled with --fmad=false.)  And an FP32 reciprocal.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace mcw {

__device__ __forceinline__ uint64_t to_bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ int hi_word(double x) { return __double2hiint(x) & 0x7fffffff; }

// A power-of-two factor by the exponent (normal, finite x).
__device__ __forceinline__ double halved(double x) { return __hiloint2double(__double2hiint(x) - 0x00100000, __double2loint(x)); }
__device__ __forceinline__ double doubled(double x) { return __hiloint2double(__double2hiint(x) + 0x00100000, __double2loint(x)); }

__device__ __forceinline__ double rsqrt_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// sqrt(x), x between 2^-255 and 2^53; h: half its reciprocal.
__device__ __forceinline__ double sqrt_res(double x, double &h) {
    const double y = rsqrt_seed(x), h0 = halved(y);
    const double g = x * y;
    const double r = fma(-g, h0, 0.5);
    const double g1 = fma(g, r, g);
    h = fma(h0, r, h0);
    return fma(fma(-g1, g1, x), h, g1);
}

// 1 / b nearly, |b| between 2^-255 and 2^53.
__device__ __forceinline__ double rcp_res(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return fma(fma(-b, y, 1.0), y, y);
}

// a / b by rb, 1 / b nearly.
__device__ __forceinline__ double quotient_res(double a, double b, double rb) {
    const double q = a * rb;
    return fma(fma(-q, b, a), rb, q);
}

// Whether the residual e lies below t's upper word and 2^-20 of it more: t is the upper word of what
// half an ulp of the result r changes the residual by, and a quarter where r may be a power of two,
// whose lower neighbour is half as far.  Rounding is monotonic, so this holds of the exact residual.
// NaN, infinities and results that are 0 or denormal are not certain.
__device__ __forceinline__ bool residual_small(double e, int r_hi, int t) {
    return hi_word(e) < t - ((r_hi & 0x000fffff) == 0 ? 0x00100000 : 0) - 1;
}

// Whether q is a / b correctly rounded: |a - q b| < |b| ulp(q) / 2.
__device__ __forceinline__ bool quotient_certain(double q, double a, double b) {
    const int qh = hi_word(q);
    return residual_small(fma(-q, b, a), qh, hi_word(b) - (1076 << 20) + (qh & 0x7ff00000));
}

// Whether g > 0 is sqrt(x) correctly rounded: |x - g^2| < g ulp(g) - ulp(g)^2 / 4.
__device__ __forceinline__ bool sqrt_certain(double g, double x) {
    const int gh = hi_word(g);
    return residual_small(fma(-g, g, x), gh, gh + (gh & 0x7ff00000) - (1075 << 20));
}

// Whether |x| lies between 2^-255 and 2^53: the ranges above.
__device__ __forceinline__ bool moderate(double x) {
    const int h = hi_word(x);
    return h >= 0x30000000 && h < 0x43400000;
}

// Whether g = sqrt_res(x) and q = quotient_res(a, b, rcp_res(b)) are sqrt(x) and a / b, of any x, a, b.
__device__ __forceinline__ bool sqrt_sure(double g, double x) {
    return (to_bits(x) >> 63) == 0 & moderate(x) & sqrt_certain(g, x);
}
__device__ __forceinline__ bool quotient_sure(double q, double a, double b) {
    return moderate(b) & quotient_certain(q, a, b);
}

// 1 / d, d >= 1 (or NaN): a Newton step on the hardware's reciprocal, by the same author, which alone
// is correctly rounded here (of every float from 1 to 2^126, which the hardware's flushes from there on).
__device__ __forceinline__ float reciprocal_rn(float d) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    const float s = fmaf(fmaf(-d, y, 1.f), y, y);
    return d > 8.5e37f ? 1.f / d : s;
}

}  // namespace mcw
