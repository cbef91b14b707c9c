// FP64 divide and square root without branches, for operands of moderate
// exponent; the callers test the operands and redo a cell or face with the
// IEEE operations (/, sqrt) where the test fails.
//
// The compiler's FP64 divide and square root test every operand pair and
// branch, so a stencil's ~75 divides per cell form as many basic blocks and
// the arithmetic of the five variables cannot overlap: the FP64 stencils were
// bound by that latency (FP64 pipe 43 % busy). Here the operands' exponents are
// tested with a few integer operations per reconstruction or face, so one
// branch remains for all of them, and quotients by the same divisor share its
// reciprocal.
//
// Divide: from the hardware's reciprocal seed y0 (rcp.approx.ftz.f64; it sees
// the upper 32 bits of b and returns as many, relative error e = 1 - b y0
// below 2^-18) y = y0 (1 + e + e^2) is 1/b to e^3 < 2^-54 before its rounding, and
//   q0 = RN(a y),  r = RN(a - b q0),  q = RN(q0 + r y),
// Markstein's correction (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990). q0 is within
// 1.6 ulp of a / b; a - b q0 is exact where q0 is within one ulp, and rounded in its
// 54th bit beyond. Either way q0 + r y misses a / b by less than 2^-51 ulp (r's
// rounding and y's error, each about 2^-53 of at most 1.6 ulp), and q is the
// correctly rounded quotient unless a / b lies that close to the middle between
// two FP64 numbers (of random operands, one pair in 2^50), where it may be the
// other neighbour. The known such pairs are a divisor whose mantissa is all ones and
// a power of two: 1 / b lies just above a middle, and from a seed below 1 / b its
// reciprocal ends on the wrong side. The lower word of y0, zero from the hardware, is
// therefore set so that y0 is raised by 2^-21: above 1 / b for such a divisor, and
// e^3 < 0 puts y on the right side. For b = 6, a / b is at least 1/6 ulp from any
// middle, so there q is always the correctly rounded quotient.
// Square root: with g = a y, h = y / 2 from the seed y ~ 1 / sqrt(a) and
// e = 1/2 - g h = (1 - a y^2) / 2, sqrt(a) = g (1 - 2 e)^-1/2 = g (1 + e + 3/2 e^2 +
// 5/2 e^3 + ...), and 1 / (2 sqrt(a)) = h (1 + e + ...) likewise: both to 2.5 |e|^3.
// Then g + (a - g^2) h is one Newton step: with g within d <= 1.6 ulp it misses
// sqrt(a) by d^2 2^-54 ulp of its own, d 2^-53 of the residual's rounding and d 2^-52
// of h, again less than 2^-51 ulp, with the same consequence.
// Nothing overflows or is flushed for divisors and square root arguments in
// [2^-900, 2^900] and dividends and quotients that are zero or in [2^-900, 2^900]
// (dividends also above, up to the largest number).
// tests/fp64_range_check.cu draws operands over all of that range and, by
// construction, quotients and roots next to a middle: of 1e10 trials of each kind
// none differs from the IEEE operation at 2^-51 ulp or more from a middle, 184 of
// some 3e9 nearer do, by one ulp.
#pragma once
#include "vb_ns.h"
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace VB_NS {
namespace d64 {

// upper word of x: sign, exponent, 20 bits
__host__ __device__ __forceinline__ uint32_t hi(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return (uint32_t)(u >> 32);
#endif
}
__host__ __device__ __forceinline__ uint32_t lo(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return (uint32_t)u;
#endif
}
constexpr uint32_t hi_pow2(int e) { return (uint32_t)(1023 + e) << 20; }
// x in [2^A, 2^B), by its sign and exponent bits (false for NaN and negatives)
template <int A, int B> __host__ __device__ __forceinline__ bool pos_in(double x) {
    return hi(x) - hi_pow2(A) < hi_pow2(B) - hi_pow2(A);
}
// |x| in [2^A, 2^B)
template <int A, int B> __host__ __device__ __forceinline__ bool abs_in(double x) {
    return (hi(x) & 0x7fffffffu) - hi_pow2(A) < hi_pow2(B) - hi_pow2(A);
}
__host__ __device__ __forceinline__ bool is_zero(double x) { return ((hi(x) & 0x7fffffffu) | lo(x)) == 0; }
// x is zero or |x| in [2^A, 2^B)
template <int A, int B> __host__ __device__ __forceinline__ bool zero_or_in(double x) {
    return abs_in<A, B>(x) || is_zero(x);
}

// a divisor with its reciprocal
struct Div {
    double b, y;
};
__host__ __device__ __forceinline__ Div divisor(double b) {
    Div d;
    d.b = b;
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = __hiloint2double(__double2hiint(y), (int)0x80000000);
    const double e = fma(-b, y, 1.0);
    d.y = fma(y, fma(e, e, e), y);
#else
    d.y = 1.0 / b;
#endif
    return d;
}
// a / b for a >= +0, or where the sign of a zero quotient does not matter
__host__ __device__ __forceinline__ double quot(double a, const Div& d) {
#ifdef __CUDA_ARCH__
    const double q = a * d.y;
    return fma(fma(-d.b, q, a), d.y, q);
#else
    return a / d.b;
#endif
}
// a / b with the sign of a zero quotient: fma(0, y, -0) above is +0
__host__ __device__ __forceinline__ double quot_s(double a, const Div& d) {
#ifdef __CUDA_ARCH__
    const double q = a * d.y;
    const double r = fma(fma(-d.b, q, a), d.y, q);
    return __hiloint2double(__double2hiint(r) | (__double2hiint(q) & (int)0x80000000), __double2loint(r));
#else
    return a / d.b;
#endif
}
// a / 6
__host__ __device__ __forceinline__ double sixth(double a) {
    Div d;
    d.b = 6.0;
    d.y = 1.0 / 6.0;
    return quot_s(a, d);
}
// square root of a > 0
__host__ __device__ __forceinline__ double root(double a) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    double g = a * y, h = 0.5 * y;
    const double e = fma(-g, h, 0.5);
    const double c = fma(1.5 * e, e, e);
    g = fma(g, c, g);
    h = fma(h, c, h);
    return fma(fma(-g, g, a), h, g);
#else
    return sqrt(a);
#endif
}

}  // namespace d64
}  // namespace VB_NS
