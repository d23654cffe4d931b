// Correctly rounded f64 square root and quotients for operands of moderate
// size, as straight-line code.
//
// The language's sqrt and / carry a range test, a branch and an out-of-line
// path each, four of them in a row in a force pair: they split the pair into
// short blocks whose latencies add up. Here the operands of a whole pair are
// range-tested once, and what follows is one block of multiply-adds the
// scheduler can interleave. Operands outside the range take the language's
// operations, so every result is the IEEE one.
//
// Method: the hardware's approximate seeds (relative error 2^-20, measured),
// one third-order Newton step (error 2^-59, so within one unit in the last
// place after rounding), then Markstein's final steps (P. Markstein, "IA-64
// and Elementary Functions", 2000; Cornea, Harrison and Tang, 1999): with y
// within one unit of 1/d, y + y (1 - d y) rounds to RN(1/d) unless d's
// significand is all ones (excluded by quot_ok); with y = RN(1/d) and q within
// one unit of n/d, q + y (n - d q) rounds to RN(n/d); with g within one unit of
// sqrt(a) and h of 1 / (2 sqrt(a)), g + h (a - g g) rounds to RN(sqrt(a)). The
// remainders are exact in a fused multiply-add. tests/test_gpu_exact_math.py
// compares both with IEEE over random operands and over the hardest ones (the
// quotients and roots nearest to a rounding boundary).
#pragma once

#include <cstdint>

namespace pe {

// 2^-128 <= a < 2^128 (positive, so neither NaN nor a negative value passes):
// no intermediate of a quotient or root of such operands leaves the normal range.
__device__ __forceinline__ bool moderate(double a) {
    return (uint32_t)__double2hiint(a) - ((1023u - 128u) << 20) < (256u << 20);
}

// zero, or of moderate magnitude: a numerator
__device__ __forceinline__ bool moderate_or_zero(double a) { return a == 0.0 || moderate(fabs(a)); }

// a divisor that recip_rn rounds correctly (its significand is not all ones)
__device__ __forceinline__ bool divisor_ok(double d) { return (uint32_t)__double2loint(d) != 0xffffffffu; }

// RN(1 / d), d moderate and divisor_ok
__device__ __forceinline__ double recip_rn(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    return fma(y, fma(-d, y, 1.0), y);
}

// RN(n / d) given y = RN(1 / d); a zero's sign may differ from n / d's
__device__ __forceinline__ double quot_rn(double n, double d, double y) {
    const double q = n * y;
    return fma(fma(-d, q, n), y, q);
}

// s = RN(sqrt(a)), a moderate; the return value is within one unit of 1 / s
__device__ __forceinline__ double sqrt_rn(double a, double* s) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    double g = a * y, h = 0.5 * y;
    const double r = fma(-h, g, 0.5);
    const double p = fma(1.5 * r, r, r);
    g = fma(g, p, g);
    h = fma(h, p, h);
    *s = fma(fma(-g, g, a), h, g);
    return h + h;
}

// RN(1 / d) from a y within one unit of it, d divisor_ok
__device__ __forceinline__ double recip_refine(double d, double y) { return fma(y, fma(-d, y, 1.0), y); }

}  // namespace pe
