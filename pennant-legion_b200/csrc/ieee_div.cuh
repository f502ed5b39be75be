// ieee_div.cuh -- correctly rounded FP64 quotients and square roots without
// branches, for operands whose ranges are checked once for a whole group.
//
// The division operator tests its operands and branches to a slow path, so
// consecutive quotients run one after another, each a chain of dependent
// FMAs; pass A needs up to 37 quotients and 25 roots a zone.  Here the same
// results are formed in straight-line code, which the compiler interleaves,
// quotients over one divisor share its reciprocal, and every operand's
// range goes into a Guard that the caller tests once: a zone with any
// operand out of range is formed again with the operators.  Only the
// dividends of quot_unchecked are the caller's to check: against their upper
// limit (Guard::below), and for what too small a one does to its result.
//
// Quotients (P. Markstein, IBM J. Res. Dev. 34 (1990) 111; M. Cornea, J.
// Harrison, P. Tang, "Scientific Computing on Itanium-based Systems", 2002).
// rcp: y0 from the reciprocal instruction, |e| = |1 - b y0| < 2^-19.9 (at
// every mantissa that it distinguishes: tests/test_gpu_ieee_div.py), y1 = y0 (1 + e + e^2), within 0.52
// ulp of 1/b, and y = y1 + y1 (1 - b y1), which is 1/b correctly rounded by
// Markstein's theorem unless b's mantissa is all ones; there 1/b rounds to a
// power of two plus one ulp.  quot: q0 = a y, r = a - b q0, q = q0 + r y, the
// correctly rounded quotient for a correctly rounded y (his second theorem).
//
// Roots: with e = 1 - s y0, s = x y0, |e| < 2^-19.0, g = s (1 + e/2 + 3/8
// e^2) is within 1.02 ulp, h likewise is 1/(2 sqrt x) to 2^-52.3, and g +
// (x - g^2) h is within 2^-53 ulp of the root before its rounding.  A root is
// that near a midpoint M/2 only if 4x - M^2 is one of a few small odd
// numbers; the test enumerates those x and tries each.
//
// In range (Guard): divisors in 2^-200 .. 2^200, dividends 0 or in 2^-700 ..
// 2^300, radicands in 2^-850 .. 2^400; no intermediate then overflows,
// underflows or loses the exactness of a remainder.
#pragma once

#include <cuda_runtime.h>

namespace pnt {
namespace ieee {

// Which operands were out of range: the largest (exponent word - lowest
// allowed) seen for divisors, for dividends and for radicands (unsigned, so
// values below the range wrap to large ones).
struct Guard {
    unsigned den = 0u, num = 0u, rad = 0u, big = 0u;

    __device__ __forceinline__ static unsigned lo2(int e) { return (unsigned)(1023 + e) << 21; }   // 2 x high word
    __device__ __forceinline__ void divisor(double b) {
        den = max(den, ((unsigned)__double2hiint(b) << 1) - lo2(-200));
    }
    __device__ __forceinline__ void dividend(double a) {
        num = max(num, ((unsigned)__double2hiint(a) << 1) - lo2(-700));
    }
    __device__ __forceinline__ void below(double a) {   // |a| < 2^300, and any zero or tiny value
        big = max(big, (unsigned)__double2hiint(a) << 1);
    }
    __device__ __forceinline__ void radicand(double x) {   // a sign bit is out of range
        rad = max(rad, (unsigned)__double2hiint(x) - ((unsigned)(1023 - 850) << 20));
    }
    __device__ __forceinline__ bool ok() const {
        return den < (400u << 21) && num < (1000u << 21) && rad < (1250u << 20) && big < lo2(300);
    }
};

// 1 / b.
__device__ __forceinline__ double rcp(double b, Guard& g) {
    g.divisor(b);
    double y0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
    const double e = __fma_rn(-b, y0, 1.0);
    const double y1 = __fma_rn(y0, __fma_rn(e, e, e), y0);
    const double y = __fma_rn(__fma_rn(-b, y1, 1.0), y1, y1);
    const unsigned ones = (unsigned)__double2loint(b) & ((unsigned)__double2hiint(b) | 0xfff00000u);
    return (ones == 0xffffffffu) ? __hiloint2double(__double2hiint(y), 1) : y;
}
// a / b from y = rcp(b) for a in range or +0; smaller a give some value
// below 2^-499.  For |a| of 2^300 or more (Guard::below) it may be a NaN.
__device__ __forceinline__ double quot_unchecked(double a, double b, double y) {
    const double q0 = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q0, a), y, q0);
}
// a / b from y = rcp(b), a not zero.
__device__ __forceinline__ double quot(double a, double b, double y, Guard& g) {
    g.dividend(a);
    return quot_unchecked(a, b, y);
}
// a / b from y = rcp(b), a possibly a zero (the quotient is then a zero with
// the XOR of the signs, which a y is).
__device__ __forceinline__ double quot0(double a, double b, double y, Guard& g) {
    const bool zero = a == 0.0;
    g.dividend(zero ? 1.0 : a);
    const double q0 = __dmul_rn(a, y);
    const double q = __fma_rn(__fma_rn(-b, q0, a), y, q0);
    return zero ? q0 : q;
}
// a / b where b is often exactly 1 and a may be of any size then.
__device__ __forceinline__ double quot1(double a, double b, Guard& g) {
    const bool one = b == 1.0;
    const double q = quot0(one ? 1.0 : a, b, rcp(b, g), g);
    return one ? a : q;
}
__device__ __forceinline__ double root(double x, Guard& g) {
    g.radicand(x);
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
    const double s = __dmul_rn(x, y0);
    const double e = __fma_rn(-s, y0, 1.0);
    const double t = __dmul_rn(e, __fma_rn(e, 0.375, 0.5));
    const double r = __fma_rn(s, t, s);
    const double hy = __dmul_rn(0.5, y0);
    const double h = __fma_rn(hy, t, hy);
    return __fma_rn(__fma_rn(-r, r, x), h, r);
}

}  // namespace ieee
}  // namespace pnt
