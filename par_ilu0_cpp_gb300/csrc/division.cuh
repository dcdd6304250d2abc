// FP64 division by a known divisor: acc / d, for the rows of U and for the pivots of a
// factorisation.  GB300 issues one FP64 instruction per warp in 64 cycles on a scheduler, and a
// division takes about nine of them (566 cycles measured), all on the chain.  With 1/d = hi +
// lo (hi = 1/d rounded towards zero, lo the remainder) the quotient is fma(acc, hi, acc *
// lo): two instructions (128 cycles), its argument within 2^-51 ulp of the exact quotient, so
// it is the correctly rounded quotient unless that lies within 2^-51 ulp of the middle between
// two numbers (double-word reciprocal, as in the literature on division by constants:
// Brisebarre, Muller, Raina, "Accelerating correctly rounded floating-point division when
// the divisor is known in advance", IEEE TC 53(8), 2004).  For divisors just below a power of
// two, 2^k (1 - m 2^-53), that happens with dividends of few bits: acc / d = 2^j (1 + m 2^-53 +
// m^2 2^-106 ..).  These (line_divisor_bad) and divisors outside 2^+-400 have hi = NaN, and a
// quotient outside 2^+-600 (or one that is not finite) is divided again.  hi and lo have the
// same sign, so a zero keeps its sign.
#pragma once

#include <cuda_runtime.h>

namespace gb300 {

constexpr int kLineDivExp = 400;
constexpr int kLineQuoExp = 600;

// Divisors that are not replaced by their reciprocals: too small or large, or with a significand
// within 2^-20 of the next power of two.
__device__ __forceinline__ bool line_divisor_bad(double d) {
    const int h = __double2hiint(d), e = (h >> 20) & 0x7FF;
    return e < 1023 - kLineDivExp || e > 1023 + kLineDivExp || (h & 0xFFFFF) == 0xFFFFF;
}
__device__ __forceinline__ void line_reciprocal(double d, double& hi, double& lo) {
    if (line_divisor_bad(d)) {
        hi = __longlong_as_double(0x7FF8000000000000ll);
        lo = 0.0;
        return;
    }
    hi = __drcp_rz(d);
    lo = fma(-d, hi, 1.0) * hi;  // 1 - d hi is exact: both factors have 53 bits, the result < 2^-52
}
__device__ __forceinline__ double line_quotient(double acc, double hi, double lo) { return fma(acc, hi, acc * lo); }
// Whether acc / d must be divided again (integer operations: the FP64 pipe is what the
// sweep waits for).  0 / d is exact already.
__device__ __forceinline__ bool line_quotient_bad(float, float) { return false; }
__device__ __forceinline__ bool line_quotient_bad(double q, double acc) {
    const unsigned qh = static_cast<unsigned>(__double2hiint(q)), ah = static_cast<unsigned>(__double2hiint(acc));
    constexpr unsigned kLow = static_cast<unsigned>(1023 - kLineQuoExp) << 21;  // exponent above the sign
    constexpr unsigned kSpan = static_cast<unsigned>(2 * kLineQuoExp) << 21;
    const unsigned nonzero = ((qh | ah) << 1) | static_cast<unsigned>(__double2loint(q)) | static_cast<unsigned>(__double2loint(acc));
    return (qh << 1) - kLow > kSpan && nonzero != 0u;
}
static __device__ __noinline__ double line_divide(double acc, const double* d) { return acc / *d; }

// 1 / d = hi + lo as line_reciprocal gives it: |hi| <= |1 / d| within an ulp and lo = hi (1 -
// d hi).  From the 20-bit estimate r0 of rcp.approx by one step of the third-order iteration
// (Chebyshev), r0 (1 + e + e^2) with e = 1 - d r0: r0 is taken 2^-18 below, so that e > 0 and
// the truncated series stays below 1 / d (by e^3 < 2^-52); both roundings go towards zero.
__device__ __forceinline__ void line_pivot_reciprocal(double d, double& hi, double& lo) {
    double r0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(d));
    r0 = __hiloint2double(__double2hiint(r0) - 4, 0);
    const double e = fma(-d, r0, 1.0);
    hi = __fma_rz(r0, __fma_rz(e, e, e), r0);
    lo = hi * fma(-d, hi, 1.0);
    if (line_divisor_bad(d)) {
        hi = __longlong_as_double(0x7FF8000000000000ll);
        lo = 0.0;
    }
}

// What a row of a sweep does last: nothing for L, for U the division by u_ii (FP64, prepared
// while the row's dependencies are awaited) or the product with its reciprocal d (FP32).  A
// division held up the other rows of its warp for 566 cycles each: FP64 GMRES on 21 x 20 x 19
// with holes 5.06 ms, now 4.00.
template <bool UPPER, class T>
struct RowFinish {
    __device__ __forceinline__ explicit RowFinish(T d_) : d(d_) {}
    __device__ __forceinline__ T operator()(T acc) const { return UPPER ? acc * d : acc; }
    T d;
};
template <>
struct RowFinish<true, double> {
    __device__ __forceinline__ explicit RowFinish(double d_) : d(d_) { line_pivot_reciprocal(d, hi, lo); }
    __device__ __forceinline__ double operator()(double acc) const {
        const double q = line_quotient(acc, hi, lo);
        return line_quotient_bad(q, acc) ? line_divide(acc, &d) : q;
    }
    double d, hi, lo;
};

}  // namespace gb300
