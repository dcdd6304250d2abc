// FP64 division by a known divisor: acc / d, for the rows of U and for the pivots of a
// factorisation.  GB300 issues one FP64 instruction per warp in 64 cycles on a scheduler, and a
// division takes about nine of them (566 cycles measured), all on the chain.  With z = 1 / d
// rounded to nearest it takes three: q0 = acc z, r = acc - d q0, q = q0 + r z.  This is the last
// step of Markstein's division ("Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990), and q is the correctly rounded quotient:
//
// with d, acc in [1, 2) (other scales are the same), z in (1/2, 1] is off by 2^-54 at most, so
// acc z is less than a unit in the last place off acc / d, and q0 one of acc / d's two
// neighbours wherever that lies next to the middle between them.  There r is exact and q0 + r z
// is off by half a unit times 2^-54 d, which is less than any quotient's distance from a middle
// (1 / (2 D) units, D the significand of d as an integer of 53 bits).  Elsewhere an error of
// that order does not matter.
//
// Two instructions, with 1 / d in two parts (fma(acc, hi, acc lo)), do not do: every divisor has
// dividends whose quotient lies nearer to a middle than their error (2^-51 units).  Testing each
// such quotient beside the chain cost more than the third instruction (128^3 FP64 backward sweep,
// us: untested 179, tested in integers 234, by a second sum 219).
//
// Divisors outside 2^+-400 have z = NaN, and a quotient outside 2^+-500 (whose r might be
// subnormal), of -0 or that is not finite is divided.
#pragma once

#include <cuda_runtime.h>

namespace gb300 {

constexpr int kLineDivExp = 400;
constexpr int kLineQuoExp = 500;

// Divisors too small or large to be replaced by their reciprocals.
__device__ __forceinline__ bool line_divisor_bad(double d) {
    const int e = (__double2hiint(d) >> 20) & 0x7FF;
    return e < 1023 - kLineDivExp || e > 1023 + kLineDivExp;
}
__device__ __forceinline__ double line_reciprocal(double d) {
    return line_divisor_bad(d) ? __longlong_as_double(0x7FF8000000000000ll) : 1.0 / d;
}
__device__ __forceinline__ double line_quotient(double acc, double d, double z) {
    const double q = acc * z;
    return fma(fma(-d, q, acc), z, q);
}
// Whether acc / d must be divided again (integer operations: the FP64 pipe is what the
// sweep waits for).  0 / d is exact already.
__device__ __forceinline__ bool line_quotient_bad(float, float) { return false; }
__device__ __forceinline__ bool line_quotient_bad(double q, double acc) {
    const unsigned qh = static_cast<unsigned>(__double2hiint(q)) << 1;
    constexpr unsigned kLow = static_cast<unsigned>(1023 - kLineQuoExp) << 21;  // exponent above the sign
    constexpr unsigned kSpan = static_cast<unsigned>(2 * kLineQuoExp) << 21;
    const unsigned nonzero = qh | static_cast<unsigned>(__double2hiint(acc)) | static_cast<unsigned>(__double2loint(q)) |
                             static_cast<unsigned>(__double2loint(acc));
    return qh - kLow > kSpan && nonzero != 0u;
}
// (not inlined: its operands are at hand, and the compiler would divide beside the test)
static __device__ __noinline__ double line_divide(double acc, double d) { return acc / d; }

// 1 / d for the kernels that need it in a chain or per row: from the 20-bit estimate r0 of
// rcp.approx by one step of the fourth-order iteration (Chebyshev), r0 (1 + e + e^2 + e^3) with
// e = 1 - d r0, |e| < 2^-19.  It is off by up to 2^-18 more than half a unit in the last place,
// for which the argument above has no room with d within 2^-18 of the next power of two: those
// divisors are divided by.
__device__ __forceinline__ double line_pivot_reciprocal(double d) {
    double r0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(d));
    const double e = fma(-d, r0, 1.0);
    const double z = fma(r0, fma(e, fma(e, e, e), e), r0);
    const bool bad = line_divisor_bad(d) || (__double2hiint(d) & 0xFFFF0) == 0xFFFF0;
    return bad ? __longlong_as_double(0x7FF8000000000000ll) : z;
}

// What a row of a sweep does last: nothing for L, for U the division by u_ii (FP64, its
// reciprocal prepared while the row's dependencies are awaited) or the product with its
// reciprocal d (FP32).  A division holds up the other rows of its warp for 566 cycles each:
// FP64 GMRES on 21 x 20 x 19 with holes took 5.06 ms with it and 4.00 without.
template <bool UPPER, class T>
struct RowFinish {
    __device__ __forceinline__ explicit RowFinish(T d_) : d(d_) {}
    __device__ __forceinline__ T operator()(T acc) const { return UPPER ? acc * d : acc; }
    T d;
};
template <>
struct RowFinish<true, double> {
    __device__ __forceinline__ explicit RowFinish(double d_) : d(d_), z(line_pivot_reciprocal(d_)) {}
    __device__ __forceinline__ double operator()(double acc) const {
        const double q = line_quotient(acc, d, z);
        return line_quotient_bad(q, acc) ? line_divide(acc, d) : q;
    }
    double d, z;
};

}  // namespace gb300
