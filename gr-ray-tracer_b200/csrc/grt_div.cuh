// Correctly rounded FP64 quotients from a shared reciprocal.
//
// The right-hand side of Hamilton's equations divides 21 times by only six
// distinct values, all positive.  Each quotient a/b is formed from
// y = RN(1/b), once per denominator, in three operations:
//   q0 = RN(a y)
//   n  = RN(b q0 - a)
//   q  = RN(q0 - n y)     = RN(a/b)
// Why that is the IEEE quotient for every a and b (no value under- or
// overflowing; significands a, b in [1, 2)):
//   a >= b: |a y - a/b| <= a 2^-54 is at most half an ulp of a/b, so q0 lies
//     within one ulp of a/b, n is exact, and q = RN(a/b) by Markstein's theorem
//     (P. W. Markstein, "Computation of elementary functions on the IBM RISC
//     System/6000 processor", IBM J. Res. Dev. 34(1), 1990: y = RN(1/b) and q0
//     within one ulp give the correctly rounded quotient).
//   a < b: q0 is within 1.5 ulp.  Within one ulp the theorem holds again.  If
//     q0 is further off, q is still RN of a value within 2^-104 of a/b, so it
//     can be wrong only if a/b lies that close to a rounding midpoint, which
//     is then 1.5 ulp from q0: the rounding of a y must supply all of its
//     half ulp and y a full ulp (2^-53) of error.  That needs
//     a 2^-54 >= 2^-53 - 2^-104, i.e. a = 2 - m 2^-52 and b = 2 - k 2^-52 with
//     k < m <= 4; but there a/b = 1 - (m - k) 2^-53 - (m - k) k 2^-106 - ..., next
//     to a representable number and not to a midpoint.
// A second residual step (five operations a quotient) changes nothing, and
// without it a right-hand side has 42 FP64 operations less of about 310 and a
// lone warp waits for two dependent ones less in each of the three quotients
// on its critical path.  Measured with the shorter refinement of grt_rn.cuh and
// without the zero tests, on one B200: 4,096 RK4 rays 3.44 to 2.97 ms, 65,536
// RK45 rays 1.71 to 1.49 ms, 4.76e6 rays in 64 images 59.6 to 51.7 ms,
// 2.1e6 disk packets 81.3 to 72.3 ms.
// Zeros: b q0 - a is +0 for either zero a (the difference of two equal values
// in round-to-nearest), so q0 - n y = q0 + (-0) = q0, the signed zero a/b; no
// test of a.  The sign trick and the comparison above need b > 0.
//
// Every value must stay away from underflow and overflow; the caller
// guarantees it (ks_rhs_rcp checks its inputs against a box in which every
// numerator, denominator and quotient of the right-hand side stays inside
// [2^-900, 2^900]) and uses IEEE divisions outside.  A single-warp ncu probe
// on B200 counts 17 instructions for an IEEE FP64 division, 12 for __drcp_rn
// and 3 for div_by.
#pragma once

#include <cuda_runtime.h>

namespace grt {
namespace dev {

__device__ __forceinline__ double div_recip(double b) { return __drcp_rn(b); }

// a / b for b > 0, y = RN(1/b).
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q0 = a * y;
    const double n = fma(b, q0, -a);
    return fma(-n, y, q0);
}

// v / 2 for a normal v whose half is normal, on the integer pipe.  Zeros,
// subnormals and the smallest normals give a negative number or NaN.
__device__ __forceinline__ double half_of(double v) {
    return __hiloint2double(__double2hiint(v) - 0x00100000, __double2loint(v));
}

// Biased exponent of v (0 for zeros and subnormals, 2047 for inf/NaN).
__device__ __forceinline__ unsigned div_exponent(double v) {
    return (static_cast<unsigned>(__double2hiint(v)) >> 20) & 0x7FFu;
}

// v is an exact zero or 2^lo <= |v| < 2^(hi+1) (lo, hi unbiased).
template <int LO, int HI>
__device__ __forceinline__ bool div_zero_or_within(double v) {
    const unsigned e = div_exponent(v);
    return e == 0u ? (v == 0.0) : (e - static_cast<unsigned>(1023 + LO)) <= static_cast<unsigned>(HI - LO);
}

// The smallest of m and the high word of |v|, an exact zero counting as large:
// a chain over several values ends at or above (1023 + lo) << 20, less one,
// when each is a zero or at least 2^lo (to within one part in 2^20).
__device__ __forceinline__ unsigned div_min_nonzero(unsigned m, double v) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(v)) & 0x7FFFFFFFu;
    const unsigned lo = static_cast<unsigned>(__double2loint(v));
    return min(m, hi + min(lo, 1u) - 1u);  // zero wraps; a subnormal stays small
}

// 2^lo <= |v| < 2^(hi+1), v finite and normal.
template <int LO, int HI>
__device__ __forceinline__ bool div_within(double v) {
    return (div_exponent(v) - static_cast<unsigned>(1023 + LO)) <= static_cast<unsigned>(HI - LO);
}

}  // namespace dev
}  // namespace grt
