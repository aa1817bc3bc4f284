// kf_div.hpp -- division by a divisor whose reciprocal is known.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define KF_HD __host__ __device__ __forceinline__
#else
#define KF_HD inline
#endif

namespace kf {

// Divisors between 2^-60 and 2^60 have a reciprocal; that of another one is NaN.
inline double div_reciprocal(double den) { return den >= 0x1p-60 && den <= 0x1p60 ? 1. / den : std::nan(""); }

// num / den with r = div_reciprocal(den): Markstein's correction (P. Markstein, IBM
// J. Res. Dev. 34, 1990): with q within an ulp and r correctly rounded, q + r (num -
// q den) is num / den correctly rounded; one step brings num r there, the second
// rounds.  Bit for bit the division where the quotient lies between 2^-900 and
// 2^900 (the remainder num - q den must not underflow); smaller ones, zeros among
// them, come within 2^-950 of it; infinities, quotients that overflow and divisors
// without a reciprocal give NaN, for which the caller divides.
KF_HD double div_by(double num, double den, double r) {
    double q = num * r;
    q = fma(fma(-q, den, num), r, q);
    return fma(fma(-q, den, num), r, q);
}

}  // namespace kf
