// Square root and quotient from an approximate reciprocal square root and fused
// remainders (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990).  For the coarse factor,
// whose critical path runs through one square root and its quotients per
// column: chains of four and three FMAs instead of two library calls.
//
// With y within an ulp or two of 1 / sqrt(s) the values before the last rounding
// are good to about 2^-102 of themselves.  So the results are those of sqrt and
// / but where the exact value lies that close to the middle between two
// doubles: about one operand in 2^48, and then the neighbouring double.
#pragma once

#include <cmath>

namespace gputo {

#if defined(__CUDACC__)
#define GPUTO_HD __host__ __device__ __forceinline__
#else
#define GPUTO_HD inline
#endif

// Pivots in this range keep the square root's products and remainder clear of
// overflow and of subnormal numbers; others take sqrt and /.  So do quotients
// of dividends from 1e-200 to 1e200 by their roots; one that is smaller than
// 1e-300 may be off by its last bits.
GPUTO_HD bool pivot_in_range(double s) { return s > 1e-200 && s < 1e200; }

// sqrt(s) for y = 1 / sqrt(s) within an ulp or two.
GPUTO_HD double sqrt_by(double s, double y)
{
    const double g = s * y;
    return fma(fma(-g, g, s), 0.5 * y, g);
}

// s / d for y = 1 / d to about 2^-51.
GPUTO_HD double div_by(double s, double d, double y)
{
    const double q = s * y;
    return fma(fma(-q, d, s), y, q);
}

}  // namespace gputo
