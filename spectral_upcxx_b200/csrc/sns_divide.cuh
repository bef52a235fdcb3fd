// Several FP64 quotients over one divisor.
//
// The reciprocal r comes from one division.  A quotient is the product q = v r
// corrected once by its remainder, q + (v - q den) r: one step of iterative
// refinement of den q = v, the remainder formed in one FMA (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev.
// 34, 1990).
//
// Bound: r and the product each round once, so q is off by less than 2^-52 + 2^-105
// of the quotient; the roundings of r and of the remainder leave the corrected value
// off by less than 2^-103 before it is rounded itself.  So it is within 1/2 + 2^-50
// ulp, where a division is within 1/2: the same value except next to a rounding
// boundary.  Conditions: 1 <= den <= 2^1000 and a quotient of 2^-960 or more.
// Below, the remainder may underflow, and q keeps the product's error: 2 ulp (or
// smallest doubles).  Infinities and NaN come out as from a division.
//
// The same operations, each rounded alike, in plain C++, where they are tested.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define SNS_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define SNS_HOST_DEVICE inline
#endif

namespace sns {

struct SharedDivisor {
  double den, r;
  SNS_HOST_DEVICE SharedDivisor(double d) : den(d), r(1.0 / d) {}
  SNS_HOST_DEVICE double under(double v) const {
    const double q = v * r;
    const double e = fma(-q, den, v);
    return e == e ? fma(e, r, q) : q;  // an infinite quotient stays infinite
  }
};

}  // namespace sns
