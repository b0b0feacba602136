// div_by.h -- x / d for a divisor whose reciprocal is at hand (device code; compiled by the host compiler in its test).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define DFDM_HD __host__ __device__ __forceinline__
#else
#define DFDM_HD inline
#endif

namespace dfdm {

// x / d with r = 1/d rounded: Markstein's correction (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990).  The product x r is within 1.5 ulp of the quotient; its remainder
// comes out of one fused multiply-add, and adding remainder times r leaves an error of half an ulp plus about 2^-52 ulp, so
// the result is the rounded quotient except where that lies within 2^-52 ulp of a rounding boundary, for operands whose
// quotient and remainder are normal numbers.  A quotient that is infinite or not a number (an infinite x, an overflow, d zero
// or infinite) is the product's, since the remainder is then not a number.  Zeros keep their sign where d > 0.
//
// Three dependent operations and a select in place of a divide, for the transforms' normalisations, the division by the wave
// numbers of the periodic y solve, the stored pressure and the wall law.  The select's test is on the exponent bits, in
// integer operations: as comparisons of doubles it cost the 64^3 FP32 step 92.1 us in place of 90.1, the time without it.
DFDM_HD double div_by(double x, double d, double r) {
    const double q = x * r, e = fma(q, d, -x), y = fma(-e, r, q);
#ifdef __CUDA_ARCH__
    const unsigned hi = (unsigned)__double2hiint(y);
#else
    uint64_t bits;
    std::memcpy(&bits, &y, sizeof bits);
    const unsigned hi = (unsigned)(bits >> 32);
#endif
    return (hi & 0x7ff00000u) != 0x7ff00000u ? y : q;
}

}  // namespace dfdm
