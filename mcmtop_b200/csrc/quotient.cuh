// quotient.cuh -- divisions by a number that several quotients share, rounded
// as the division rounds.
//
// The divisor's correctly rounded reciprocal gives a quotient within an ulp,
// which two fused-multiply-add corrections round correctly (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990: from a quotient within one ulp and a correctly rounded reciprocal the
// correction rounds correctly).  A zero dividend gives a zero whose sign is not
// the division's; the sums that take these quotients start from +0 and do not
// see it.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#ifndef __CUDA_ARCH__
#include <string.h>
#endif

namespace mcm {

// a / b, y = RN(1 / b), for a dividend and a divisor well inside the exponent
// range.
__host__ __device__ __forceinline__ double quotient(double a, double b, double y) {
    double q = a * y;
    double r = fma(-b, q, a);
    q = fma(r, y, q);
    r = fma(-b, q, a);
    return fma(r, y, q);
}
// The high word of v without its sign, times two.
__host__ __device__ __forceinline__ unsigned high_word(double v) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(v) << 1;
#else
    unsigned long long bits;
    memcpy(&bits, &v, sizeof bits);
    return (unsigned)(bits >> 32) << 1;
#endif
}
__host__ __device__ __forceinline__ unsigned low_word(double v) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2loint(v);
#else
    unsigned long long bits;
    memcpy(&bits, &v, sizeof bits);
    return (unsigned)bits;
#endif
}
// |v| in about [2^-500, 2^500]: neither the quotient nor the remainders of
// `quotient` overflow or lose bits.
__host__ __device__ __forceinline__ bool divisor_in_range(double v) { return high_word(v) - (523u << 21) < (1000u << 21); }
// The same, or zero (as a divisor zero has no finite reciprocal).
__host__ __device__ __forceinline__ bool dividend_in_range(double v) {
    return divisor_in_range(v) || (high_word(v) | low_word(v)) == 0u;
}
__host__ __device__ __forceinline__ double divide(double a, double b, double y) {
    return dividend_in_range(a) && divisor_in_range(b) ? quotient(a, b, y) : a / b;
}

}  // namespace mcm
