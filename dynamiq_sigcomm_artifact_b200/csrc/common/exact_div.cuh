// Division by a denominator that many values share, correctly rounded, from one reciprocal.
//
// P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM Journal of Research
// and Development 34(1), 1990: with r = 1 / b correctly rounded and q within one unit of a / b, the residual
// fma(-b, q, a) is exact and fma(residual, r, q) is a / b correctly rounded.  a * r may be two units off, so the step
// is taken twice.  Holds while nothing under- or overflows on the way: quotients that are tiny, huge or not finite go
// through the ordinary division.  Five multiply-adds a value, and no branch for a zero numerator.
#pragma once
#include <cuda_runtime.h>

namespace dq {

// The divisor is positive.
struct SharedDivisor {
  float b, r;
  __device__ __forceinline__ explicit SharedDivisor(float divisor) : b(divisor), r(1.0f / divisor) {}

  // the caller knows that the numerator, the divisor and the quotient are within 1e-20 .. 1e20 or does not mind an
  // error of a few units in a quotient below (its sign is right, and zero comes out as zero)
  __device__ __forceinline__ float in_range(float a) const {
    float q = __fmul_rn(a, r);
    q = __fmaf_rn(__fmaf_rn(-b, q, a), r, q);
    return __fmaf_rn(__fmaf_rn(-b, q, a), r, q);
  }

  __device__ __forceinline__ float operator()(float a) const {
    float q = in_range(a);
    const float m = fabsf(q), n = fabsf(a);
    if (!(m >= 1e-20f && m <= 1e20f && n >= 1e-20f && n <= 1e20f)) q = a == 0.0f ? a : __fdiv_rn(a, b);
    return q;
  }
};

}  // namespace dq
