// Correctly rounded a / b from y = 1 / b (correctly rounded): P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor"
// (IBM J. Res. Dev. 34, 1990). When q is within an ulp of a / b, the remainder
// r = a - b q is exact in one fused multiply-add and q + r y rounds to a / b.
// The first correction brings a y within an ulp, the second rounds. Many
// quotients share one divisor here, and this is five dependent operations
// where a division is a long sequence. Outside a range where no intermediate
// can overflow or lose bits it divides.
#pragma once
#include <cmath>

namespace cs {

__host__ __device__ __forceinline__ bool div_rn_divisor(double b) {
  const double ab = fabs(b);
  return ab > 1e-80 && ab < 1e80;
}
// Whether div_rn_fast(a, ...) is the quotient (up to the sign of a zero): a is
// zero or its exponent lies in [-664, 664]. An integer test, off the FP64 pipe.
__host__ __device__ __forceinline__ bool div_rn_dividend(double a) {
#ifdef __CUDA_ARCH__
  const int hi = __double2hiint(a) & 0x7fffffff, lo = __double2loint(a);
#else
  long long bits;
  __builtin_memcpy(&bits, &a, 8);
  const int hi = (int)((unsigned long long)bits >> 32) & 0x7fffffff, lo = (int)bits;
#endif
  return (unsigned)(hi - (359 << 20)) < (unsigned)(1329 << 20) || (hi | lo) == 0;
}
__host__ __device__ __forceinline__ double div_rn_fast(double a, double b, double y) {
  const double q0 = a * y;
  const double q1 = fma(fma(-b, q0, a), y, q0);
  return fma(fma(-b, q1, a), y, q1);
}

}  // namespace cs
