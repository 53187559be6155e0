// Quotients from a kept reciprocal.
#pragma once
#include <cuda_runtime.h>

namespace wtk {

// a / b from y = RN(1 / b) (__drcp_rn or 1.0 / b), correctly rounded: the quotient
// estimate a y is within two units in the last place, one residual correction
// makes it faithful and, by Markstein's theorem (P. Markstein, IBM J. Res. Dev.
// 34(1), 1990), the second rounds it as the division does.  That holds for a normal
// quotient, b and y normal (|b| in 2^-1022 .. 2^1022: the divisors are edge lengths and
// densities) and no underflow in the residual (|a| above 2^-960 or so).  A zero,
// subnormal, infinite or NaN estimate is returned as it is, with its sign: the
// division's value, but for a last unit of a subnormal one.  Five dependent operations
// replace a division's some fifteen instructions wherever quotients share a divisor.
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q0 = a * y;
  const double q1 = fma(fma(-b, q0, a), y, q0);
  const double q2 = fma(fma(-b, q1, a), y, q1);
  return ((unsigned)__double2hiint(q0) & 0x7ff00000u) - 0x00100000u < 0x7fe00000u ? q2 : q0;
}

}  // namespace wtk
