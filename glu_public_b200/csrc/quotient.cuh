// Division by a divisor whose reciprocal is known, for the chains of pivots.
#pragma once

#include <cuda_runtime.h>

namespace glu {

__device__ __forceinline__ bool finite_bits(double x) {
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

// x / d from r = 1 / d with one FMA correction (Markstein's division: q = x r, e = x - q d,
// q + e r; Muller et al., Handbook of Floating-Point Arithmetic, 2nd ed., sec. 4.7): within an ulp
// of x / d, three dependent operations, and no slow path for the zeros a padded or nearly dense
// block is full of.  An infinite or NaN first quotient (overflow) is returned as it is.  Only for
// a plain_divisor: a test in here, a branch on the chain of pivots, made the passes that wait for
// that chain 5 to 6 % slower, so the callers look at a block's divisors together, off the chain
// (n = 2,000 384 -> 388 us a pass, 128 x 128 x 2 nodes 4.06 -> 4.08 ms, n = 20,000 5.10 -> 5.08),
// and divide where there is another.
__device__ __forceinline__ double quotient(double x, double d, double r) {
  const double q = x * r;
  const double e = fma(fma(-q, d, x), r, q);
  return finite_bits(q) ? e : q;
}

// Whether 1 / d can stand for d: not where d is subnormal (1 / d overflows below 2^-1024) or
// infinite.  For a zero or a NaN it makes no difference.
__device__ __forceinline__ bool plain_divisor(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), e = hi & 0x7ff00000u;
  const bool fraction = ((hi & 0xfffffu) | (unsigned)__double2loint(d)) != 0u;
  return e == 0u ? !fraction : (e != 0x7ff00000u || fraction);
}

}  // namespace glu
