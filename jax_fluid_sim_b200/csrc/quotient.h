// Quotients with a common divisor.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define DGB_HD __host__ __device__ __forceinline__
#else
#define DGB_HD inline
#endif

namespace dgb {

DGB_HD double product(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}

// a / b, given inv = 1 / b to a rounding or two: q = a inv is off by a few units in the last place, its residual a - q b
// is formed in a fused product, and q + residual inv rounds as the quotient does (Markstein, Computation of elementary
// functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).  Three products in place of a
// division.  refine = false: q alone, for operands whose residual is not finite.
DGB_HD double quotient(double a, double b, double inv, bool refine = true) {
  const double q = product(a, inv);
  return refine ? fma(fma(-q, b, a), inv, q) : q;
}

// Whether quotient(a, b, inv) has a finite residual: not where an operand or the quotient is infinite or no number.
DGB_HD bool refinable(double a, double b, double inv) {
  const double r = fma(-product(a, inv), b, a);
#ifdef __CUDA_ARCH__
  return (__double2hiint(r) & 0x7ff00000) != 0x7ff00000;
#else
  uint64_t bits;
  memcpy(&bits, &r, sizeof(bits));
  return (bits >> 52 & 0x7ff) != 0x7ff;
#endif
}

}  // namespace dgb
