// quotient.cuh -- correctly rounded quotients from a reciprocal, on the device and on
// the host.
#pragma once
#ifdef __CUDACC__
#define AIFMM_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define AIFMM_HD inline
#endif

// one rounding each
AIFMM_HD double mul_rn(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
AIFMM_HD double fma_rn(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}

// a / b correctly rounded, y = 1 / b correctly rounded: P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34
// (1990), Theorem: from a q within one unit in the last place, q + (a - b q) y rounds
// to a / b.  The first correction brings a y there, the second rounds.  a, b, the
// quotient and the remainders stay away from the ends of the exponent range
// (kQuotLo, kQuotHi below).
AIFMM_HD double quotient(double a, double b, double y) {
  double q = mul_rn(a, y);
  q = fma_rn(fma_rn(-b, q, a), y, q);
  return fma_rn(fma_rn(-b, q, a), y, q);
}
constexpr double kQuotLo = 1e-20, kQuotHi = 1e20;  // R; the recurrences' values lie in 1e-270 .. 1e230
