// rules.h -- decisions of the library that need no GPU, apart from it so that they
// can be checked without one.
#pragma once
#ifdef __CUDACC__
#define ALDIC_RULE __host__ __device__ __forceinline__
#else
#include <cmath>
#define ALDIC_RULE inline
#endif

namespace aldic {

// Whether kernels on GPU `device` may use a caller's memory where it lies: memory of
// that GPU (type 2, cudaMemoryTypeDevice, and where) and managed memory (3).  Another
// GPU's memory is copied: without peer access a kernel's access to it ends the context.
ALDIC_RULE bool memory_in_place(int type, int where, int device) {
  return type == 3 || (type == 2 && where == device);
}

// Sample variance of `count` >= 2 whole numbers from their sum and sum of squares.
// The difference is exact; its products pass 2^63 for some ten million subsets.
ALDIC_RULE double sample_variance(long long count, long long sum, long long squares) {
  return (double)((__int128)count * squares - (__int128)sum * sum) / (double)count / (double)(count - 1);
}

ALDIC_RULE double fused(double a, double b, double c) {  // a b + c, rounded once
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return fma(a, b, c);
#endif
}

// n / s within one unit in the last place, from y, the correctly rounded 1 / s.  Their
// product alone is within 1.5 units of it (the reciprocal's error and its own
// rounding: 1.4996 seen); its remainder's share makes it faithful.
ALDIC_RULE double faithful_quotient(double n, double s, double y) {
  const double q = n * y;
  return fused(fused(-q, s, n), y, q);
}
// n / s correctly rounded: with y the correctly rounded reciprocal and q a quotient
// within one unit in the last place, the remainder n - q s is exact and q + (n - q s) y
// rounds to n / s (P. W. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990; a divisor whose significand
// is all ones excepted).  No step may under- or overflow.
ALDIC_RULE double rounded_quotient(double n, double s, double y) {
  const double q = faithful_quotient(n, s, y);
  return fused(fused(-q, s, n), y, q);
}

}  // namespace aldic
