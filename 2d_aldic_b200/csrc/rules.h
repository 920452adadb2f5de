// rules.h -- decisions of the library that need no GPU, apart from it so that they
// can be checked without one.
#pragma once
#ifdef __CUDACC__
#define ALDIC_RULE __host__ __device__ __forceinline__
#else
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

}  // namespace aldic
