// search.cuh -- the geometry of the whole-field integer search, shared by its
// kernels (k_search.cu, k_search_mma.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace aldic {

constexpr size_t kSmemMax = 227 * 1024;

struct SearchGeom {
  int W, H;
  int gx1, gy1, nx, ny, step;
  int w, sx, sy;
  int tw, twp, dw, dh, cr, cc, nsx, dpw, dph;
  const double *mu;  // device pointer: ROI mean of the deformed image
};

__device__ __forceinline__ unsigned fkey(float x) {  // order-preserving float -> unsigned
  const unsigned u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// the tensor-core search of 8- (bytes 1) and 16-bit images: whether a geometry
// fits it, and the search itself, over all grid points or those of list
// {count, points...} (device memory).  tab: the window table of box_table.  f
// and g are 4-byte aligned and may be read up to 16 bytes beyond the image.  *err
// becomes 3 where a wait gave up (after `tries` polls); the points of that CTA that
// were not done have NaN then.
bool search_mma_fits(const SearchGeom &G, int bytes);
template <typename T>
int search_mma(const T *f, const T *g, const SearchGeom &G, const uint4 *tab, const int *list, double *x,
               double *y, double *u, double *v, double *cc, int *err, unsigned tries, cudaStream_t st);

// tab[y W + x]: sums of g and g^2 over the tw x tw window with its first pixel
// at (x, y) (0-based) and 1/sqrt(tw^2 sum g^2 - (sum g)^2), for every window of
// the geometry's search regions: {sum, sum of squares, 1/sqrt, 0} of 8-bit
// images, {sum, sum of squares low word, high word, 1/sqrt} of 16-bit ones
template <typename T>
int box_table(const T *g, const SearchGeom &G, uint4 *tab, cudaStream_t st);

}  // namespace aldic
