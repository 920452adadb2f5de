// fe_node.cuh -- the right-hand side of Subproblem 2 at a node of the uniform
// mesh (Subpb2.m:88-149), for the kernels that form it (k_grid.cu) and the small
// solves that form it for themselves (fdm.cu).
#pragma once
#include <cuda_runtime.h>

namespace aldic {

// Its two parts: what beta multiplies, the shape function's gradient times
// F - udual, and what mu multiplies, the shape function times U - vdual; for u, v.
struct FeParts {
  double ku, kv, mu, mv;
};

// The 3 x 3 Gauss rule there is exact for these integrands, so their values are
// used: a node's gradient integrates to +-h/2 over each of its elements, the
// shape functions' products to the 1-D masses 1, 4, 1 (times h/6) of either
// direction, with half the diagonal at a border.
__device__ __forceinline__ FeParts fe_rhs_node(int M, int N, double h, int i, int j,
                                               const double *__restrict__ U, const double *__restrict__ F,
                                               const double *__restrict__ ud, const double *__restrict__ vd) {
  const long long k = (long long)j * M + i;
  const int l = i > 0, r = i < M - 1, d = j > 0, u = j < N - 1;
  double nu = 0.0, nv = 0.0;
#pragma unroll
  for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
    for (int di = -1; di <= 1; ++di) {
      const int w = (di < 0 ? l : di > 0 ? r : 2 * (l + r)) * (dj < 0 ? d : dj > 0 ? u : 2 * (d + u));
      if (!w) continue;
      const long long q = k + di + (long long)dj * M;
      nu += w * (U[2 * q] - vd[2 * q]);
      nv += w * (U[2 * q + 1] - vd[2 * q + 1]);
    }
  // F - W, slots [F11 F21 F12 F22]
  const double gx = 0.5 * h * ((l - r) * (d + u)), gy = 0.5 * h * ((d - u) * (l + r)), mh = h * h / 36.0;
  FeParts p;
  p.ku = gx * (F[4 * k] - ud[4 * k]) + gy * (F[4 * k + 2] - ud[4 * k + 2]);
  p.kv = gx * (F[4 * k + 1] - ud[4 * k + 1]) + gy * (F[4 * k + 3] - ud[4 * k + 3]);
  p.mu = mh * nu;
  p.mv = mh * nv;
  return p;
}

}  // namespace aldic
