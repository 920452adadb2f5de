// k_image.cu -- image preparation (a1 normalisation, a2 gradients) and the
// standalone bicubic sampler (a3, ba_interp2).
//
// Normalisation follows funNormalizeImg.m:22-39; for integer images the ROI
// sums are exact (integer atomics), so mean/std match the CPU restatement bit
// for bit.  Gradients follow funImgGradient.m:53-78 with the symmetric taps
// paired; the FP64 arithmetic is written with explicit round-to-nearest
// intrinsics so no FMA contraction changes the result.
#include "aldic_internal.cuh"
#include "kernels.cuh"
#include "rules.h"

namespace aldic {

// ------------------------------------------------------------------ ROI stats
// Exact sums of the pixels and their squares, a warp a row: whole 16-byte words
// between the row's ragged ends, one atomic a block.  4096 x 4096, 16 bit: 10 us
// (a division a pixel and two atomics a warp took 122).
template <typename T>
__global__ void __launch_bounds__(256)
    k_roi_sums_int(const T *__restrict__ img, int W, int x0, int x1, int y0, int y1,
                   unsigned long long *__restrict__ sums) {
  constexpr int kVec = 16 / sizeof(T);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long s1 = 0, s2 = 0;
  for (int y = y0 + blockIdx.x * 8 + warp; y <= y1; y += gridDim.x * 8) {
    const T *p = img + (long long)(y - 1) * W + (x0 - 1), *end = p + (x1 - x0 + 1);
    const T *v0 = (const T *)(((uintptr_t)p + 15) & ~(uintptr_t)15);
    const T *v1 = (const T *)((uintptr_t)end & ~(uintptr_t)15);
    if (v0 > v1) v0 = v1 = end;  // no whole word
    for (const T *q = p + lane; q < v0 && q < end; q += 32) {
      s1 += *q;
      s2 += (unsigned long long)*q * *q;
    }
    for (const T *q = v1 + lane; q < end; q += 32) {
      s1 += *q;
      s2 += (unsigned long long)*q * *q;
    }
    for (const T *q = v0 + lane * kVec; q < v1; q += 32 * kVec) {
      const uint4 u = *(const uint4 *)q;
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
      uint32_t a = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (sizeof(T) == 1) {
          a = __dp4a(w[e], 0x01010101u, a);
          s2 += __dp4a(w[e], w[e], 0u);
        } else {
          const uint32_t lo = w[e] & 0xffffu, hi = w[e] >> 16;
          a += lo + hi;
          s2 += (unsigned long long)lo * lo;
          s2 += (unsigned long long)hi * hi;
        }
      }
      s1 += a;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  __shared__ unsigned long long sh[2][8];
  if (lane == 0) {
    sh[0][warp] = s1;
    sh[1][warp] = s2;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned long long t = 0;
    for (int w = 0; w < 8; ++w) t += sh[threadIdx.x][w];
    if (t) atomicAdd(&sums[threadIdx.x], t);
  }
}

// deterministic per-block partials of sum(v - m)^p, p in {1,2}
template <typename T>
__global__ void k_roi_partials(const T *__restrict__ img, int W, int x0, int x1, int y0,
                               int y1, const double *__restrict__ mean, int pw,
                               double *__restrict__ part) {
  const int rw = x1 - x0 + 1;
  const long long n = (long long)rw * (y1 - y0 + 1);
  const double m = pw == 2 ? *mean : 0.0;
  double s = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int y = y0 + (int)(i / rw), x = x0 + (int)(i % rw);
    const double v = (double)img[(long long)(y - 1) * W + (x - 1)] - m;
    s += pw == 2 ? v * v : v;
  }
  s = warp_sum(s);
  __shared__ double sh[32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sh[k];
    part[blockIdx.x] = t;
  }
}

__global__ void k_stats_int_final(const unsigned long long *sums, long long n, double *out) {
  const double m = (double)sums[0] / (double)n;
  const double ssd = __dsub_rn((double)sums[1], __dmul_rn(m, (double)sums[0]));
  out[0] = m;
  out[1] = sqrt(ssd / (double)(n - 1));
}

__global__ void k_sum_partials(const double *part, int np, long long n, int pw, double *out) {
  double t = 0;
  for (int k = 0; k < np; ++k) t += part[k];
  if (pw == 1) out[0] = t / (double)n;
  else out[1] = sqrt(t / (double)(n - 1));
}

int roi_stats(const void *img, int dtype, int W, const int roi[4], double *d_stats,
              unsigned long long *d_isums, double *d_part, cudaStream_t st) {
  const long long n = (long long)(roi[1] - roi[0] + 1) * (roi[3] - roi[2] + 1);
  const int blocks = 296, threads = 256, iblocks = 592;
  if (dtype == 0 || dtype == 1) {
    ALDIC_CUDA(cudaMemsetAsync(d_isums, 0, 2 * sizeof(unsigned long long), st));
    if (dtype == 0)
      k_roi_sums_int<uint8_t><<<iblocks, threads, 0, st>>>((const uint8_t *)img, W, roi[0],
                                                          roi[1], roi[2], roi[3], d_isums);
    else
      k_roi_sums_int<uint16_t><<<iblocks, threads, 0, st>>>((const uint16_t *)img, W, roi[0],
                                                           roi[1], roi[2], roi[3], d_isums);
    k_stats_int_final<<<1, 1, 0, st>>>(d_isums, n, d_stats);
  } else {
    for (int pw = 1; pw <= 2; ++pw) {
      if (dtype == 2)
        k_roi_partials<float><<<blocks, threads, 0, st>>>((const float *)img, W, roi[0], roi[1],
                                                          roi[2], roi[3], d_stats, pw, d_part);
      else
        k_roi_partials<double><<<blocks, threads, 0, st>>>((const double *)img, W, roi[0],
                                                           roi[1], roi[2], roi[3], d_stats, pw,
                                                           d_part);
      k_sum_partials<<<1, 1, 0, st>>>(d_part, blocks, n, pw, d_stats);
    }
  }
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

// ------------------------------------------------------------------ normalise
// (v - m) / s correctly rounded, s the same for every pixel: rounded_quotient's five
// operations in place of a division's thirty.  Deviations out of the range where no
// step under- or overflows, 0 or NaN among them, are divided by.
struct Norm {
  double m, s, y;
  bool by_product;
  __device__ __forceinline__ explicit Norm(const double *stats) : m(stats[0]), s(stats[1]) {
    y = __ddiv_rn(1.0, s);
    by_product = s > 1e-100 && s < 1e100 && (__double_as_longlong(s) & 0xfffffffffffffll) != 0xfffffffffffffll;
  }
  __device__ __forceinline__ double operator()(double v) const {
    const double n = __dsub_rn(v, m);
    if (!by_product || !(fabs(n) > 1e-100 && fabs(n) < 1e100)) return __ddiv_rn(n, s);
    return rounded_quotient(n, s, y);
  }
};

template <typename T>
__global__ void k_normalize(const T *__restrict__ img, long long n,
                            const double *__restrict__ stats, double *__restrict__ o64,
                            float *__restrict__ o32) {
  const Norm norm(stats);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double v = norm((double)img[i]);
    o64[i] = v;
    o32[i] = __double2float_rn(v);
  }
}

int normalize(const void *img, int dtype, long long n, const double *d_stats, double *o64,
              float *o32, cudaStream_t st) {
  const int blocks = 1184, threads = 256;
  switch (dtype) {
    case 0: k_normalize<uint8_t><<<blocks, threads, 0, st>>>((const uint8_t *)img, n, d_stats, o64, o32); break;
    case 1: k_normalize<uint16_t><<<blocks, threads, 0, st>>>((const uint16_t *)img, n, d_stats, o64, o32); break;
    case 2: k_normalize<float><<<blocks, threads, 0, st>>>((const float *)img, n, d_stats, o64, o32); break;
    default: k_normalize<double><<<blocks, threads, 0, st>>>((const double *)img, n, d_stats, o64, o32); break;
  }
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

// ---------------------------------------------------- row-cubic coefficients
// The Keys cubic (a = -1/2) of ba_interp2.cpp along one row as a polynomial:
// with taps g_k (k = 0..3 at offsets -1..2 from the floor column) and
// fraction t, sum_k w_k(t) g_k = a0 + a1 t + a2 t^2 + a3 t^3, where row p of
// the 4 x 4 matrix behind keys_rows holds the t^p coefficients of the four
// Keys weights.  q[y W + x] = (a0, a1, a2, a3) of row y with floor column x,
// from the FP64 image and rounded once to FP32 (zeros where the stencil
// leaves the row: the IC-GN out-of-image test keeps every sampled floor
// column in [2, W-3]).  A bicubic sample is then four Horner rules over tu
// on consecutive rows and one cubic over tv -- and consecutive rows of a
// subset column share three of their four stencil rows.
__device__ __forceinline__ void keys_rows(const double g[4], double a[4]) {
  a[0] = g[1];
  a[1] = 0.5 * (g[2] - g[0]);
  a[2] = g[0] - 2.5 * g[1] + 2.0 * g[2] - 0.5 * g[3];
  a[3] = 0.5 * (g[3] - g[0]) + 1.5 * (g[1] - g[2]);
}

__global__ void k_row_cubic(const double *__restrict__ g, int W, long long n,
                            float4 *__restrict__ q) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % W);
    if (x < 1 || x > W - 3) {
      q[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      continue;
    }
    const double t[4] = {__ldg(g + i - 1), __ldg(g + i), __ldg(g + i + 1), __ldg(g + i + 2)};
    double a[4];
    keys_rows(t, a);
    q[i] = make_float4((float)a[0], (float)a[1], (float)a[2], (float)a[3]);
  }
}

int row_cubic(const double *g, int W, int H, float4 *q, cudaStream_t st) {
  k_row_cubic<<<1184, 256, 0, st>>>(g, W, (long long)W * H, q);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

// q[i] = (gx[i], gy[i]): the two FP32 gradients of a pixel in one 8-byte load
__global__ void k_pair(const float *__restrict__ gx, const float *__restrict__ gy, long long n,
                       float2 *__restrict__ q) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    q[i] = make_float2(gx[i], gy[i]);
}

int grad_pairs(const float *gx, const float *gy, long long n, float2 *q, cudaStream_t st) {
  k_pair<<<1184, 256, 0, st>>>(gx, gy, n, q);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}


// Both at once: the normalised image and its row cubics, a row in segments of 256
// columns, whose normalised values and the three beside them lie in shared memory.
// Bound by memory: 4096 x 4096, 16 bit, writes 28 bytes a pixel; 104 us (the
// copy rate allows 77), 146 us as two kernels that wrote the image and read it back.
template <typename T>
__global__ void __launch_bounds__(256)
    k_normalize_cubic(const T *__restrict__ img, int W, int H, const double *__restrict__ stats,
                      double *__restrict__ o64, float *__restrict__ o32, float4 *__restrict__ q) {
  const Norm norm(stats);
  __shared__ double row[2][256 + 3];
  const int segs = (W + 255) / 256, t = threadIdx.x;
  int at = 0;
  for (long long b = blockIdx.x; b < (long long)segs * H; b += gridDim.x, at ^= 1) {
    const int y = (int)(b / segs), x0 = (int)(b - (long long)y * segs) * 256, x = x0 + t;
    const T *p = img + (long long)y * W;
    const long long i = (long long)y * W + x;
    double *r = row[at];
    double v = 0.0;
    if (x < W) {
      v = norm((double)p[x]);
      o64[i] = v;
      o32[i] = __double2float_rn(v);
    }
    r[t + 1] = v;
    if (t < 3) {  // column x0 - 1 and the two after the segment
      const int xe = t == 0 ? x0 - 1 : x0 + 255 + t;
      r[t == 0 ? 0 : 256 + t] = xe >= 0 && xe < W ? norm((double)p[xe]) : 0.0;
    }
    __syncthreads();  // the other buffer is read no more
    if (x < W) {
      if (x < 1 || x > W - 3) {
        q[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        const double g[4] = {r[t], r[t + 1], r[t + 2], r[t + 3]};
        double a[4];
        keys_rows(g, a);
        q[i] = make_float4((float)a[0], (float)a[1], (float)a[2], (float)a[3]);
      }
    }
  }
}

int normalize_cubic(const void *img, int dtype, int W, int H, const double *d_stats, double *o64, float *o32,
                    float4 *q, cudaStream_t st) {
  const int blocks = 148 * 8;
  switch (dtype) {
    case 0: k_normalize_cubic<uint8_t><<<blocks, 256, 0, st>>>((const uint8_t *)img, W, H, d_stats, o64, o32, q); break;
    case 1: k_normalize_cubic<uint16_t><<<blocks, 256, 0, st>>>((const uint16_t *)img, W, H, d_stats, o64, o32, q); break;
    case 2: k_normalize_cubic<float><<<blocks, 256, 0, st>>>((const float *)img, W, H, d_stats, o64, o32, q); break;
    default: k_normalize_cubic<double><<<blocks, 256, 0, st>>>((const double *)img, W, H, d_stats, o64, o32, q); break;
  }
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

// ------------------------------------------------------------------ gradient
__device__ __forceinline__ double grad7(const double *f, long long i, long long s) {
  const double c1 = 0.75, c2 = 3.0 / 20.0, c3 = 1.0 / 60.0;
  const double a = __dmul_rn(c1, __dsub_rn(f[i + s], f[i - s]));
  const double b = __dmul_rn(c2, __dsub_rn(f[i + 2 * s], f[i - 2 * s]));
  const double c = __dmul_rn(c3, __dsub_rn(f[i + 3 * s], f[i - 3 * s]));
  return __dadd_rn(__dsub_rn(a, b), c);
}

__global__ void k_gradient(const double *__restrict__ f, const double *__restrict__ mask, int W,
                           int H, double *__restrict__ gx64, double *__restrict__ gy64,
                           float *__restrict__ gx32, float *__restrict__ gy32) {
  const long long n = (long long)W * H;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(i / W), x = (int)(i % W);
    double tx = 0.0, ty = 0.0;
    if (x >= 3 && x < W - 3 && y >= 3 && y < H - 3) {
      const double m = mask ? mask[i] : 1.0;
      tx = __dmul_rn(grad7(f, i, 1), m);
      ty = __dmul_rn(grad7(f, i, W), m);
    }
    gx64[i] = tx;
    gy64[i] = ty;
    gx32[i] = __double2float_rn(tx);
    gy32[i] = __double2float_rn(ty);
  }
}

int gradient(const double *f, const double *mask, int W, int H, double *gx64, double *gy64,
             float *gx32, float *gy32, cudaStream_t st) {
  k_gradient<<<1184, 256, 0, st>>>(f, mask, W, H, gx64, gy64, gx32, gy32);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

// ------------------------------------------------------------------ ba_interp2
// ba_interp2.cpp:133-182 restated with explicit rounding so both precisions
// reproduce the reference's compiled results bit for bit.
__device__ __forceinline__ long long corner_index(double cf, long long extent) {
  const double lo = -4.0, hi = (double)extent + 4.0;
  const double c = cf < lo ? lo : (cf > hi ? hi : cf);
  return (long long)(c - 1.0);
}
__device__ __forceinline__ long long clampll(long long v, long long lo, long long hi) {
  return v < lo ? lo : (v > hi ? hi : v);
}

__device__ __forceinline__ void weights_f64(double d, double w[4]) {
  const double d2 = __dmul_rn(d, d), d3 = __dmul_rn(d2, d);
  w[0] = __dmul_rn(0.5, __dsub_rn(__dadd_rn(-d, __dmul_rn(2.0, d2)), d3));
  w[1] = __dmul_rn(0.5, __dadd_rn(__dsub_rn(2.0, __dmul_rn(5.0, d2)), __dmul_rn(3.0, d3)));
  w[2] = __dmul_rn(0.5, __dsub_rn(__dadd_rn(d, __dmul_rn(4.0, d2)), __dmul_rn(3.0, d3)));
  w[3] = __dmul_rn(0.5, __dadd_rn(-d2, d3));
}

// float inputs: the weight polynomials run in double from float powers
__device__ __forceinline__ void weights_f32(float d, float w[4]) {
  const float d2 = __fmul_rn(d, d), d3 = __fmul_rn(d2, d);
  const double D = d, D2 = d2, D3 = d3;
  w[0] = __double2float_rn(__dmul_rn(0.5, __dsub_rn(__dadd_rn((double)(-d), __dmul_rn(2.0, D2)), D3)));
  w[1] = __double2float_rn(__dmul_rn(0.5, __dadd_rn(__dsub_rn(2.0, __dmul_rn(5.0, D2)), __dmul_rn(3.0, D3))));
  w[2] = __double2float_rn(__dmul_rn(0.5, __dsub_rn(__dadd_rn(D, __dmul_rn(4.0, D2)), __dmul_rn(3.0, D3))));
  w[3] = __double2float_rn(__dmul_rn(0.5, (double)__fadd_rn(-d2, d3)));
}

__device__ __forceinline__ void weights(double d, double w[4]) { weights_f64(d, w); }
__device__ __forceinline__ void weights(float d, float w[4]) { weights_f32(d, w); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }

__device__ __forceinline__ double quiet_nan(double) { return __longlong_as_double(0x7ff8000000000000ll); }
__device__ __forceinline__ float quiet_nan(float) { return __int_as_float(0x7fc00000); }

// one point: 4 x 4 taps, columns c[k] apart, rows r[k]
template <typename T, typename I>
__device__ __forceinline__ T interp_sum(const T *__restrict__ F, const I c[4], const I r[4], const T wx[4],
                                        const T wy[4]) {
  T acc = 0;
#pragma unroll
  for (int rr = 0; rr < 4; ++rr) {
    T s = mul(wx[0], F[c[0] + r[rr]]);
    s = add(s, mul(wx[1], F[c[1] + r[rr]]));
    s = add(s, mul(wx[2], F[c[2] + r[rr]]));
    s = add(s, mul(wx[3], F[c[3] + r[rr]]));
    acc = rr == 0 ? mul(wy[0], s) : add(acc, mul(wy[rr], s));
  }
  return acc;
}

// A thread a point.  A point whose taps all lie inside the image (and a plane
// below 2^31 elements) takes 32-bit indices from one conversion a coordinate;
// the others the clamped 64-bit ones of the reference.  The next point's
// coordinates are on their way during the taps of this one.
// What bounds it: 16 gathers a point through L1 and, in FP64, 63 operations
// without fused multiply-adds (the reference's rounding).  2048 x 2048 FP64,
// as many points: 48 us (134 MB, 21 us at the copy rate); 81 us with 64-bit
// indices and a floor in FP64 at every point.  Registers decide: 24 warps an SM
// hold a point's 16 taps in flight; 28 or 32 warps spill and take 59 to 63 us.
template <typename T>
__global__ void __launch_bounds__(128, 6)
    k_interp(const T *__restrict__ F, long long M, long long N, long long P, const T *__restrict__ X,
             const T *__restrict__ Y, long long n, T *__restrict__ Z) {
  const long long LO = M * N, step = (long long)gridDim.x * blockDim.x;
  const bool narrow = LO < (1ll << 31);
  // x < xe: floor(x) <= N - 2, also where N - 1 is no number of the type
  const T xe = (T)(narrow ? N - 1 : 0), ye = (T)(narrow ? M - 1 : 0);
  const int m = (int)M;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  T xn = 0, yn = 0;
  if (i < n) {
    xn = X[i];
    yn = Y[i];
  }
  for (; i < n; i += step) {
    const T x = xn, y = yn;
    if (i + step < n) {
      xn = X[i + step];
      yn = Y[i + step];
    }
    T wx[4], wy[4];
    if (x >= (T)2 && x < xe && y >= (T)2 && y < ye) {
      const int xi = (int)x, yi = (int)y;
      weights(x - (T)xi, wx);
      weights(y - (T)yi, wy);
      const int o = (xi - 2) * m + (yi - 2);
      const int c[4] = {o, o + m, o + 2 * m, o + 3 * m}, r[4] = {0, 1, 2, 3};
      for (long long j = 0; j < P; ++j) Z[i + j * n] = interp_sum(F + j * LO, c, r, wx, wy);
      continue;
    }
    if (!isfinite(x) || !isfinite(y)) {
      for (long long j = 0; j < P; ++j) Z[i + j * n] = quiet_nan(T());
      continue;
    }
    const T xf = floor(x), yf = floor(y);
    weights(add(x, -xf), wx);
    weights(add(y, -yf), wy);
    const long long xc = corner_index((double)xf, N), yc = corner_index((double)yf, M);
    long long c[4], r[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      c[k] = clampll(xc - 1 + k, 0, N - 1) * M;
      r[k] = clampll(yc - 1 + k, 0, M - 1);
    }
#pragma unroll 1
    for (long long j = 0; j < P; ++j) Z[i + j * n] = interp_sum(F + j * LO, c, r, wx, wy);
  }
}

int interp_f64(const double *F, long long M, long long N, long long P, const double *X,
               const double *Y, long long n, double *Z, cudaStream_t st) {
  if (n <= 0) return OK;
  long long blocks = (n + 127) / 128;
  if (blocks > 148 * 30) blocks = 148 * 30;
  k_interp<double><<<(int)blocks, 128, 0, st>>>(F, M, N, P, X, Y, n, Z);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

int interp_f32(const float *F, long long M, long long N, long long P, const float *X,
               const float *Y, long long n, float *Z, cudaStream_t st) {
  if (n <= 0) return OK;
  long long blocks = (n + 127) / 128;
  if (blocks > 148 * 30) blocks = 148 * 30;
  k_interp<float><<<(int)blocks, 128, 0, st>>>(F, M, N, P, X, Y, n, Z);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

}  // namespace aldic
