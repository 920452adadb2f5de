// k_searchmg.cu -- multigrid integer search (func/funIntegerSearchMg.m), the
// search IntegerSearch.m:117-120 runs when InitFFTSearchMethod is neither 1
// nor 2: one global shift from the whole ROI, then regions split level by
// level down to the subset size, each refined within +-5 px of its parent's
// shift, and the last level's displacements fitted onto the node grid.
//
// Device side:
//   * summed-area tables of f, f^2, g, g^2 (exact 64-bit for integer images)
//     give every window sum of the normalised cross-correlation in O(1);
//   * level 1: normxcorr2 of the whole f ROI against the g ROI for every
//     shift by an FP64 FFT cross-correlation (own kernels: radix 8 in
//     registers, tiled transposes; the two real inputs packed into one
//     complex row, two real output rows into one; the NCC map is formed and
//     searched by the last transform), then findpeak's 3x3 fit;
//   * intermediate levels: the 13 x 14 cropped map of every region from
//     exact integer products -- CTAs over (region, row band, 256-column
//     tile), each thread a register window over 13 horizontal shifts, packed
//     byte products for integer images;
//   * last level: the full (2a+9) x (2b+9) map of every region in shared
//     memory (for compute_qFactor), with register-blocked strips of 8 shifts.
// Host side: the region bookkeeping of funIntegerSearchMg.m (splits, border
// clamps, even widths, NaN propagation) and the gridfit 'springs' normal
// equations of the scattered last-level data, solved by the CSR PCG.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <type_traits>
#include <vector>

#include "aldic_internal.cuh"
#include "kernels.cuh"
#include "ncc.cuh"

namespace aldic {

namespace {

constexpr int kCropR = 13, kCropC = 14, kCrop = kCropR * kCropC;  // 13 x 14 crop
constexpr int kBand = 8, kSegs = 16;                               // intermediate levels
constexpr int kStrip = 8;                                          // last level
constexpr int kMaxFinal = 80;  // largest last-level region side (about winsize + 1)
constexpr int kMaxFFT = 8192;  // largest FFT length (ROI up to 4096 px per side)

// S: window sums; V: a pixel in shared memory (of floats, and their sums of
// products); G: a sum of products in memory
template <typename P> struct MgT;
template <> struct MgT<uint8_t> {
  using S = long long;
  using V = unsigned int;
  using G = unsigned long long;
  static constexpr bool integer = true;
};
template <> struct MgT<uint16_t> : MgT<uint8_t> {};
template <> struct MgT<float> {
  using S = double;
  using V = double;
  using G = double;
  static constexpr bool integer = false;
};
template <> struct MgT<double> : MgT<float> {};

struct MgReg {
  int tx, ty, a, b;  // template f(tx : tx+a-1, ty : ty+b-1), 1-based
  int dx, dy;        // region g(dx : dx+a+9, dy : dy+b+9), 1-based
  int valid;
  int pad;
};

// rectangle sum of a (W+1) x (H+1) summed-area table over 0-based pixels
// [x0, x1) x [y0, y1)
template <typename S>
__device__ __forceinline__ S rect_sum(const S *__restrict__ sat, int W1, int x0, int x1, int y0,
                                      int y1) {
  return sat[(long long)y1 * W1 + x1] - sat[(long long)y0 * W1 + x1] -
         sat[(long long)y1 * W1 + x0] + sat[(long long)y0 * W1 + x0];
}

template <typename S>
__device__ __forceinline__ double combine(long long mn, S st, S st2, S stdv, S sd, S sd2, S st_pad,
                                          long long n_pad, double mu) {
  if constexpr (std::is_integral<S>::value) {
    return ncc_combine_wide(mn, (long long)st, (long long)st2, (long long)stdv, (long long)sd,
                            (long long)sd2, (long long)st_pad, n_pad, mu);
  } else {
    return ncc_combine_f((double)mn, (double)st, (double)st2, (double)stdv, (double)sd,
                         (double)sd2, (double)st_pad, (double)n_pad, mu);
  }
}

// ------------------------------------------------------------ summed-area tables
// sat[0..3] = f, f^2, g, g^2, each (W+1) x (H+1), row 0 and column 0 zero.
// Bound by the writes of the tables (32 bytes a pixel, 134 MB at 2048 x 2048):
// they are written once.  (Rows, then columns in place in two passes moved them
// five times, 208 us; this takes 77 us.)
// Pass 1: sums of each column over chunks of kSatChunk rows, read from the images.
constexpr int kSatChunk = 16;
template <typename P>
__global__ void k_sat_chunks(const P *__restrict__ f, const P *__restrict__ g, int W, int H,
                             typename MgT<P>::S *__restrict__ tot) {
  using S = typename MgT<P>::S;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, ch = blockIdx.y, nch = gridDim.y;
  if (x >= W) return;
  const int y0 = ch * kSatChunk, y1 = min(H, y0 + kSatChunk);
  S a[4] = {0, 0, 0, 0};
  for (int y = y0; y < y1; ++y) {
    const S u = (S)f[(long long)y * W + x], v = (S)g[(long long)y * W + x];
    a[0] += u;
    a[1] += u * u;
    a[2] += v;
    a[3] += v * v;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) tot[((long long)q * nch + ch) * W + x] = a[q];
}
// Pass 2: each chunk's entry becomes the column's sum above the chunk.
template <typename S>
__global__ void k_sat_above(S *__restrict__ tot, int W, int nch) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= W) return;
  S *p = tot + (long long)blockIdx.y * nch * W + x;
  S acc = 0;
  for (int c0 = 0; c0 < nch; c0 += 32) {
    S v[32];  // all on their way at once
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = c0 + e < nch ? p[(long long)(c0 + e) * W] : S(0);
#pragma unroll
    for (int e = 0; e < 32; ++e)
      if (c0 + e < nch) {
        p[(long long)(c0 + e) * W] = acc;
        acc += v[e];
      }
  }
}
// Pass 3: the rows of a chunk: running column sums in registers, scanned along x
// a warp a kSatSpan columns, the warps' totals and those of the columns to the
// left through shared memory.
constexpr int kSatThreads = 256, kSatItems = 8, kSatSpan = 32 * kSatItems;
template <typename P>
__global__ void __launch_bounds__(kSatThreads)
    k_sat_fill(const P *__restrict__ f, const P *__restrict__ g, int W, int H,
               const typename MgT<P>::S *__restrict__ tot, typename MgT<P>::S *__restrict__ sat) {
  using S = typename MgT<P>::S;
  constexpr int kWarps = kSatThreads / 32;
  __shared__ S warp_tot[2][kWarps], left[kSatChunk];
  const int q = blockIdx.y, ch = blockIdx.x, nch = gridDim.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const P *img = q < 2 ? f : g;
  const bool sq = q & 1;
  const long long W1 = W + 1;
  S *out = sat + q * W1 * (H + 1);
  const int y0 = ch * kSatChunk, rows = min(H - y0, kSatChunk);
  if (ch == 0)
    for (int x = threadIdx.x; x <= W; x += kSatThreads) out[x] = 0;
  if (threadIdx.x < rows) {
    left[threadIdx.x] = 0;
    out[(y0 + 1 + threadIdx.x) * W1] = 0;
  }
  for (int x0 = 0; x0 < W; x0 += kWarps * kSatSpan) {
    S col[kSatItems];
    const int xw = x0 + warp * kSatSpan + lane;
#pragma unroll
    for (int e = 0; e < kSatItems; ++e) {
      const int x = xw + 32 * e;
      col[e] = x < W ? tot[((long long)q * nch + ch) * W + x] : S(0);
    }
    P next[kSatItems];  // the row to come, on its way during this one's scan
    auto fetch = [&](int r) {
#pragma unroll
      for (int e = 0; e < kSatItems; ++e) {
        const int x = xw + 32 * e;
        next[e] = r < rows && x < W ? img[(long long)(y0 + r) * W + x] : P(0);
      }
    };
    fetch(0);
    __syncthreads();  // left is set
    for (int r = 0; r < rows; ++r) {
      S v[kSatItems], run = 0;
      S px[kSatItems];
#pragma unroll
      for (int e = 0; e < kSatItems; ++e) px[e] = (S)next[e];
      fetch(r + 1);
#pragma unroll
      for (int e = 0; e < kSatItems; ++e) {
        col[e] += sq ? px[e] * px[e] : px[e];
        S t = col[e];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const S n = __shfl_up_sync(0xffffffffu, t, o);
          if (lane >= o) t += n;
        }
        v[e] = run + t;
        run += __shfl_sync(0xffffffffu, t, 31);
      }
      if (lane == 0) warp_tot[r & 1][warp] = run;
      __syncthreads();
      S before = left[r];
#pragma unroll
      for (int w = 0; w < kWarps; ++w) before += w < warp ? warp_tot[r & 1][w] : S(0);
#pragma unroll
      for (int e = 0; e < kSatItems; ++e) {
        const int x = xw + 32 * e;
        if (x < W) out[(y0 + 1 + r) * W1 + x + 1] = before + v[e];
      }
      if (x0 + kWarps * kSatSpan < W) {  // the row's sum so far, for the columns to come
        __syncthreads();
        if (threadIdx.x == kSatThreads - 1) left[r] = before + v[kSatItems - 1];
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ FFT (FP64)
// Stockham autosort transform of one row, a CTA of L / 8 threads a row: passes
// of radix 8 (a radix-2 or radix-4 pass first when log2 L is not a multiple of
// 3), every thread eight values in registers: read L/R apart, twiddled, an
// R-point DFT, handed on Ns apart through shared memory (entry e at e + e/8, so
// that no pass has a bank conflict) -- natural order in and out, no bit reversal.
// The first pass reads and the last writes what the caller gives, so a row is
// not staged.  Twiddles come from a table laid out as the passes read them:
// exp(-2 pi i k q / 8 Ns) at (q - 1) Ns + k of the pass.
// What bounds it at 4096: three exchanges of 128 KB a row through shared memory,
// some 3000 cycles, and as many of FP64; two CTAs an SM overlap them with the
// loads.  A pass over 4096 rows took 450 us with staged rows, 8-way conflicts
// and one CTA an SM; 123 us now (half of its rows zeros that are not read).
__global__ void k_fft_twiddle(double2 *tw, int L, int logL) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int rem = logL % 3;
  int at = t, Ns = rem == 1 ? 2 : rem == 2 ? 4 : 8;
  for (; Ns < L && at >= 7 * Ns; Ns *= 8) at -= 7 * Ns;
  if (Ns >= L) return;
  const int q = 1 + at / Ns, k = at % Ns;
  double s, c;
  sincospi(2.0 * (double)(k * q) / (8.0 * Ns), &s, &c);
  tw[t] = make_double2(c, -s);
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// times -i (forward) or +i (inverse)
__device__ __forceinline__ double2 cmi(double2 a, bool inv) {
  return inv ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

template <int R, bool inv>
__device__ __forceinline__ void dft_reg(double2 *a) {
  if constexpr (R == 2) {
    const double2 t = a[0];
    a[0] = cadd(t, a[1]);
    a[1] = csub(t, a[1]);
  } else if constexpr (R == 4) {
    const double2 c0 = cadd(a[0], a[2]), c2 = csub(a[0], a[2]);
    const double2 c1 = cadd(a[1], a[3]), c3 = cmi(csub(a[1], a[3]), inv);
    a[0] = cadd(c0, c1);
    a[2] = csub(c0, c1);
    a[1] = cadd(c2, c3);
    a[3] = csub(c2, c3);
  } else {
    constexpr double h = 0.70710678118654752440;
    // decimation in frequency: sums feed the even outputs, twiddled
    // differences the odd ones
    const double2 b0 = cadd(a[0], a[4]), b1 = cadd(a[1], a[5]), b2 = cadd(a[2], a[6]),
                  b3 = cadd(a[3], a[7]);
    const double2 d1 = csub(a[1], a[5]), d3 = csub(a[3], a[7]);
    const double2 b4 = csub(a[0], a[4]);
    const double2 b6 = cmi(csub(a[2], a[6]), inv);
    // W8 = (1 - i)/sqrt2, W8^3 = (-1 - i)/sqrt2 (conjugates for the inverse)
    const double2 b5 = inv ? make_double2(h * (d1.x - d1.y), h * (d1.x + d1.y))
                           : make_double2(h * (d1.x + d1.y), h * (d1.y - d1.x));
    const double2 b7 = inv ? make_double2(-h * (d3.x + d3.y), h * (d3.x - d3.y))
                           : make_double2(h * (d3.y - d3.x), -h * (d3.x + d3.y));
    const double2 c0 = cadd(b0, b2), c2 = csub(b0, b2), c1 = cadd(b1, b3), c3 = cmi(csub(b1, b3), inv);
    const double2 c4 = cadd(b4, b6), c6 = csub(b4, b6), c5 = cadd(b5, b7), c7 = cmi(csub(b5, b7), inv);
    a[0] = cadd(c0, c1);
    a[4] = csub(c0, c1);
    a[2] = cadd(c2, c3);
    a[6] = csub(c2, c3);
    a[1] = cadd(c4, c5);
    a[5] = csub(c4, c5);
    a[3] = cadd(c6, c7);
    a[7] = csub(c6, c7);
  }
}

__device__ __forceinline__ int fft_pos(int e) { return e + (e >> 3); }
__host__ __device__ inline int fft_threads(int L) { return L / 8 < 32 ? 32 : L / 8; }
inline size_t fft_smem(int L) { return sizeof(double2) * (size_t)(L + L / 8 + 1); }

template <int R, bool INV, bool FIRST, bool LAST, typename Load, typename Store>
__device__ __forceinline__ void stockham_pass(double2 *s, int L, int Ns, const double2 *__restrict__ tw, Load load,
                                              Store store) {
  constexpr int G = 8 / R;  // groups a thread
  const int nj = L / R;
  double2 v[G][R];
#pragma unroll
  for (int t = 0; t < G; ++t) {
    const int j = threadIdx.x + t * blockDim.x;
    if (j < nj) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[t][q] = FIRST ? load(j + q * nj) : s[fft_pos(j + q * nj)];
    }
  }
  if (!FIRST) __syncthreads();
#pragma unroll
  for (int t = 0; t < G; ++t) {
    const int j = threadIdx.x + t * blockDim.x;
    if (j < nj) {
      const int k = j & (Ns - 1);
      if (!FIRST) {
#pragma unroll
        for (int q = 1; q < R; ++q) {
          double2 w = __ldg(&tw[(q - 1) * Ns + k]);
          if (INV) w.y = -w.y;
          v[t][q] = cmul(v[t][q], w);
        }
      }
      dft_reg<R, INV>(v[t]);
      const int base = (j - k) * R + k;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        if (LAST) store(base + q * Ns, v[t][q]);
        else s[fft_pos(base + q * Ns)] = v[t][q];
      }
    }
  }
  if (!LAST) __syncthreads();
}

// a row of L = 2^logL <= 8192 entries from load(e) to store(e, value)
template <bool INV, typename Load, typename Store>
__device__ __forceinline__ void fft_row(double2 *s, int L, int logL, const double2 *__restrict__ tw, Load load,
                                        Store store) {
  const int rem = logL % 3, R0 = rem == 1 ? 2 : rem == 2 ? 4 : 8;
  if (L == R0) {
    if (rem == 1) stockham_pass<2, INV, true, true>(s, L, 1, tw, load, store);
    else if (rem == 2) stockham_pass<4, INV, true, true>(s, L, 1, tw, load, store);
    else stockham_pass<8, INV, true, true>(s, L, 1, tw, load, store);
    return;
  }
  if (rem == 1) stockham_pass<2, INV, true, false>(s, L, 1, tw, load, store);
  else if (rem == 2) stockham_pass<4, INV, true, false>(s, L, 1, tw, load, store);
  else stockham_pass<8, INV, true, false>(s, L, 1, tw, load, store);
  int Ns = R0;
  for (; Ns * 8 < L; Ns *= 8) {
    stockham_pass<8, INV, false, false>(s, L, Ns, tw, load, store);
    tw += 7 * Ns;
  }
  stockham_pass<8, INV, false, true>(s, L, Ns, tw, load, store);
}

// Level 1 packs its two real inputs into one complex row,
// z(x) = (f - mean f) + i (g - mu) over the ROI and zero beyond; rows y < b only.
template <typename P>
__global__ void __launch_bounds__(1024)
    k_fft_pack_rows(const P *__restrict__ f, const P *__restrict__ g, int W, int H, int x1, int y1, int a, int b,
                    const typename MgT<P>::S *__restrict__ sat, const double *__restrict__ mu_g,
                    double2 *__restrict__ Z, int L, int logL, const double2 *__restrict__ tw) {
  extern __shared__ double2 s[];
  const int y = blockIdx.x;
  double2 *row = Z + (long long)y * L;
  const long long W1 = W + 1, o = (long long)(y1 - 1 + y) * W + (x1 - 1);
  const double st = (double)rect_sum(sat, (int)W1, x1 - 1, x1 - 1 + a, y1 - 1, y1 - 1 + b);
  const double mean_t = st / ((double)a * (double)b);
  const double mu = *mu_g;
  fft_row<false>(
      s, L, logL, tw,
      [&](int x) { return x < a ? make_double2((double)f[o + x] - mean_t, (double)g[o + x] - mu) : make_double2(0.0, 0.0); },
      [&](int x, double2 v) { row[x] = v; });
}

// columns [kx][ky], in place; entries from `len` on are zeros that nobody wrote
__global__ void __launch_bounds__(1024)
    k_fft_cols(double2 *__restrict__ Z, int L, int logL, const double2 *__restrict__ tw, int len) {
  extern __shared__ double2 s[];
  double2 *row = Z + (long long)blockIdx.x * L;
  fft_row<false>(s, L, logL, tw, [&](int y) { return y < len ? row[y] : make_double2(0.0, 0.0); },
                 [&](int y, double2 v) { row[y] = v; });
}

// The correlation's spectrum and its inverse along y: with Z = F + i G (F, G
// transforms of the two real inputs), F(k) = (Z(k) + conj Z(-k)) / 2, G(k) =
// (Z(k) - conj Z(-k)) / 2i, and sum_p t(p) d(p + s) has the transform conj(F) G.
// The correlation is real, so kx beyond P1 / 2 is the conjugate of P1 - kx and not
// formed.  Z is [kx][ky], C [kx][oy].
__global__ void __launch_bounds__(1024)
    k_fft_spectrum(const double2 *__restrict__ Z, double2 *__restrict__ C, int P1, int L, int logL,
                   const double2 *__restrict__ tw) {
  extern __shared__ double2 s[];
  const int kx = blockIdx.x;
  const double2 *zk = Z + (long long)kx * L, *zm = Z + (long long)((P1 - kx) & (P1 - 1)) * L;
  double2 *row = C + (long long)kx * L;
  fft_row<true>(
      s, L, logL, tw,
      [&](int ky) {
        const double2 z = zk[ky], w = zm[(L - ky) & (L - 1)];
        const double2 F = make_double2(0.5 * (z.x + w.x), 0.5 * (z.y - w.y));
        const double2 Gm = make_double2(z.x - w.x, z.y + w.y);  // Z(k) - conj Z(-k)
        const double2 G = make_double2(0.5 * Gm.y, -0.5 * Gm.x);
        return make_double2(F.x * G.x + F.y * G.y, F.x * G.y - F.y * G.x);
      },
      [&](int y, double2 v) { row[y] = v; });
}

// out (C x R, rows ldo apart) = in (R x C, rows ldi apart)^T
__global__ void k_transpose_c(const double2 *__restrict__ in, double2 *__restrict__ out, int R, int Cn, int ldi,
                              int ldo) {
  __shared__ double2 t[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int r = r0 + k, c = c0 + threadIdx.x;
    if (r < R && c < Cn) t[k][threadIdx.x] = in[(long long)r * ldi + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int c = c0 + k, r = r0 + threadIdx.x;
    if (r < R && c < Cn) out[(long long)c * ldo + r] = t[threadIdx.x][k];
  }
}

// Level-1 normalised cross-correlation at map entry e of the (2a-1) x (2b-1)
// map (column-major, rows = x shifts): D offset (ox, oy) of the template.
template <typename S>
struct L1Args {
  const S *sat;          // the four tables
  long long plane;       // one table's entries
  int W1, gx0, gy0;      // table row length, 0-based ROI origin
  int a, b;
  long long mn;
  double *c;             // correlation, unscaled: row oy + b - 1, column ox mod P1
  int P1;
  double inv;            // 1 / (P1 P2)
  const double *mu;
  bool narrow;           // mn sum(g^2) < 2^63
};

// what every entry shares
template <typename S>
struct L1Consts {
  S st, st2;
  double denT, mu;
};
template <typename S>
__device__ __forceinline__ L1Consts<S> l1_consts(const L1Args<S> &A) {
  L1Consts<S> K;
  K.st = rect_sum(A.sat, A.W1, A.gx0, A.gx0 + A.a, A.gy0, A.gy0 + A.b);
  K.st2 = rect_sum(A.sat + A.plane, A.W1, A.gx0, A.gx0 + A.a, A.gy0, A.gy0 + A.b);
  if constexpr (std::is_integral<S>::value)
    K.denT = (double)((__int128)A.mn * K.st2 - (__int128)K.st * K.st);
  else
    K.denT = (double)A.mn * K.st2 - K.st * K.st;
  K.mu = *A.mu;
  return K;
}
// window part of the denominator; n_in entries of the window lie in the region
template <typename S>
__device__ __forceinline__ double l1_den(const L1Args<S> &A, double mu, S sd, S sd2, long long n_in) {
  const long long n_pad = A.mn - n_in;
  double C0, Cc = 0.0;
  if constexpr (std::is_integral<S>::value) {
    if (A.narrow) {  // the products below hold in 64 bits too: the same numbers
      C0 = (double)(A.mn * sd2 - sd * sd);
      if (n_pad > 0) Cc = mu * ((double)(n_pad * n_in) * mu - 2.0 * (double)(sd * n_pad));
    } else {
      C0 = (double)((__int128)A.mn * sd2 - (__int128)sd * sd);
      if (n_pad > 0) Cc = mu * ((double)((__int128)n_pad * n_in) * mu - 2.0 * (double)((__int128)sd * n_pad));
    }
  } else {
    C0 = (double)A.mn * sd2 - sd * sd;
    if (n_pad > 0) Cc = mu * ((double)n_pad * (double)n_in * mu - 2.0 * (sd * (double)n_pad));
  }
  return C0 + Cc;
}
__device__ __forceinline__ double l1_r(double num, double denT, double den) {
  if (!(den > 0.0)) return 0.0;
  double r = num / sqrt(denT * den);
  if (fabs(r) - 1.0 > kSqrtEps) r = 0.0;
  return r;
}

// NCC at shift (ox, oy) from the stored correlation
template <typename S>
__device__ double l1_ncc(const L1Args<S> &A, const L1Consts<S> &K, int ox, int oy) {
  const int x0 = max(0, ox), x1 = min(A.a, A.a + ox), y0 = max(0, oy), y1 = min(A.b, A.b + oy);
  if (x1 <= x0 || y1 <= y0) return 0.0;
  const S *satg = A.sat + 2 * A.plane;
  const S sd = rect_sum(satg, A.W1, A.gx0 + x0, A.gx0 + x1, A.gy0 + y0, A.gy0 + y1);
  const S sd2 = rect_sum(satg + A.plane, A.W1, A.gx0 + x0, A.gx0 + x1, A.gy0 + y0, A.gy0 + y1);
  const double cv = A.c[(long long)(oy + A.b - 1) * A.P1 + (ox & (A.P1 - 1))] * A.inv;
  return l1_r((double)A.mn * cv, K.denT, l1_den(A, K.mu, sd, sd2, (long long)(x1 - x0) * (y1 - y0)));
}

__device__ __forceinline__ void argmax_merge(double &bv, long long &bi, double v, long long i) {
  if (v > bv || (v == bv && i < bi)) {
    bv = v;
    bi = i;
  }
}
__device__ __forceinline__ void argmax_warp(double &bv, long long &bi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    argmax_merge(bv, bi, __shfl_xor_sync(0xffffffffu, bv, o), __shfl_xor_sync(0xffffffffu, bi, o));
}

// The last inverse transform, along x, two rows oy at once (the correlation is
// real: row oy in the real part, oy + 1 in the imaginary part), and the maximum
// over the two rows' map entries.  The window sums of a row need two table rows,
// and one varying column of them; the root and the division are formed only
// where num^2 reaches the thread's best entry so far.  C is [oy mod P2][kx] with
// rows ldc apart.
template <typename S>
__global__ void __launch_bounds__(1024)
    k_fft_ncc(const double2 *__restrict__ C, int ldc, int P2, const __grid_constant__ L1Args<S> A, int logL,
              const double2 *__restrict__ tw, double *__restrict__ pv, long long *__restrict__ pi) {
  extern __shared__ double2 s[];
  __shared__ double sv[32];
  __shared__ long long si[32];
  const int L = A.P1, rows = 2 * A.b - 1;
  const int r0 = 2 * blockIdx.x, two = r0 + 1 < rows;
  const double2 *ca = C + (long long)((r0 - (A.b - 1)) & (P2 - 1)) * ldc;
  const double2 *cb = C + (long long)((r0 + 1 - (A.b - 1)) & (P2 - 1)) * ldc;
  fft_row<true>(
      s, L, logL, tw,
      [&](int kx) {
        const bool up = kx <= L / 2;
        const int k = up ? kx : L - kx;
        const double2 u = ca[k], v = two ? cb[k] : make_double2(0.0, 0.0);
        return up ? make_double2(u.x - v.y, u.y + v.x) : make_double2(u.x + v.y, v.x - u.y);
      },
      [&](int x, double2 v) { s[fft_pos(x)] = v; });
  __syncthreads();
  const L1Consts<S> K = l1_consts(A);
  double bv = -1e300;
  long long bi = 0x7fffffffffffffffll;
  for (int h = 0; h <= two; ++h) {
    const int r = r0 + h, oy = r - (A.b - 1), y0 = max(0, oy), y1 = min(A.b, A.b + oy);
    const S *g0 = A.sat + 2 * A.plane + (long long)(A.gy0 + y0) * A.W1 + A.gx0;
    const S *g1 = g0 + (long long)(y1 - y0) * A.W1;
    const S *q0 = g0 + A.plane, *q1 = g1 + A.plane;
    const S ga = g1[A.a] - g0[A.a], gz = g1[0] - g0[0], qa = q1[A.a] - q0[A.a], qz = q1[0] - q0[0];
    double *crow = A.c + (long long)r * L;
    for (int x = threadIdx.x; x < L; x += blockDim.x) {
      const double2 cc = s[fft_pos(x)];
      const double c = h ? cc.y : cc.x;
      crow[x] = c;
      const int ox = x < A.a ? x : x - L;
      if (ox <= -A.a) continue;  // no entry of the map
      const int e = ox >= 0 ? ox : A.a + ox;  // the window's inner edge
      const S ge = g1[e] - g0[e], qe = q1[e] - q0[e];
      const S sd = ox >= 0 ? ga - ge : ge - gz, sd2 = ox >= 0 ? qa - qe : qe - qz;
      const double den = l1_den(A, K.mu, sd, sd2, (long long)(A.a - abs(ox)) * (y1 - y0));
      const double num = (double)A.mn * (c * A.inv);
      if (bv > 0.0 && (!(num > 0.0) || num * num < bv * bv * (1.0 - 1e-12) * (K.denT * den))) continue;
      argmax_merge(bv, bi, l1_r(num, K.denT, den), (long long)r * (2 * A.a - 1) + (ox + A.a - 1));
    }
  }
  argmax_warp(bv, bi);
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = bv;
    si[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const bool in = threadIdx.x < blockDim.x / 32;
    bv = in ? sv[threadIdx.x] : -1e300;
    bi = in ? si[threadIdx.x] : 0x7fffffffffffffffll;
    argmax_warp(bv, bi);
    if (threadIdx.x == 0) {
      pv[blockIdx.x] = bv;
      pi[blockIdx.x] = bi;
    }
  }
}

// out = {row, col, max_f} of findpeak over the level-1 map, {constant template}; one warp
template <typename S>
__global__ void k_mg_l1_peak(const __grid_constant__ L1Args<S> A, const double *__restrict__ pv,
                             const long long *__restrict__ pi, int np, double *__restrict__ out) {
  const int lane = threadIdx.x;
  double bv = -1e300;
  long long bi = 0x7fffffffffffffffll;
  for (int k = lane; k < np; k += 32) argmax_merge(bv, bi, pv[k], pi[k]);
  argmax_warp(bv, bi);
  const L1Consts<S> K = l1_consts(A);
  const int nr = 2 * A.a - 1, nc = 2 * A.b - 1;
  const int r = (int)(bi % nr), c = (int)(bi / nr);
  double rp = r + 1, cp = c + 1, mf = bv;
  if (!(r == 0 || r == nr - 1 || c == 0 || c == nc - 1)) {
    const double mine = lane < 9 ? l1_ncc(A, K, r + lane % 3 - 1 - (A.a - 1), c + lane / 3 - 1 - (A.b - 1)) : 0.0;
    double u9[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) u9[q] = __shfl_sync(0xffffffffu, mine, q);
    findpeak_fit9(u9, r, c, &rp, &cp, &mf);
  }
  if (lane == 0) {
    out[0] = rp;
    out[1] = cp;
    out[2] = mf;
    out[3] = K.denT > 0.0 ? 0.0 : 1.0;
  }
}

// ------------------------------------------------------------ intermediate levels
// Exact sum of t * d over one (region, 8-row band, 256-column tile) for the
// 13 x 14 shifts of the crop, added into acc[region][182] (column-major,
// rows = ox + 1, ox in [-1, 11]; columns oy + 1, oy in [-1, 12]).  D pixels
// outside the region read 0 (their padding is the mu term of the NCC).
// Column segment per thread: 16 columns (8 for FP64 pixels, to keep the
// static shared memory of the tile under 48 KB); 16 segments per tile.
template <typename P> struct CropCfg {
  static constexpr int SW = sizeof(typename MgT<P>::V) == 8 ? 8 : 16;
  static constexpr int TILE = kSegs * SW;
};

// Four pixels of a row as the words of its byte planes (16 bit: high, low), zeros
// outside columns [lo, hi); row points at column 0.  A word that lies inside is
// read as aligned words (the images have spare bytes behind them).
template <typename P>
__device__ __forceinline__ void four_pixels(const P *row, int x, int lo, int hi, uint32_t w[sizeof(P)]) {
  if (x >= lo && x + 4 <= hi) {
    const uintptr_t at = (uintptr_t)(row + x);
    const uint32_t *q = (const uint32_t *)(at & ~(uintptr_t)3);
    const uint32_t sh = 8 * (uint32_t)(at & 3);
    if constexpr (sizeof(P) == 1) {
      w[0] = __funnelshift_r(q[0], q[1], sh);
    } else {
      const uint32_t v0 = __funnelshift_r(q[0], q[1], sh), v1 = __funnelshift_r(q[1], q[2], sh);
      w[0] = __byte_perm(v0, v1, 0x7531);
      w[1] = __byte_perm(v0, v1, 0x6420);
    }
    return;
  }
#pragma unroll
  for (int p = 0; p < (int)sizeof(P); ++p) w[p] = 0;
  for (int e = 0; e < 4; ++e)
    if (x + e >= lo && x + e < hi) {
      const uint32_t v = row[x + e];
#pragma unroll
      for (int p = 0; p < (int)sizeof(P); ++p) w[p] |= ((v >> (8 * (sizeof(P) - 1 - p))) & 255u) << (8 * e);
    }
}

// The sums of products of byte planes: one (8 bit) or high x high, the mixed two,
// low x low (16 bit), each exact in 32 bits.
template <int PL>
struct PlaneSums {
  uint32_t s[PL == 1 ? 1 : 3];
  __device__ __forceinline__ void add(const uint32_t t[PL], const uint32_t d[PL]) {
    if constexpr (PL == 1) {
      s[0] = __dp4a(t[0], d[0], s[0]);
    } else {
      s[0] = __dp4a(t[0], d[0], s[0]);
      s[1] = __dp4a(t[0], d[1], s[1]);
      s[1] = __dp4a(t[1], d[0], s[1]);
      s[2] = __dp4a(t[1], d[1], s[2]);
    }
  }
  __device__ __forceinline__ unsigned long long total() const {
    if constexpr (PL == 1) return s[0];
    return ((unsigned long long)s[0] << 16) + ((unsigned long long)s[1] << 8) + s[PL == 1 ? 0 : 2];
  }
};

// The crop's sums of 8- and 16-bit images, four products an instruction: bands
// of 32 rows and 256 columns in shared memory as packed words, a thread one y
// shift and 16 columns, its region words shifted to the four byte offsets in
// registers for all 13 x shifts.  In a region narrower than the tile the spare
// threads take every second, fourth ... row.  All levels of a 2048 x 2048 search
// (3.8 G products): 171 us, 815 us with one product an instruction and
// 16-way bank conflicts.
constexpr int kBandI = 32, kTileI = 256;
template <typename P>
__global__ void __launch_bounds__(224) k_mg_crop_int(const P *__restrict__ f, const P *__restrict__ g, int W,
                                                     const MgReg *__restrict__ regs,
                                                     unsigned long long *__restrict__ acc) {
  constexpr int PL = sizeof(P), TW = kTileI / 4, DW = TW + 4, DR = kBandI + kCropC - 1;
  __shared__ __align__(16) uint32_t Ts[PL][kBandI][TW], Ds[PL][DR][DW];
  const MgReg R = regs[blockIdx.x];
  if (!R.valid) return;
  const int q0 = blockIdx.y * kBandI, x0 = blockIdx.z * kTileI;
  if (q0 >= R.b || x0 >= R.a) return;
  const int nq = min(kBandI, R.b - q0), nx = min(kTileI, R.a - x0);
  const int dwid = R.a + 10, dhgt = R.b + 10;
  const int words = (nx + 15) / 16 * 4;  // of a template row, whole segments
  for (int e = threadIdx.x; e < nq * words; e += blockDim.x) {
    const int qq = e / words, m = e - qq * words;
    uint32_t w[PL];
    four_pixels(f + (long long)(R.ty - 1 + q0 + qq) * W + (R.tx - 1 + x0), 4 * m, 0, nx, w);
#pragma unroll
    for (int p = 0; p < PL; ++p) Ts[p][qq][m] = w[p];
  }
  const int dwords = words + 4, drows = nq + kCropC - 1;
  for (int e = threadIdx.x; e < drows * dwords; e += blockDim.x) {
    const int r = e / dwords, m = e - r * dwords, yl = q0 - 1 + r;  // region row
    uint32_t w[PL] = {};
    if (yl >= 0 && yl < dhgt) {
      // column c of the tile is the region's x0 - 1 + c
      const P *row = g + (long long)(R.dy - 1 + yl) * W + (R.dx - 1);
      four_pixels(row, x0 - 1 + 4 * m, 0, dwid, w);
    }
#pragma unroll
    for (int p = 0; p < PL; ++p) Ds[p][r][m] = w[p];
  }
  __syncthreads();
  const int oyi = threadIdx.x / kSegs, lane16 = threadIdx.x % kSegs;  // oy = oyi - 1
  int ns = 1;  // segments, a power of two
  while (ns < words / 4) ns <<= 1;
  const int seg = lane16 & (ns - 1), every = kSegs / ns;
  PlaneSums<PL> s[kCropR] = {};
  if (4 * seg < words) {
    for (int qq = lane16 / ns; qq < nq; qq += every) {
      uint32_t t[PL][4], d[PL][8];
#pragma unroll
      for (int p = 0; p < PL; ++p) {
        *(uint4 *)t[p] = *(const uint4 *)&Ts[p][qq][4 * seg];
        *(uint4 *)d[p] = *(const uint4 *)&Ds[p][qq + oyi][4 * seg];
        *(uint4 *)(d[p] + 4) = *(const uint4 *)&Ds[p][qq + oyi][4 * seg + 4];
      }
#pragma unroll
      for (int sh = 0; sh < 4; ++sh) {
        uint32_t v[7][PL];
#pragma unroll
        for (int j = 0; j < 7; ++j)
#pragma unroll
          for (int p = 0; p < PL; ++p) v[j][p] = sh ? __funnelshift_r(d[p][j], d[p][j + 1], 8 * sh) : d[p][j];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t ti[PL];
#pragma unroll
          for (int p = 0; p < PL; ++p) ti[p] = t[p][i];
#pragma unroll
          for (int m = 0; m < 4; ++m)
            if (4 * m + sh < kCropR) s[4 * m + sh].add(ti, v[i + m]);
        }
      }
    }
  }
  // the 16 threads of a y shift: at most 32 x 256 products of 2^16, twice
  const unsigned half = 0xffffu << (threadIdx.x & 16);
#pragma unroll
  for (int k = 0; k < kCropR; ++k) {
#pragma unroll
    for (uint32_t &v : s[k].s) v = __reduce_add_sync(half, v);
    const unsigned long long v = s[k].total();
    if (lane16 == 0 && v) atomicAdd(&acc[(long long)blockIdx.x * kCrop + oyi * kCropR + k], v);
  }
}

template <typename P>
__global__ void __launch_bounds__(224) k_mg_crop(const P *__restrict__ f, const P *__restrict__ g,
                                                 int W, const MgReg *__restrict__ regs,
                                                 typename MgT<P>::G *__restrict__ acc) {
  using V = typename MgT<P>::V;
  using G = typename MgT<P>::G;
  constexpr int kTile = CropCfg<P>::TILE, kSeg = CropCfg<P>::SW;
  constexpr int TS = kTile + 4;             // template row stride
  constexpr int DS = kTile + 16 + 4;        // region row stride (tile + 12 halo, padded)
  constexpr int DR = kBand + kCropC - 1;    // region rows: band + 13
  __shared__ V Ts[kBand][TS];
  __shared__ V Ds[DR][DS];
  const MgReg R = regs[blockIdx.x];
  if (!R.valid) return;
  const int q0 = blockIdx.y * kBand, x0 = blockIdx.z * kTile;
  if (q0 >= R.b || x0 >= R.a) return;
  const int nq = min(kBand, R.b - q0), nx = min(kTile, R.a - x0);
  const int dwid = R.a + 10, dhgt = R.b + 10;
  for (int e = threadIdx.x; e < kBand * kTile; e += blockDim.x) {
    const int qq = e / kTile, xx = e - qq * kTile;
    V t = 0;
    if (qq < nq && xx < nx)
      t = (V)f[(long long)(R.ty - 1 + q0 + qq) * W + (R.tx - 1 + x0 + xx)];
    Ts[qq][xx] = t;
  }
  for (int e = threadIdx.x; e < DR * (kTile + 16); e += blockDim.x) {
    const int r = e / (kTile + 16), cidx = e - r * (kTile + 16);
    const int yl = q0 - 1 + r, xl = x0 - 1 + cidx;  // region-local
    V d = 0;
    if (yl >= 0 && yl < dhgt && xl >= 0 && xl < dwid && cidx < nx + 12)
      d = (V)g[(long long)(R.dy - 1 + yl) * W + (R.dx - 1 + xl)];
    Ds[r][cidx] = d;
  }
  __syncthreads();
  const int oyi = threadIdx.x / kSegs, seg = threadIdx.x - oyi * kSegs;  // oy = oyi - 1
  const int xs = seg * kSeg;
  V s[kCropR];
#pragma unroll
  for (int k = 0; k < kCropR; ++k) s[k] = 0;
  if (xs < nx) {
    for (int qq = 0; qq < nq; ++qq) {
      const V *dr = &Ds[qq + oyi][xs];  // region row q0 + qq + oy
      const V *tr = &Ts[qq][xs];
      V win[kSeg + kCropR - 1];
#pragma unroll
      for (int k = 0; k < kSeg + kCropR - 1; ++k) win[k] = dr[k];
#pragma unroll
      for (int xx = 0; xx < kSeg; ++xx) {
        const V t = tr[xx];
#pragma unroll
        for (int k = 0; k < kCropR; ++k) s[k] += t * win[xx + k];
      }
    }
  }
  // reduce over the 16 column segments of the same oy (consecutive lanes)
#pragma unroll
  for (int k = 0; k < kCropR; ++k) {
    G v = (G)s[k];
#pragma unroll
    for (int o = kSegs / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, kSegs);
    if (seg == 0 && v != G(0)) atomicAdd(&acc[(long long)blockIdx.x * kCrop + oyi * kCropR + k], v);
  }
}

// first maximum of a crop, by one warp
__device__ __forceinline__ int crop_max(const double *map) {
  const int lane = threadIdx.x & 31;
  double bv = map[lane];
  long long bi = lane;
  for (int e = lane + 32; e < kCrop; e += 32) argmax_merge(bv, bi, map[e], e);
  argmax_warp(bv, bi);
  return (int)bi;
}

// NCC of the 182 crop entries from the products and the window sums, then
// findpeak: res[region] = {u offset, v offset, Phi, ok}.
template <typename P>
__global__ void k_mg_crop_peak(const MgReg *__restrict__ regs, int W, int H,
                               const typename MgT<P>::S *__restrict__ sat,
                               const typename MgT<P>::G *__restrict__ acc,
                               const double *__restrict__ mu_g, double *__restrict__ res) {
  using S = typename MgT<P>::S;
  __shared__ double map[kCrop];
  __shared__ int s_flat;
  const MgReg R = regs[blockIdx.x];
  double *o = res + (long long)blockIdx.x * 8;
  if (!R.valid) {
    if (threadIdx.x == 0) o[3] = 0.0;
    return;
  }
  const int W1 = W + 1;
  const long long plane = (long long)W1 * (H + 1);
  const S *sf = sat, *sf2 = sat + plane, *sg = sat + 2 * plane, *sg2 = sat + 3 * plane;
  const long long mn = (long long)R.a * R.b;
  const int tx0i = R.tx - 1, ty0i = R.ty - 1, dx0i = R.dx - 1, dy0i = R.dy - 1;
  const S st = rect_sum(sf, W1, tx0i, tx0i + R.a, ty0i, ty0i + R.b);
  const S st2 = rect_sum(sf2, W1, tx0i, tx0i + R.a, ty0i, ty0i + R.b);
  if (threadIdx.x == 0) {
    bool flat;
    if constexpr (MgT<P>::integer)
      flat = ((__int128)mn * (long long)st2 - (__int128)(long long)st * (long long)st) == 0;
    else
      flat = !((double)mn * (double)st2 - (double)st * (double)st > 0.0);
    s_flat = flat;
  }
  const double mu = *mu_g;
  for (int e = threadIdx.x; e < kCrop; e += blockDim.x) {
    const int ox = e % kCropR - 1, oy = e / kCropR - 1;
    const int tx0 = max(0, -ox), tx1 = min(R.a, R.a + 10 - ox);
    const int ty0 = max(0, -oy), ty1 = min(R.b, R.b + 10 - oy);
    double r = 0.0;
    if (tx1 > tx0 && ty1 > ty0) {
      const long long n_in = (long long)(tx1 - tx0) * (ty1 - ty0);
      const S st_in = rect_sum(sf, W1, tx0i + tx0, tx0i + tx1, ty0i + ty0, ty0i + ty1);
      const S sd = rect_sum(sg, W1, dx0i + tx0 + ox, dx0i + tx1 + ox, dy0i + ty0 + oy, dy0i + ty1 + oy);
      const S sd2 = rect_sum(sg2, W1, dx0i + tx0 + ox, dx0i + tx1 + ox, dy0i + ty0 + oy, dy0i + ty1 + oy);
      const S stdv = (S)acc[(long long)blockIdx.x * kCrop + e];
      r = combine<S>(mn, st, st2, stdv, sd, sd2, st - st_in, mn - n_in, mu);
    }
    map[e] = r;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  if (s_flat) {
    if (threadIdx.x == 0) o[3] = 0.0;
    return;
  }
  const int im = crop_max(map);
  if (threadIdx.x == 0) {
    double rp, cp, mf;
    findpeak_fit(map, kCropR, kCropC, im, &rp, &cp, &mf);
    o[0] = __dsub_rn(rp, 7.0);
    o[1] = __dsub_rn(cp, 7.0);
    o[2] = mf;
    o[3] = 1.0;
  }
}

// ------------------------------------------------------------ last level
// One CTA per region: the full normxcorr2 map (2a+9) x (2b+9) in shared
// memory, compute_qFactor over it, findpeak on its 13 x 14 crop.
// res[region] = {u offset, v offset, Phi, ok, PCE, 1/entropy}.
// k_mg_full's operands of integer images as words: of a template row, of a region
// row, and the zero columns before the region's first (strips start at shifts a
// multiple of kStrip from -(a - 1), so each starts a word)
struct FullWords {
  int tw, dw, pad;
  __host__ __device__ explicit FullWords(int a) : tw((a + 3) / 4), dw((2 * a + 12) / 4 + 3), pad(a - 1) {}
};

template <typename P>
__global__ void __launch_bounds__(256) k_mg_full(const P *__restrict__ f, const P *__restrict__ g,
                                                 int W, int H, const MgReg *__restrict__ regs,
                                                 const typename MgT<P>::S *__restrict__ sat,
                                                 const double *__restrict__ mu_g,
                                                 double *__restrict__ res) {
  using S = typename MgT<P>::S;
  using V = typename MgT<P>::V;
  constexpr int PL = MgT<P>::integer ? sizeof(P) : 1;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[64];
  __shared__ int hist[30];
  __shared__ double crop[kCrop];
  const MgReg R = regs[blockIdx.x];
  double *o = res + (long long)blockIdx.x * 8;
  if (!R.valid) {
    if (threadIdx.x == 0) o[3] = 0.0;
    return;
  }
  const int a = R.a, b = R.b, dw = a + 10, dh = b + 10;
  const int fr = a + dw - 1, fc = b + dh - 1, nm = fr * fc;
  double *map = (double *)smem;
  // floats: template rows padded with 8 zero columns, region rows with kStrip zero
  // columns on the left and kStrip + 8 on the right.  Integers: words of a byte
  // plane, template rows from column 0, region rows so that every strip's first
  // shift starts a word; zeros around
  const int TP = a + 8, DP = dw + 2 * kStrip + 8;
  V *Ts = (V *)(map + nm);
  V *Ds = Ts + TP * b;
  const FullWords FW(a);
  uint32_t *const Tw = (uint32_t *)(map + nm), *const Dw = Tw + PL * b * FW.tw;
  if constexpr (MgT<P>::integer) {
    for (int e = threadIdx.x; e < b * FW.tw; e += blockDim.x) {
      const int ty = e / FW.tw, m = e - ty * FW.tw;
      uint32_t w[PL];
      four_pixels(f + (long long)(R.ty - 1 + ty) * W + (R.tx - 1), 4 * m, 0, a, w);
#pragma unroll
      for (int p = 0; p < PL; ++p) Tw[p * b * FW.tw + e] = w[p];
    }
    for (int e = threadIdx.x; e < dh * FW.dw; e += blockDim.x) {
      const int yy = e / FW.dw, m = e - yy * FW.dw;
      uint32_t w[PL];
      four_pixels(g + (long long)(R.dy - 1 + yy) * W + (R.dx - 1), 4 * m - FW.pad, 0, dw, w);
#pragma unroll
      for (int p = 0; p < PL; ++p) Dw[p * dh * FW.dw + e] = w[p];
    }
  } else {
    for (int e = threadIdx.x; e < TP * b; e += blockDim.x) {
      const int ty = e / TP, tx = e - ty * TP;
      Ts[e] = tx < a ? (V)f[(long long)(R.ty - 1 + ty) * W + (R.tx - 1 + tx)] : (V)0;
    }
    for (int e = threadIdx.x; e < dh * DP; e += blockDim.x) {
      const int yy = e / DP, xx = e - yy * DP - kStrip;
      Ds[e] = (xx >= 0 && xx < dw) ? (V)g[(long long)(R.dy - 1 + yy) * W + (R.dx - 1 + xx)] : (V)0;
    }
  }
  if (threadIdx.x < 30) hist[threadIdx.x] = 0;
  const int W1 = W + 1;
  const long long plane = (long long)W1 * (H + 1);
  const S *sf = sat, *sf2 = sat + plane, *sg = sat + 2 * plane, *sg2 = sat + 3 * plane;
  const long long mn = (long long)a * b;
  const int tx0i = R.tx - 1, ty0i = R.ty - 1, dx0i = R.dx - 1, dy0i = R.dy - 1;
  const S st = rect_sum(sf, W1, tx0i, tx0i + a, ty0i, ty0i + b);
  const S st2 = rect_sum(sf2, W1, tx0i, tx0i + a, ty0i, ty0i + b);
  bool flat;
  if constexpr (MgT<P>::integer)
    flat = ((__int128)mn * (long long)st2 - (__int128)(long long)st * (long long)st) == 0;
  else
    flat = !((double)mn * (double)st2 - (double)st * (double)st > 0.0);
  if (flat) {
    if (threadIdx.x == 0) o[3] = 0.0;
    return;
  }
  const double mu = *mu_g;
  __syncthreads();
  double denT = 0.0;
  if constexpr (MgT<P>::integer) denT = (double)(mn * st2 - st * st);
  // NCC of map entry (i, j) from its sum of products.  8 bit: window sums below
  // 2^32, so that the tables' low words give them, and products of 32-bit factors
  auto entry = [&](int i, int j, S stdv) {
    const int ox = i - (a - 1), oy = j - (b - 1);
    const int tx0 = max(0, -ox), tx1 = min(a, dw - ox), ty0 = max(0, -oy), ty1 = min(b, dh - oy);
    if (tx1 <= tx0 || ty1 <= ty0) return 0.0;
    if constexpr (sizeof(P) == 1) {
      auto sum = [&](const S *table, int x, int y) {
        const uint32_t *t = (const uint32_t *)(table + (long long)y * W1 + x);
        const int w2 = 2 * (tx1 - tx0), up = 2 * W1 * (ty1 - ty0);
        return (t[up + w2] - t[w2]) - (t[up] - t[0]);
      };
      const uint32_t m = a * b, n_in = (tx1 - tx0) * (ty1 - ty0), n_pad = m - n_in, s1 = (uint32_t)st;
      const uint32_t pad = s1 - sum(sf, tx0i + tx0, ty0i + ty0);
      const int xg = dx0i + tx0 + ox, yg = dy0i + ty0 + oy;
      const uint32_t sd = sum(sg, xg, yg), sd2 = sum(sg2, xg, yg);
      auto times = [](uint32_t u, uint32_t v) { return (long long)((unsigned long long)u * v); };
      // ncc_combine's operations on the same integers
      double num = (double)(times(m, (uint32_t)stdv) - times(s1, sd)), den = (double)(times(m, sd2) - times(sd, sd));
      double B = 0.0, Cc = 0.0;
      if (n_pad > 0) {
        B = __dmul_rn(mu, (double)(times(m, pad) - times(s1, n_pad)));
        Cc = __dmul_rn(mu, __dsub_rn(__dmul_rn((double)(n_pad * n_in), mu), __dmul_rn(2.0, (double)times(sd, n_pad))));
      }
      num = __dadd_rn(num, B);
      den = __dadd_rn(den, Cc);
      if (!(den > 0.0)) return 0.0;
      const double r = __ddiv_rn(num, __dsqrt_rn(__dmul_rn(denT, den)));
      return __dsub_rn(fabs(r), 1.0) > kSqrtEps ? 0.0 : r;
    }
    const long long n_in = (long long)(tx1 - tx0) * (ty1 - ty0);
    const S st_in = rect_sum(sf, W1, tx0i + tx0, tx0i + tx1, ty0i + ty0, ty0i + ty1);
    const S sd = rect_sum(sg, W1, dx0i + tx0 + ox, dx0i + tx1 + ox, dy0i + ty0 + oy, dy0i + ty1 + oy);
    const S sd2 = rect_sum(sg2, W1, dx0i + tx0 + ox, dx0i + tx1 + ox, dy0i + ty0 + oy, dy0i + ty1 + oy);
    // at most 80 x 80 pixels: 64-bit products hold
    if constexpr (MgT<P>::integer)
      return ncc_combine(mn, st, st2, stdv, sd, sd2, st - st_in, mn - n_in, mu);
    else
      return combine<S>(mn, st, st2, stdv, sd, sd2, st - st_in, mn - n_in, mu);
  };
  // strips of kStrip consecutive x shifts (map rows) at one y shift
  const int nsr = (fr + kStrip - 1) / kStrip;
  if constexpr (MgT<P>::integer) {
    // Four products an instruction (4096 regions of 33 x 33: the kernel 0.57 ms,
    // 1.64 ms with one): per template word one new region word, three
    // shifted ones (the other three are the last word's) and eight dp4a.  The
    // y shifts t and t + b + 10 (t < b - 1) overlap t + 1 and b - 1 - t rows: a
    // thread takes both, so each has the same b rows, and the 11 full ones alone.
    unsigned long long *const raw = (unsigned long long *)map;
    const int nv = b + 10;
    for (int sI = threadIdx.x; sI < nsr * nv; sI += blockDim.x) {
      const int i0 = sI / nv * kStrip, v = sI % nv, ox0 = i0 - (a - 1);
      const bool pair = v < b - 1;
      const int r1 = pair ? v + 1 : b;  // rows of the first y shift
      const int wa = max(0, -(ox0 + kStrip - 1)) >> 2, wb = (min(a, dw - ox0) + 3) >> 2;
      PlaneSums<PL> s[kStrip] = {};
      int j = v, ty = pair ? b - 1 - v : max(0, (b - 1) - v);
      const int dcol = (FW.pad + ox0) >> 2;  // the region word of template word 0
      for (int r = 0; r < b; ++r, ++ty) {
        if (r == r1) {  // on to the second y shift
#pragma unroll
          for (int k = 0; k < kStrip; ++k) {
            if (i0 + k < fr) raw[(long long)j * fr + i0 + k] = s[k].total();
            s[k] = PlaneSums<PL>{};
          }
          j = v + b + 10;
          ty = 0;
        }
        const uint32_t *tr = Tw + ty * FW.tw;
        const uint32_t *dr = Dw + (ty + j - (b - 1)) * FW.dw + dcol;
        uint32_t d0[PL], d1[PL], lo[4][PL];
#pragma unroll
        for (int p = 0; p < PL; ++p) {
          d0[p] = dr[p * dh * FW.dw + wa];
          d1[p] = dr[p * dh * FW.dw + wa + 1];
          lo[0][p] = d0[p];
#pragma unroll
          for (int e = 1; e < 4; ++e) lo[e][p] = __funnelshift_r(d0[p], d1[p], 8 * e);
        }
        for (int m = wa; m < wb; ++m) {
          uint32_t t[PL], hi[4][PL];
#pragma unroll
          for (int p = 0; p < PL; ++p) {
            t[p] = tr[p * b * FW.tw + m];
            const uint32_t d2 = dr[p * dh * FW.dw + m + 2];
            hi[0][p] = d1[p];
#pragma unroll
            for (int e = 1; e < 4; ++e) hi[e][p] = __funnelshift_r(d1[p], d2, 8 * e);
            d1[p] = d2;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[e].add(t, lo[e]);
            s[e + 4].add(t, hi[e]);
#pragma unroll
            for (int p = 0; p < PL; ++p) lo[e][p] = hi[e][p];
          }
        }
      }
#pragma unroll
      for (int k = 0; k < kStrip; ++k)
        if (i0 + k < fr) raw[(long long)j * fr + i0 + k] = s[k].total();
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nm; e += blockDim.x) map[e] = entry(e % fr, e / fr, (S)raw[e]);
  } else {
    // the template columns run in chunks of 8 over zero-padded rows, so the 8 x 8
    // products of a chunk are fully unrolled in registers
    for (int sI = threadIdx.x; sI < nsr * fc; sI += blockDim.x) {
      const int j = sI / nsr, i0 = (sI - j * nsr) * kStrip;
      const int oy = j - (b - 1), ox0 = i0 - (a - 1);
      const int ty0 = max(0, -oy), ty1 = min(b, dh - oy);
      const int txa = max(0, -(ox0 + kStrip - 1)), txb = min(a, dw - ox0);
      V s[kStrip];
#pragma unroll
      for (int k = 0; k < kStrip; ++k) s[k] = 0;
      for (int ty = ty0; ty < ty1; ++ty) {
        const V *tr = Ts + ty * TP;
        const V *dr = Ds + (ty + oy) * DP + kStrip + ox0;  // dr[tx + k]: region x = tx + ox0 + k
        for (int tx = txa; tx < txb; tx += 8) {
          V tv[8], dv[15];
#pragma unroll
          for (int q = 0; q < 8; ++q) tv[q] = tr[tx + q];
#pragma unroll
          for (int q = 0; q < 15; ++q) dv[q] = dr[tx + q];
#pragma unroll
          for (int q = 0; q < 8; ++q)
#pragma unroll
            for (int k = 0; k < kStrip; ++k) s[k] += tv[q] * dv[q + k];
        }
      }
#pragma unroll
      for (int k = 0; k < kStrip; ++k)
        if (i0 + k < fr) map[(long long)j * fr + i0 + k] = entry(i0 + k, j, (S)s[k]);
    }
  }
  __syncthreads();
  // compute_qFactor: min, then peak and sum of squares of cc - min, histogram
  const int tid = threadIdx.x, nth = blockDim.x;
  double mnv = 1e300;
  for (int e = tid; e < nm; e += nth) mnv = fmin(mnv, map[e]);
  for (int k = 16; k > 0; k >>= 1) mnv = fmin(mnv, __shfl_xor_sync(0xffffffffu, mnv, k));
  if ((tid & 31) == 0) red[tid >> 5] = mnv;
  __syncthreads();
  if (tid == 0) {
    for (int k = 1; k < nth / 32; ++k) mnv = fmin(mnv, red[k]);
    red[32] = mnv;
  }
  __syncthreads();
  mnv = red[32];
  __syncthreads();
  double pk = 0, ss = 0;
  for (int e = tid; e < nm; e += nth) {
    const double v = map[e] - mnv;
    pk = fmax(pk, v);
    ss += v * v;
  }
  for (int k = 16; k > 0; k >>= 1) {
    pk = fmax(pk, __shfl_xor_sync(0xffffffffu, pk, k));
    ss += __shfl_xor_sync(0xffffffffu, ss, k);
  }
  if ((tid & 31) == 0) {
    red[tid >> 5] = pk;
    red[32 + (tid >> 5)] = ss;
  }
  __syncthreads();
  if (tid == 0) {
    double Pk = 0, Sq = 0;
    for (int k = 0; k < nth / 32; ++k) {
      Pk = fmax(Pk, red[k]);
      Sq += red[32 + k];
    }
    red[0] = Pk;
    red[1] = Sq;
  }
  __syncthreads();
  const double peak = red[0], sumsq = red[1];
  for (int e = tid; e < nm; e += nth) {
    const double v = map[e] - mnv;
    int bb = peak > 0 ? (int)floor(v / peak * 30.0) : 0;
    bb = bb > 29 ? 29 : (bb < 0 ? 0 : bb);
    atomicAdd(&hist[bb], 1);
  }
  // crop rows a-2 .. a+10, columns b-2 .. b+11 (0-based) of the full map
  for (int e = tid; e < kCrop; e += nth) {
    const int r = e % kCropR, c = e / kCropR;
    crop[e] = map[(long long)(b - 2 + c) * fr + (a - 2 + r)];
  }
  __syncthreads();
  if (tid < 32) {
    const double n = (double)nm;
    // the entropy's terms a lane each, added in their order
    double term = 0.0;
    if (tid < 30) {
      const double p = hist[tid] / n;
      if (p > 0) term = p * log(1.0 / p);
    }
    double ent = 0;
    for (int k = 0; k < 30; ++k) ent += __shfl_sync(0xffffffffu, term, k);
    const int im = crop_max(crop);
    if (tid == 0) {
      o[4] = (peak * peak) / (sumsq / n);
      o[5] = 1.0 / ent;
      double rp, cp, mf;
      findpeak_fit(crop, kCropR, kCropC, im, &rp, &cp, &mf);
      o[0] = __dsub_rn(rp, 7.0);
      o[1] = __dsub_rn(cp, 7.0);
      o[2] = mf;
      o[3] = 1.0;
    }
  }
}

// ------------------------------------------------------------ gridfit gather
// A'A (9 coefficients per node, (di, dj) in row-major 3 x 3 order) and A'z of
// gridfit's triangle interpolation (gridfit.m:484-493) from the points of the
// four cells around each node.  Points are sorted by cell (cell = iy (nx-1) +
// ix, start[] its offsets); px, py their coordinates, pz their nr values
// (point-major).  rhs is field-major (nr x nx*ny).
__global__ void k_mg_ata(int nx, int ny, double x0, double y0, double h,
                         const int *__restrict__ start, const double *__restrict__ px,
                         const double *__restrict__ py, const double *__restrict__ pz, int nr,
                         double *__restrict__ ata, double *__restrict__ rhs) {
  const long long n = (long long)nx * ny;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k % nx), j = (int)(k / nx);
    double c9[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    double r[5] = {0, 0, 0, 0, 0};
    for (int cj = j - 1; cj <= j; ++cj)
      for (int ci = i - 1; ci <= i; ++ci) {
        if (ci < 0 || ci >= nx - 1 || cj < 0 || cj >= ny - 1) continue;
        const int c = cj * (nx - 1) + ci;
        for (int p = start[c]; p < start[c + 1]; ++p) {
          const double tx = fmin(1.0, fmax(0.0, (px[p] - (x0 + ci * h)) / h));
          const double ty = fmin(1.0, fmax(0.0, (py[p] - (y0 + cj * h)) / h));
          const double t1 = fmin(tx, ty), t2 = fmax(tx, ty);
          // the triangle's nodes and weights
          const int ni[3] = {ci, ci + 1, tx > ty ? ci + 1 : ci};
          const int nj[3] = {cj, cj + 1, tx > ty ? cj : cj + 1};
          const double wt[3] = {1 - t2, t1, t2 - t1};
          int me = -1;
          for (int q = 0; q < 3; ++q)
            if (ni[q] == i && nj[q] == j) me = q;
          if (me < 0) continue;
          const double wk = wt[me];
          for (int q = 0; q < 3; ++q) c9[(nj[q] - j + 1) * 3 + (ni[q] - i + 1)] += wk * wt[q];
          for (int m = 0; m < nr; ++m) r[m] += wk * pz[(long long)p * nr + m];
        }
      }
    for (int q = 0; q < 9; ++q) ata[9 * k + q] = c9[q];
    for (int m = 0; m < nr; ++m) rhs[m * n + k] = r[m];
  }
}

// ------------------------------------------------------------ host bookkeeping
struct Region {
  double xf[2], yf[2], xg[2], yg[2];
};

inline double mceil(double v) { return std::isfinite(v) ? std::ceil(v) : NAN; }
inline long long mround(double v) { return v >= 0 ? (long long)std::floor(v + 0.5) : -(long long)std::floor(-v + 0.5); }

// funIntegerSearchMg.m:37-46 / :180-199 (comparisons with NaN are false)
void clamp_region(Region &q, double bg, int W, int H) {
  if (q.xg[0] < bg) { const double t = q.xg[0]; q.xg[0] = bg; q.xf[0] = q.xf[0] + bg - t; }
  if (q.yg[0] < bg) { const double t = q.yg[0]; q.yg[0] = bg; q.yf[0] = q.yf[0] + bg - t; }
  if (q.xg[1] > W - bg) { const double t = q.xg[1]; q.xg[1] = W - bg; q.xf[1] = q.xf[1] + (W - bg) - t; }
  if (q.yg[1] > H - bg) { const double t = q.yg[1]; q.yg[1] = H - bg; q.yf[1] = q.yf[1] + (H - bg) - t; }
}
// :47-48 / :200-208: mod(width, 2) == 1 -> shrink both by one
void make_even(Region &q) {
  const double dx = q.xf[1] - q.xf[0], dy = q.yf[1] - q.yf[0];
  if (std::isfinite(dx) && std::fmod(dx, 2.0) == 1.0) { q.xf[1] -= 1; q.xg[1] -= 1; }
  if (std::isfinite(dy) && std::fmod(dy, 2.0) == 1.0) { q.yf[1] -= 1; q.yg[1] -= 1; }
}

bool int_range(double lo, double hi, int lim) {
  return std::isfinite(lo) && std::isfinite(hi) && lo == std::floor(lo) && hi == std::floor(hi) &&
         lo >= 1 && lo <= hi && hi <= lim;
}

// Device descriptor of one region (valid = the correlation does not raise).
MgReg describe(const Region &q, int W, int H) {
  MgReg r{};
  const bool ok = int_range(q.xf[0], q.xf[1], W) && int_range(q.yf[0], q.yf[1], H) &&
                  int_range(q.xg[0] - 5, q.xg[1] + 5, W) && int_range(q.yg[0] - 5, q.yg[1] + 5, H);
  if (!ok) return r;
  r.tx = (int)q.xf[0];
  r.ty = (int)q.yf[0];
  r.a = (int)(q.xf[1] - q.xf[0]) + 1;
  r.b = (int)(q.yf[1] - q.yf[0]) + 1;
  r.dx = (int)q.xg[0] - 5;
  r.dy = (int)q.yg[0] - 5;
  // g is sliced with the f width (xg = xf + shift), so the region is a + 10 wide
  r.valid = (int)(q.xg[1] - q.xg[0]) == r.a - 1 && (int)(q.yg[1] - q.yg[0]) == r.b - 1 &&
            (long long)r.a * r.b >= 2;
  return r;
}

template <typename P>
int run_levels(MgWork &w, const P *f, const P *g, int W, int H, const double *mu_g,
               const int gridx_in[2], const int gridy_in[2], int winsize, bool qfactors,
               MgData &out, cudaStream_t st) {
  using S = typename MgT<P>::S;
  using G = typename MgT<P>::G;
  const long long W1 = W + 1, plane = W1 * (H + 1);
  int rc;
  auto t_last = std::chrono::steady_clock::now();
  auto lap = [&](int slot) {
    const auto now = std::chrono::steady_clock::now();
    out.t_ms[slot] += std::chrono::duration<double, std::milli>(now - t_last).count();
    t_last = now;
  };
  // summed-area tables
  const int nch = (H + kSatChunk - 1) / kSatChunk;
  if ((rc = w.sat.ensure(sizeof(S) * 4 * plane))) return rc;
  if ((rc = w.tot.ensure(sizeof(S) * 4 * (size_t)nch * W))) return rc;
  S *sat = w.sat.as<S>();
  const unsigned cols = (unsigned)((W + 127) / 128);
  k_sat_chunks<P><<<dim3(cols, nch), 128, 0, st>>>(f, g, W, H, w.tot.as<S>());
  k_sat_above<S><<<dim3(cols, 4), 128, 0, st>>>(w.tot.as<S>(), W, nch);
  k_sat_fill<P><<<dim3(nch, 4), kSatThreads, 0, st>>>(f, g, W, H, w.tot.as<S>(), sat);
  ALDIC_CUDA(cudaGetLastError());

  // ---- level 1: whole ROI (funIntegerSearchMg.m:9-35)
  const double bg = (double)(1 + mround(0.75 * winsize));
  int gx[2] = {gridx_in[0], gridx_in[1]}, gy[2] = {gridy_in[0], gridy_in[1]};
  if (gx[0] < bg) gx[0] = (int)bg;
  if (gy[0] < bg) gy[0] = (int)bg;
  if (gx[1] > W - bg) gx[1] = W - (int)bg;
  if (gy[1] > H - bg) gy[1] = H - (int)bg;
  const int a = gx[1] - gx[0] + 1, b = gy[1] - gy[0] + 1;
  ALDIC_CHECK(a >= 2 && b >= 2, E_ARG, "multigrid search: the ROI is empty after the border trim");
  int P1 = 1, P2 = 1, l1 = 0, l2 = 0;
  while (P1 < 2 * a - 1) { P1 <<= 1; l1++; }
  while (P2 < 2 * b - 1) { P2 <<= 1; l2++; }
  ALDIC_CHECK(P1 <= kMaxFFT && P2 <= kMaxFFT, E_ARG,
              "multigrid search: the ROI is wider than 4096 px");
  if (P1 < 2) { P1 = 2; l1 = 1; }
  if (P2 < 2) { P2 = 2; l2 = 1; }
  // the second plane also holds P2 rows of P1 / 2 + 8
  const size_t zn = (size_t)P1 * P2 + 8 * (size_t)P2;
  if ((rc = w.fft.ensure(sizeof(double2) * 2 * zn))) return rc;
  if ((rc = w.tw.ensure(sizeof(double2) * (size_t)(P1 + P2)))) return rc;
  double2 *Z0 = w.fft.as<double2>(), *Z1 = Z0 + zn;
  double2 *tw1 = w.tw.as<double2>(), *tw2 = tw1 + P1;
  k_fft_twiddle<<<(P1 + 255) / 256, 256, 0, st>>>(tw1, P1, l1);
  k_fft_twiddle<<<(P2 + 255) / 256, 256, 0, st>>>(tw2, P2, l2);
  const size_t sm1 = fft_smem(P1), sm2 = fft_smem(P2);
  const int th1 = fft_threads(P1), th2 = fft_threads(P2);
  ALDIC_CUDA(cudaFuncSetAttribute(k_fft_pack_rows<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm1));
  ALDIC_CUDA(cudaFuncSetAttribute(k_fft_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2));
  ALDIC_CUDA(cudaFuncSetAttribute(k_fft_spectrum, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2));
  ALDIC_CUDA(cudaFuncSetAttribute(k_fft_ncc<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm1));
  L1Args<S> L1;
  L1.sat = sat;
  L1.plane = plane;
  L1.W1 = (int)W1;
  L1.gx0 = gx[0] - 1;
  L1.gy0 = gy[0] - 1;
  L1.a = a;
  L1.b = b;
  L1.mn = (long long)a * b;
  L1.c = (double *)Z0;  // free by then
  L1.P1 = P1;
  L1.inv = 1.0 / ((double)P1 * (double)P2);
  L1.mu = mu_g;
  const double most = sizeof(P) == 1 ? 255.0 : 65535.0;
  L1.narrow = (double)L1.mn * (double)L1.mn * most * most < 9e18;
  const int np = (2 * b - 1 + 1) / 2, half = P1 / 2 + 1, ldc = P1 / 2 + 8;
  if ((rc = w.part.ensure((sizeof(double) + sizeof(long long)) * np + 64))) return rc;
  double *pv = w.part.as<double>();
  long long *pi = (long long *)(pv + np);
  double *peak = (double *)(pi + np);
  const dim3 tb(32, 8);
  k_fft_pack_rows<P><<<b, th1, sm1, st>>>(f, g, W, H, gx[0], gy[0], a, b, sat, mu_g, Z0, P1, l1, tw1);  // [y][kx]
  k_transpose_c<<<dim3((P1 + 31) / 32, (b + 31) / 32), tb, 0, st>>>(Z0, Z1, b, P1, P1, P2);
  k_fft_cols<<<P1, th2, sm2, st>>>(Z1, P2, l2, tw2, b);                                                 // [kx][ky]
  k_fft_spectrum<<<half, th2, sm2, st>>>(Z1, Z0, P1, P2, l2, tw2);                                      // [kx][oy]
  k_transpose_c<<<dim3((P2 + 31) / 32, (half + 31) / 32), tb, 0, st>>>(Z0, Z1, half, P2, P2, ldc);
  k_fft_ncc<S><<<np, th1, sm1, st>>>(Z1, ldc, P2, L1, l1, tw1, pv, pi);                                 // [oy][ox]
  k_mg_l1_peak<S><<<1, 32, 0, st>>>(L1, pv, pi, np, peak);
  ALDIC_CUDA(cudaGetLastError());
  double pk3[4];
  ALDIC_CUDA(cudaMemcpyAsync(pk3, peak, sizeof(pk3), cudaMemcpyDeviceToHost, st));
  ALDIC_CUDA(cudaStreamSynchronize(st));
  ALDIC_CHECK(pk3[3] == 0.0, E_ARG, "multigrid search: the ROI of the reference image is constant");
  const double ut = pk3[0] - a, vt = pk3[1] - b;
  out.l1_u = ut;
  out.l1_v = vt;
  out.l1_cc = pk3[2];
  lap(0);

  // ---- shift the g ROI, clamp, even widths (:23-48)
  Region r0;
  r0.xf[0] = gx[0]; r0.xf[1] = gx[1]; r0.yf[0] = gy[0]; r0.yf[1] = gy[1];
  r0.xg[0] = gx[0] + mceil(ut); r0.xg[1] = gx[1] + mceil(ut);
  r0.yg[0] = gy[0] + mceil(vt); r0.yg[1] = gy[1] + mceil(vt);
  clamp_region(r0, bg, W, H);
  make_even(r0);
  std::vector<Region> cur{r0};
  std::vector<double> ucur{mceil(ut)}, vcur{mceil(vt)};
  double wx = r0.xf[1] - r0.xf[0], wy = r0.yf[1] - r0.yf[0];
  double ratio = wx / wy;
  const double wsz = winsize;
  int levels = 1;
  for (;;) {
    // ---- split (:58-147)
    std::vector<Region> nw;
    std::vector<double> un, vn;
    const int mode = ratio > 2 ? 0 : (ratio < 0.5 ? 1 : 2);
    if (mode == 0) wx /= 2; else if (mode == 1) wy /= 2; else { wx /= 2; wy /= 2; }
    const int rep = mode == 2 ? 4 : 2;
    nw.reserve(cur.size() * rep);
    for (size_t t = 0; t < cur.size(); ++t) {
      const Region &q = cur[t];
      const bool sx = q.xf[1] - q.xf[0] > wsz, sy = q.yf[1] - q.yf[0] > wsz;
      const double mxf = 0.5 * (q.xf[0] + q.xf[1]), mxg = 0.5 * (q.xg[0] + q.xg[1]);
      const double myf = 0.5 * (q.yf[0] + q.yf[1]), myg = 0.5 * (q.yg[0] + q.yg[1]);
      if (mode == 0 && sx) {
        Region lo = q, hi = q;
        lo.xf[1] = mxf; lo.xg[1] = mxg; hi.xf[0] = mxf; hi.xg[0] = mxg;
        nw.push_back(lo); nw.push_back(hi);
      } else if (mode == 1 && sy) {
        Region lo = q, hi = q;
        lo.yf[1] = myf; lo.yg[1] = myg; hi.yf[0] = myf; hi.yg[0] = myg;
        nw.push_back(lo); nw.push_back(hi);
      } else if (mode == 2 && sx && sy) {
        for (int jy = 0; jy < 2; ++jy)
          for (int ix = 0; ix < 2; ++ix) {
            Region s = q;
            if (ix == 0) { s.xf[1] = mxf; s.xg[1] = mxg; } else { s.xf[0] = mxf; s.xg[0] = mxg; }
            if (jy == 0) { s.yf[1] = myf; s.yg[1] = myg; } else { s.yf[0] = myf; s.yg[0] = myg; }
            nw.push_back(s);
          }
      } else {
        for (int k = 0; k < rep; ++k) nw.push_back(q);
      }
      for (int k = 0; k < rep; ++k) { un.push_back(ucur[t]); vn.push_back(vcur[t]); }
    }
    const bool last = wx < wsz && wy < wsz;
    levels++;
    const int n = (int)nw.size();
    ALDIC_CHECK(n <= (1 << 24), E_ARG, "multigrid search: too many regions");
    // ---- correlate every region (:148-172)
    std::vector<MgReg> hr(n);
    int amax = 0, bmax = 0;
    for (int t = 0; t < n; ++t) {
      hr[t] = describe(nw[t], W, H);
      if (hr[t].valid) { amax = std::max(amax, hr[t].a); bmax = std::max(bmax, hr[t].b); }
    }
    if ((rc = w.regs.ensure(sizeof(MgReg) * n))) return rc;
    if ((rc = w.res.ensure(sizeof(double) * 8 * n))) return rc;
    ALDIC_CUDA(cudaMemcpyAsync(w.regs.p, hr.data(), sizeof(MgReg) * n, cudaMemcpyHostToDevice, st));
    MgReg *dr = w.regs.as<MgReg>();
    double *dres = w.res.as<double>();
    if (last && qfactors) {
      ALDIC_CHECK(amax <= kMaxFinal && bmax <= kMaxFinal, E_ARG,
                  "multigrid search: last-level regions larger than 80 px");
      const int dwm = amax + 10, dhm = bmax + 10;
      const size_t sm = sizeof(double) * (size_t)(amax + dwm - 1) * (bmax + dhm - 1) +
                        sizeof(typename MgT<P>::V) *
                            ((size_t)(amax + 8) * bmax + (size_t)dhm * (dwm + 2 * kStrip + 8)) + 16;
      ALDIC_CHECK(sm <= 200 * 1024, E_ARG, "multigrid search: last-level map too large for shared memory");
      size_t use = sm;
      if constexpr (MgT<P>::integer) {  // operands as packed words: less than that
        const FullWords fw(amax);
        use = sizeof(double) * (size_t)(amax + dwm - 1) * (bmax + dhm - 1) +
              sizeof(P) * sizeof(uint32_t) * ((size_t)bmax * fw.tw + (size_t)dhm * fw.dw) + 16;
      }
      ALDIC_CUDA(cudaFuncSetAttribute(k_mg_full<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)use));
      if (amax > 0) k_mg_full<P><<<n, 256, use, st>>>(f, g, W, H, dr, sat, mu_g, dres);
    } else {
      if ((rc = w.acc.ensure(sizeof(G) * (size_t)kCrop * n))) return rc;
      ALDIC_CUDA(cudaMemsetAsync(w.acc.p, 0, sizeof(G) * (size_t)kCrop * n, st));
      if (amax > 0) {
        constexpr bool kInt = MgT<P>::integer;
        constexpr int kTile = kInt ? kTileI : CropCfg<P>::TILE, kRows = kInt ? kBandI : kBand;
        const dim3 grid(n, (bmax + kRows - 1) / kRows, (amax + kTile - 1) / kTile);
        ALDIC_CHECK(grid.y <= 65535 && grid.z <= 65535, E_ARG, "multigrid search: region too large");
        if constexpr (kInt)
          k_mg_crop_int<P><<<grid, 224, 0, st>>>(f, g, W, dr, w.acc.as<G>());
        else
          k_mg_crop<P><<<grid, 224, 0, st>>>(f, g, W, dr, w.acc.as<G>());
        k_mg_crop_peak<P><<<n, 192, 0, st>>>(dr, W, H, sat, w.acc.as<G>(), mu_g, dres);
      }
    }
    ALDIC_CUDA(cudaGetLastError());
    std::vector<double> hres((size_t)8 * n, 0.0);
    ALDIC_CUDA(cudaMemcpyAsync(hres.data(), dres, sizeof(double) * 8 * n, cudaMemcpyDeviceToHost, st));
    ALDIC_CUDA(cudaStreamSynchronize(st));
    lap(last ? 2 : 1);
    std::vector<double> phi(n, 0.0), q1(n, NAN), q2(n, NAN);
    int failed = 0;
    for (int t = 0; t < n; ++t) {
      const double *o = &hres[(size_t)8 * t];
      if (hr[t].valid && o[3] == 1.0) {
        un[t] += o[0];
        vn[t] += o[1];
        phi[t] = o[2];
        if (last && qfactors) { q1[t] = o[4]; q2[t] = o[5]; }
      } else {
        un[t] = vn[t] = NAN;
        phi[t] = 0.0;
        failed++;
      }
    }
    if (last) {
      // :173-178: q-factors normalised over the regions (NaN ignored)
      for (std::vector<double> *q : {&q1, &q2}) {
        double mn = INFINITY, mx = -INFINITY;
        for (double v : *q) if (!std::isnan(v) && v < mn) mn = v;
        for (double v : *q) if (!std::isnan(v) && v - mn > mx) mx = v - mn;
        for (double &v : *q) v = (v - mn) / mx;
      }
      out.tx.resize(n); out.ty.resize(n);
      for (int t = 0; t < n; ++t) {
        out.tx[t] = 0.5 * (nw[t].xf[0] + nw[t].xf[1]);
        out.ty[t] = 0.5 * (nw[t].yf[0] + nw[t].yf[1]);
      }
      out.u = un; out.v = vn; out.phi = phi; out.q1 = q1; out.q2 = q2;
      out.gridx[0] = gx[0]; out.gridx[1] = gx[1];
      out.gridy[0] = gy[0]; out.gridy[1] = gy[1];
      out.levels = levels;
      out.failed = failed;
      return OK;
    }
    // ---- next level's g regions (:179-209)
    for (int t = 0; t < n; ++t) {
      Region &q = nw[t];
      const double cu = mceil(un[t]), cv = mceil(vn[t]);
      q.xg[0] = q.xf[0] + cu; q.xg[1] = q.xf[1] + cu;
      q.yg[0] = q.yf[0] + cv; q.yg[1] = q.yf[1] + cv;
      clamp_region(q, bg, W, H);
    }
    for (auto &q : nw) make_even(q);
    ratio = wx / wy;
    cur.swap(nw);
    ucur.resize(n); vcur.resize(n);
    for (int t = 0; t < n; ++t) { ucur[t] = mceil(un[t]); vcur[t] = mceil(vn[t]); }
  }
}

}  // namespace

int search_mg_levels(MgWork &w, const void *f, const void *g, int dtype, int W, int H,
                     const double *mu_g, const int gridx[2], const int gridy[2], int winsize,
                     bool qfactors, MgData &out, cudaStream_t st) {
  ALDIC_CHECK(winsize > 0, E_ARG, "multigrid search: winsize must be positive");
  switch (dtype) {
    case 0: return run_levels<uint8_t>(w, (const uint8_t *)f, (const uint8_t *)g, W, H, mu_g, gridx, gridy, winsize, qfactors, out, st);
    case 1: return run_levels<uint16_t>(w, (const uint16_t *)f, (const uint16_t *)g, W, H, mu_g, gridx, gridy, winsize, qfactors, out, st);
    case 2: return run_levels<float>(w, (const float *)f, (const float *)g, W, H, mu_g, gridx, gridy, winsize, qfactors, out, st);
    default: return run_levels<double>(w, (const double *)f, (const double *)g, W, H, mu_g, gridx, gridy, winsize, qfactors, out, st);
  }
}

// funIntegerSearchMg.m:210-244: node grid from the borders of the extreme
// regions; returns false when the grid is empty.
bool search_mg_grid(const MgData &d, int winsize, int step, int W, int H, MgGrid &grid) {
  const int n = (int)d.tx.size();
  if (n == 0) return false;
  int ix1 = 0, ix2 = 0, iy1 = 0, iy2 = 0;
  for (int t = 1; t < n; ++t) {
    if (d.tx[t] < d.tx[ix1]) ix1 = t;
    if (d.tx[t] > d.tx[ix2]) ix2 = t;
    if (d.ty[t] < d.ty[iy1]) iy1 = t;
    if (d.ty[t] > d.ty[iy2]) iy2 = t;
  }
  const double bx1 = mceil(1 + 1.25 * winsize + d.u[ix1]), bx2 = mceil(1 + 1.25 * winsize + d.u[ix2]);
  const double by1 = mceil(1 + 1.25 * winsize + d.v[iy1]), by2 = mceil(1 + 1.25 * winsize + d.v[iy2]);
  double gx0 = d.gridx[0], gx1 = d.gridx[1], gy0 = d.gridy[0], gy1 = d.gridy[1];
  if (gx0 < bx1) gx0 = bx1;
  if (gy0 < by1) gy0 = by1;
  if (gx1 > W - bx2 + 1) gx1 = W - bx2 + 1;
  if (gy1 > H - by2 + 1) gy1 = H - by2 + 1;
  grid.x0 = gx0;
  grid.y0 = gy0;
  grid.nx = gx1 >= gx0 ? (int)std::floor((gx1 - gx0) / step) + 1 : 0;
  grid.ny = gy1 >= gy0 ? (int)std::floor((gy1 - gy0) / step) + 1 : 0;
  grid.step = step;
  return grid.nx >= 2 && grid.ny >= 2;
}

// gridfit(x, y, z, xList, yList, 'regularizer', 'springs') of u, v, Phi and
// the two q-factors (gridfit.m:328-596 with smoothness 1, triangle
// interpolation, autoscale on uniform nodes): the normal equations
// (A'A + (NA/NR)^2 Areg'Areg) z = A'data.  The springs part is the gridfit
// stencil of the grid PCG; A'A and A'z are gathered per node from the points
// of its four cells (k_mg_ata, points sorted by cell on the host: fixed
// order, no atomics); one solve per set of fields sharing a NaN pattern.
int search_mg_fit(GridWork &gw, MgWork &w, MgData &d, const MgGrid &grid, int nfields,
                  double *out, cudaStream_t st) {
  const auto t0 = std::chrono::steady_clock::now();
  struct Lap {
    MgData &d;
    std::chrono::steady_clock::time_point t0;
    ~Lap() {
      d.t_ms[3] += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
  } lap{d, t0};
  const int nx = grid.nx, ny = grid.ny;
  const long long ng = (long long)nx * ny;
  const double h = grid.step;
  const double xmax = grid.x0 + (nx - 1) * h, ymax = grid.y0 + (ny - 1) * h;
  const int n = (int)d.tx.size();
  // data strictly inside the grid (funIntegerSearchMg.m:232-234)
  std::vector<int> sel;
  for (int t = 0; t < n; ++t)
    if (d.tx[t] > grid.x0 && d.tx[t] < xmax && d.ty[t] > grid.y0 && d.ty[t] < ymax) sel.push_back(t);
  const std::vector<double> *fields[5] = {&d.u, &d.v, &d.phi, &d.q1, &d.q2};
  const int nf = std::min(std::max(nfields, 1), 5);
  std::vector<int> group(nf, -1);
  std::vector<std::vector<int>> members;
  for (int fi = 0; fi < nf; ++fi) {
    if (group[fi] >= 0) continue;
    group[fi] = (int)members.size();
    members.push_back({fi});
    for (int fj = fi + 1; fj < nf; ++fj) {
      if (group[fj] >= 0) continue;
      bool same = true;
      for (int t : sel)
        if (std::isnan((*fields[fi])[t]) != std::isnan((*fields[fj])[t])) { same = false; break; }
      if (same) { group[fj] = group[fi]; members.back().push_back(fj); }
    }
  }
  double NR = 0;  // norm(Areg, 1)
  const double sq2 = 1.0 / std::sqrt(2.0);
  for (int j = 0; j < std::min(ny, 3); ++j)
    for (int i = 0; i < std::min(nx, 3); ++i) {
      double sreg = (i > 0) + (i < nx - 1) + (j > 0) + (j < ny - 1);
      sreg += sq2 * ((i > 0 && j > 0) + (i < nx - 1 && j > 0) + (i > 0 && j < ny - 1) +
                     (i < nx - 1 && j < ny - 1));
      NR = std::max(NR, sreg);
    }
  const long long ncell = (long long)(nx - 1) * (ny - 1);
  int rc;
  for (const auto &mem : members) {
    const int nr = (int)mem.size();
    std::vector<int> pts;
    for (int t : sel)
      if (!std::isnan((*fields[mem[0]])[t])) pts.push_back(t);
    const long long np = (long long)pts.size();
    ALDIC_CHECK(np >= 3, E_ARG, "multigrid search: gridfit has fewer than 3 data points");
    // histc cells (the last node belongs to the last cell), counting sort by
    // cell (stable: region order inside a cell), column sums of A for NA
    std::vector<int> cell(np), start(ncell + 1, 0);
    std::vector<double> colsum(ng, 0.0);
    for (long long q = 0; q < np; ++q) {
      const double x = d.tx[pts[q]], y = d.ty[pts[q]];
      int ix = (int)std::floor((x - grid.x0) / h), iy = (int)std::floor((y - grid.y0) / h);
      ix = std::min(std::max(ix, 0), nx - 2);
      iy = std::min(std::max(iy, 0), ny - 2);
      cell[q] = iy * (nx - 1) + ix;
      start[cell[q] + 1]++;
      const double tx = std::min(1.0, std::max(0.0, (x - (grid.x0 + ix * h)) / h));
      const double ty = std::min(1.0, std::max(0.0, (y - (grid.y0 + iy * h)) / h));
      const double t1 = std::min(tx, ty), t2 = std::max(tx, ty);
      const long long k0 = (long long)iy * nx + ix;
      colsum[k0] += 1 - t2;
      colsum[k0 + nx + 1] += t1;
      colsum[tx > ty ? k0 + 1 : k0 + nx] += t2 - t1;
    }
    double NA = 0;
    for (double c : colsum) NA = std::max(NA, c);
    for (long long c = 0; c < ncell; ++c) start[c + 1] += start[c];
    std::vector<int> fill(start.begin(), start.end() - 1);
    std::vector<double> hp((size_t)(2 + nr) * np);  // x | y | values (point-major)
    for (long long q = 0; q < np; ++q) {
      const long long o = fill[cell[q]]++;
      hp[o] = d.tx[pts[q]];
      hp[np + o] = d.ty[pts[q]];
      for (int m = 0; m < nr; ++m) hp[2 * np + o * nr + m] = (*fields[mem[m]])[pts[q]];
    }
    const size_t bytes = sizeof(int) * (ncell + 1) + sizeof(double) * hp.size() + sizeof(double) * 9 * ng + 64;
    if ((rc = w.csr.ensure(bytes))) return rc;
    int *dstart = w.csr.as<int>();
    double *dp = (double *)(((uintptr_t)(dstart + ncell + 1) + 15) & ~(uintptr_t)15);
    double *data = dp + hp.size();
    ALDIC_CUDA(cudaMemcpyAsync(dstart, start.data(), sizeof(int) * (ncell + 1), cudaMemcpyHostToDevice, st));
    ALDIC_CUDA(cudaMemcpyAsync(dp, hp.data(), sizeof(double) * hp.size(), cudaMemcpyHostToDevice, st));
    k_mg_ata<<<(unsigned)std::min<long long>((ng + 255) / 256, 148 * 16), 256, 0, st>>>(
        nx, ny, grid.x0, grid.y0, h, dstart, dp, dp + np, dp + 2 * np, nr, data, gw.b);
    ALDIC_CUDA(cudaGetLastError());
    ALDIC_CUDA(cudaMemsetAsync(gw.x, 0, sizeof(double) * nr * ng, st));
    ALDIC_CUDA(cudaMemsetAsync(gw.mask, 1, (size_t)nr * ng, st));
    const double lam2 = (NA / NR) * (NA / NR);
    bool ran = false;
    if ((rc = cluster_ata(gw, data, nx, ny, nr, lam2, 1e-13, 20000, st, &ran))) return rc;
    if (!ran && (rc = grid_pcg(gw, OP_GRIDFIT, nx, ny, nr, 0.0, 0.0, 1.0, lam2, 1e-13, 20000, st, nullptr,
                               nullptr, data)))
      return rc;
    for (int m = 0; m < nr; ++m)
      ALDIC_CUDA(cudaMemcpyAsync(out + (size_t)mem[m] * ng, gw.x + (size_t)m * ng, sizeof(double) * ng,
                                 cudaMemcpyDeviceToDevice, st));
    ALDIC_CUDA(cudaStreamSynchronize(st));  // host vectors above are reused next group
  }
  return OK;
}

}  // namespace aldic
