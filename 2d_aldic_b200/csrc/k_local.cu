// k_local.cu -- the node-grid systems whose solution at a node depends on its
// neighbourhood only, solved tile by tile in shared memory instead of by a
// grid-wide iteration:
//   gridfit 'springs' of data on the nodes (gridfit.m:523-596)   k_fit_tile
//   spring inpainting of scattered unknown nodes (inpaint_nans)  k_fill_tile
// Both leave the field-major work vectors (b, x, mask) as k_pcg expects them
// and a gate word: 0 the result is complete, 1 k_pcg continues from x, 2 (not
// finite: infinities or overflow in the data) k_pcg starts over from the data.
// k_pcg is launched behind them and returns at once on 0, so the pair can be
// captured in a graph without a host decision.
#include "aldic_internal.cuh"
#include "kernels.cuh"

namespace aldic {

namespace {

// ------------------------------------------------------------------ gridfit
// A = W + lam2 L, W = 1 at nodes with data, L the graph Laplacian of the
// axial springs and half that of the diagonal ones; lam2 = 1 / norm1^2 =
// 0.0215 on any grid with an interior.  Scaled by its diagonal D, A is the
// identity minus a matrix whose row sums are at most 6 lam2 / (1 + 6 lam2) =
// 0.114 at nodes with data, so the eigenvalues of D^-1 A lie in 1 +- 0.114
// there, and a Chebyshev iteration on [1 - kFitRho, 1 + kFitRho] gains
// (1 - sqrt(1 - rho^2)) / rho = 0.077 a step: kFitSteps of them reduce the
// error by 1e-13 (a single node without data, within 1 +- 0.2, by 1e-9 of
// its own start error).  A step needs the 8 neighbours only, so a CTA that
// loads a halo of kFitHalo > kFitSteps + 1 nodes computes the result of the
// whole grid's iteration on its tile with no exchange: one launch instead of
// a grid barrier an iteration.  The tiles also form the exact residual of the
// result; where |r| > rtol |b| (clusters of nodes without data), k_pcg goes
// on from it, with the same stopping test as ever.
//
// Shape: 64 x 64 region, 32 x 32 tile, 1024 threads, a thread marching 4 rows
// of a column (x, d, b, 1/D in registers; 14 shared loads for 4 nodes).  The
// launch is bound by latency: a CTA an SM, and two fields of 243 x 243 are 128
// CTAs, so more threads with fewer rows won (18.6 us under ncu with cold
// caches, against 22 for 512 threads with 8 rows).  k_pcg alone took 63 us;
// behind the tiles, with nothing to do, it takes 2.6.
constexpr int kFitTile = 32, kFitHalo = 16, kFitReg = kFitTile + 2 * kFitHalo, kFitPitch = kFitReg + 2;
constexpr int kFitRows = 4, kFitThreads = kFitReg * kFitReg / kFitRows;
constexpr int kFitSteps = 12;
constexpr double kFitRho = 0.15;
static_assert(kFitHalo >= kFitSteps + 2, "the residual and the convolution read one more ring");

struct FitArgs {
  FieldMap in, guess, out;       // guess.p[0] == null: nodes without data start from 0
  const int *bad;                // status per node (null: none): < 0 or > 99 has no data
  double *b, *x, *part;
  unsigned char *mask;
  int *gate;                     // {gate, ticket}
  int *iters;                    // most iterations of a solve so far
  unsigned int *bar;             // k_pcg's grid barrier words, reset here
  double lam2, rtol;
  double ca[kFitSteps], cb[kFitSteps];  // d <- ca d + cb D^-1 r
  // the diagonal and its inverse by data / no data and the number of
  // neighbours along x and y
  double dg[2][3][3], di[2][3][3];
  int M, N, nf;
};

template <bool CONV>
__global__ void __launch_bounds__(kFitThreads, 1) k_fit_tile(const __grid_constant__ FitArgs A) {
  extern __shared__ double fit_sh[];
  double *const buf0 = fit_sh, *const buf1 = fit_sh + kFitPitch * kFitPitch;
  __shared__ double red[kFitThreads / 32][2];
  __shared__ int s_last;
  const int M = A.M, N = A.N, f = blockIdx.y;
  const long long n = (long long)M * N;
  const int tx = (M + kFitTile - 1) / kFitTile, ty0 = (int)blockIdx.x / tx, tx0 = (int)blockIdx.x - ty0 * tx;
  const int cx = threadIdx.x & (kFitReg - 1), r0 = (threadIdx.x / kFitReg) * kFitRows;
  const int gi = tx0 * kFitTile - kFitHalo + cx;
  const int gj0 = ty0 * kFitTile - kFitHalo + r0;
  const bool col_in = gi >= 0 && gi < M;
  // the rim around the region reads as no node
  for (int k = threadIdx.x; k < 8 * kFitPitch; k += kFitThreads) {
    double *buf = k & 1 ? buf1 : buf0;
    const int e = (k >> 1) & 3, t = k >> 3;
    buf[e == 0 ? t : e == 1 ? (kFitPitch - 1) * kFitPitch + t
                            : t * kFitPitch + (e == 2 ? 0 : kFitPitch - 1)] = 0.0;
  }
  const double *const src = A.in.p[f];
  const long long ss = A.in.stride[f];
  const double lam = A.lam2;
  double x[kFitRows], d[kFitRows], b[kFitRows], di[kFitRows];
  unsigned int known = 0;
  const int nxn = (gi > 0) + (gi < M - 1);
#pragma unroll
  for (int q = 0; q < kFitRows; ++q) {
    const int gj = gj0 + q;
    x[q] = d[q] = b[q] = di[q] = 0.0;
    if (col_in && gj >= 0 && gj < N) {
      const long long k = (long long)gj * M + gi;
      const double v = src[k * ss];
      const int st = A.bad ? A.bad[k] : 0;
      const bool ok = !(st < 0 || st > 99) && !isnan(v);
      known |= (ok ? 1u : 0u) << q;
      b[q] = ok ? v : 0.0;
      x[q] = ok ? v : (A.guess.p[0] ? A.guess.p[f][k * A.guess.stride[f]] : 0.0);
      const int nyn = (gj > 0) + (gj < N - 1);
      di[q] = A.di[ok][nxn][nyn];
    }
  }
  __syncthreads();
  const int at = (r0 + 1) * kFitPitch + cx + 1;
#pragma unroll
  for (int q = 0; q < kFitRows; ++q) buf0[at + q * kFitPitch] = x[q];
  __syncthreads();
  // side sums left + right of rows -1 .. kFitRows, and the centre values
  // above and below the strip, of the current iterate
  double sl[kFitRows + 2], top, bot;
  auto gather = [&](const double *cur) {
#pragma unroll
    for (int q = 0; q < kFitRows + 2; ++q) {
      const double *p = cur + at + (q - 1) * kFitPitch;
      sl[q] = p[-1] + p[1];
    }
    top = cur[at - kFitPitch];
    bot = cur[at + kFitRows * kFitPitch];
  };
#pragma unroll 1
  for (int s = 0; s < kFitSteps; ++s) {
    const double *cur = (s & 1) ? buf1 : buf0;
    double *nxt = (s & 1) ? buf0 : buf1;
    gather(cur);
    const double ca = A.ca[s], cb = A.cb[s];
    double up = top;
#pragma unroll
    for (int q = 0; q < kFitRows; ++q) {
      const double dn = q + 1 < kFitRows ? x[q + 1] : bot;
      const double nb = (sl[q + 1] + (up + dn)) + 0.5 * (sl[q] + sl[q + 2]);
      up = x[q];
      d[q] = ca * d[q] + cb * (di[q] * fma(lam, nb, b[q]) - x[q]);
      // a node outside the grid keeps di = 0 and x = 0: d = -cb x = 0
      x[q] += d[q];
      nxt[at + q * kFitPitch] = x[q];
    }
    __syncthreads();
  }
  gather((kFitSteps & 1) ? buf1 : buf0);
  double rr = 0.0, bb = 0.0;
  const bool mine = cx >= kFitHalo && cx < kFitHalo + kFitTile && col_in && r0 >= kFitHalo &&
                    r0 < kFitHalo + kFitTile;
  if (mine) {
    const double e1 = 0.1353352832366127, e2 = 0.01831563888873418;  // exp(-2), exp(-4)
#pragma unroll
    for (int q = 0; q < kFitRows; ++q) {
      const int gj = gj0 + q;
      if (gj >= N) continue;
      const double up = q > 0 ? x[q - 1] : top, dn = q + 1 < kFitRows ? x[q + 1] : bot;
      const double ax = sl[q + 1] + (up + dn), dg = sl[q] + sl[q + 2];
      const int nyn = (gj > 0) + (gj < N - 1);
      const double r = fma(lam, ax + 0.5 * dg, b[q]) - x[q] * A.dg[(known >> q) & 1u][nxn][nyn];
      rr += r * r;
      bb += b[q] * b[q];
      const long long k = (long long)gj * M + gi;
      const long long o = f * n + k;
      double v = x[q];
      if (CONV)  // the 3 x 3 Gaussian of nanconv, normalised over the nodes there are
        v = (x[q] + e1 * ax + e2 * dg) / (1.0 + e1 * (nxn + nyn) + e2 * (nxn * nyn));
      A.b[o] = b[q];
      A.x[o] = x[q];
      A.mask[o] = (known >> q) & 1u;
      A.out.p[f][k * A.out.stride[f]] = v;
    }
  }
  rr = warp_sum(rr);
  bb = warp_sum(bb);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    red[wid][0] = rr;
    red[wid][1] = bb;
  }
  __syncthreads();
  const int tiles = gridDim.x, t = blockIdx.x;
  if (threadIdx.x == 0) {
    double sr = 0.0, sb = 0.0;
    for (int w = 0; w < kFitThreads / 32; ++w) {
      sr += red[w][0];
      sb += red[w][1];
    }
    double *p = A.part + 2 * ((long long)f * tiles + t);
    p[0] = sr;
    p[1] = sb;
    __threadfence();
    s_last = atomicAdd(&A.gate[1], 1) == tiles * (int)gridDim.y - 1;
  }
  __syncthreads();
  if (!s_last) return;
  // the last CTA: the residual of every field, in tile order
  __threadfence();
  int need = 0;
  if (wid < A.nf) {
    double sr = 0.0, sb = 0.0;
    for (int q = lane; q < tiles; q += 32) {
      const double *p = A.part + 2 * ((long long)wid * tiles + q);
      sr += __ldcg(p);
      sb += __ldcg(p + 1);
    }
    sr = warp_sum(sr);
    sb = warp_sum(sb);
    if (!(isfinite(sr) && isfinite(sb))) need = 2;
    else if (sr > A.rtol * A.rtol * sb) need = 1;
  }
  const int any2 = __syncthreads_or(need == 2), any1 = __syncthreads_or(need == 1);
  if (threadIdx.x == 0) {
    atomicMax(A.iters, kFitSteps);
    A.gate[0] = any2 ? 2 : (any1 ? 1 : 0);
    A.gate[1] = 0;
    A.bar[0] = A.bar[1] = 0;
  }
}

// ------------------------------------------------------------------ inpainting
// Unknown entries, their right-hand sides (sums of known neighbours) and start
// values (their mean) of nf fields; resets the gate.
struct FillArgs {
  FieldMap vals;
  const unsigned char *bad;  // flag per node (null: none), besides NaN entries
  double *b, *x;
  unsigned char *mask;
  int *gate;
  int *iters;  // most iterations of a solve so far
  unsigned int *bar;
  double rtol;
  int M, N, nf;
};

__global__ void k_fill_load(const __grid_constant__ FillArgs A) {
  const int M = A.M, N = A.N, f = blockIdx.y;
  const long long n = (long long)M * N;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    A.gate[0] = A.gate[1] = 0;
    A.bar[0] = A.bar[1] = 0;
  }
  const double *vals = A.vals.p[f];
  const long long s = A.vals.stride[f];
  auto known = [&](long long q) { return !(A.bad && A.bad[q]) && !isnan(vals[q * s]); };
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x) {
    const bool kn = known(k);
    double bv = 0.0;
    int kc = 0;
    if (kn) {
      bv = vals[k * s];
    } else {
      const int i = (int)(k % M), j = (int)(k / M);
      if (i > 0 && known(k - 1)) { bv += vals[(k - 1) * s]; ++kc; }
      if (i < M - 1 && known(k + 1)) { bv += vals[(k + 1) * s]; ++kc; }
      if (j > 0 && known(k - M)) { bv += vals[(k - M) * s]; ++kc; }
      if (j < N - 1 && known(k + M)) { bv += vals[(k + M) * s]; ++kc; }
    }
    A.mask[f * n + k] = !kn;
    A.b[f * n + k] = bv;
    A.x[f * n + k] = kn ? bv : (kc > 0 ? bv / kc : 0.0);
  }
}

// The unknown nodes fall into 4-connected clusters that only know their rim of
// known nodes, so each cluster is a system of its own.  A CTA takes a 32 x 32
// tile with a halo of 24, keeps the unknown nodes connected to one in its tile
// (bit-parallel flood fill by one warp) and solves them by conjugate gradients
// in shared memory: the operator is nearly 4 I on the diagonal, so no
// preconditioner, and the two dot products of an iteration share one reduction
// (Chronopoulos and Gear, J. Comput. Appl. Math. 25, 1989).  An iteration costs
// two block barriers instead of a grid barrier.  A cluster that leaves the
// region, more than kFillCap nodes, or an iteration that does not converge set
// the gate and keep their start values for k_pcg.  The refill of LocalICGN's
// six fields (ncu): 146 -> 17 us at 243 x 243 with 0.6 % of the nodes flagged,
// 450 -> 33 us at 43 x 43 with 41 %.
constexpr int kFillTile = 32, kFillHalo = 24, kFillReg = kFillTile + 2 * kFillHalo;
constexpr int kFillPitch = kFillReg + 2, kFillWords = 3, kFillThreads = 256;
constexpr int kFillPer = 8, kFillCap = kFillPer * kFillThreads, kFillMaxit = 4000;
static_assert(kFillReg <= 32 * kFillWords && kFillReg <= 96, "row bits and the flood's three rows a lane");

struct FillShared {
  double r[kFillPitch * kFillPitch];
  double red[2][kFillThreads / 32][3];
  unsigned int unk[kFillReg + 1][kFillWords];   // unknown entries
  unsigned int need[kFillReg + 1][kFillWords];  // those of the tile's clusters
  int base[kFillReg + 1][kFillWords];
  unsigned short list[kFillCap];
  int count;
};

__global__ void __launch_bounds__(kFillThreads, 2) k_fill_tile(const __grid_constant__ FillArgs A) {
  extern __shared__ char fill_raw[];
  FillShared &S = *(FillShared *)fill_raw;
  const int M = A.M, N = A.N, f = blockIdx.y;
  const long long n = (long long)M * N;
  const unsigned char *mask = A.mask + f * n;
  const int tx = (M + kFillTile - 1) / kFillTile, tyq = (int)blockIdx.x / tx;
  const int ti = ((int)blockIdx.x - tyq * tx) * kFillTile, tj = tyq * kFillTile;
  int any = 0;
  for (int q = threadIdx.x; q < kFillTile * kFillTile; q += kFillThreads) {
    const int i = ti + (q & (kFillTile - 1)), j = tj + q / kFillTile;
    if (i < M && j < N) any |= mask[(long long)j * M + i];
  }
  if (!__syncthreads_or(any)) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ox = ti - kFillHalo, oy = tj - kFillHalo;
  for (int q = wid; q <= kFillReg; q += kFillThreads / 32)
#pragma unroll
    for (int w = 0; w < kFillWords; ++w) {
      const int c = 32 * w + lane, i = ox + c, j = oy + q;
      const bool u = q < kFillReg && c < kFillReg && i >= 0 && i < M && j >= 0 && j < N &&
                     mask[(long long)j * M + i];
      const unsigned int bits = __ballot_sync(0xffffffffu, u);
      if (lane == 0) S.unk[q][w] = bits;
    }
  for (int q = threadIdx.x; q < kFillPitch * kFillPitch; q += kFillThreads) S.r[q] = 0.0;
  __syncthreads();
  if (wid == 0) {
    // rows 3 lane .. 3 lane + 2 of the region in this lane
    unsigned int m[3][kFillWords], c[3][kFillWords];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int w = 0; w < kFillWords; ++w) {
        const int q = 3 * lane + a;
        const unsigned int tile = w == 0 ? 0xff000000u : (w == 1 ? 0x00ffffffu : 0u);
        m[a][w] = q <= kFillReg ? S.unk[q][w] : 0u;
        c[a][w] = (q >= kFillHalo && q < kFillHalo + kFillTile) ? m[a][w] & tile : 0u;
      }
    static_assert(kFillHalo == 24 && kFillTile == 32, "the tile's column bits above");
    bool open = false;
    int sweep = 0;
    for (; sweep < kFillReg * kFillReg; ++sweep) {
      unsigned int ch = 0;
#pragma unroll
      for (int w = 0; w < kFillWords; ++w) {
        const unsigned int above = __shfl_up_sync(0xffffffffu, c[2][w], 1);
        const unsigned int below = __shfl_down_sync(0xffffffffu, c[0][w], 1);
        const unsigned int v0 = (c[0][w] | (lane > 0 ? above : 0u) | c[1][w]) & m[0][w];
        const unsigned int v2 = (c[2][w] | c[1][w] | (lane < 31 ? below : 0u)) & m[2][w];
        const unsigned int v1 = (c[1][w] | v0 | v2) & m[1][w];
        ch |= (v0 ^ c[0][w]) | (v1 ^ c[1][w]) | (v2 ^ c[2][w]);
        c[0][w] = v0;
        c[1][w] = v1;
        c[2][w] = v2;
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const unsigned int o0 = c[a][0], o1 = c[a][1], o2 = c[a][2];
        c[a][0] |= ((o0 << 1) | (o0 >> 1) | (o1 << 31)) & m[a][0];
        c[a][1] |= ((o1 << 1) | (o0 >> 31) | (o1 >> 1) | (o2 << 31)) & m[a][1];
        c[a][2] |= ((o2 << 1) | (o1 >> 31) | (o2 >> 1)) & m[a][2];
        ch |= (c[a][0] ^ o0) | (c[a][1] ^ o1) | (c[a][2] ^ o2);
      }
      if (!__any_sync(0xffffffffu, ch != 0)) break;
    }
    // a needed node on the region's edge where the grid goes on
    int cnt = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int q = 3 * lane + a;
      const unsigned int row = c[a][0] | c[a][1] | c[a][2];
      open |= (q == 0 && oy > 0 && row) || (q == kFillReg - 1 && oy + kFillReg < N && row);
      open |= (ox > 0 && (c[a][0] & 1u)) ||
              (ox + kFillReg < M && (c[a][(kFillReg - 1) / 32] >> ((kFillReg - 1) & 31) & 1u));
#pragma unroll
      for (int w = 0; w < kFillWords; ++w) cnt += __popc(c[a][w]);
    }
    int scan = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, scan, o);
      if (lane >= o) scan += v;
    }
    const int total = __shfl_sync(0xffffffffu, scan, 31);
    int pos = scan - cnt;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int w = 0; w < kFillWords; ++w) {
        const int q = 3 * lane + a;
        if (q <= kFillReg) {
          S.need[q][w] = c[a][w];
          S.base[q][w] = pos;
        }
        pos += __popc(c[a][w]);
      }
    if (__any_sync(0xffffffffu, open) || total > kFillCap || sweep >= kFillReg * kFillReg) {
      if (lane == 0) S.count = -1;
    } else if (lane == 0) {
      S.count = total;
    }
  }
  __syncthreads();
  const int cnt = S.count;
  if (cnt < 0) {
    if (threadIdx.x == 0) atomicExch(A.gate, 1);
    return;
  }
  if (threadIdx.x < kFillReg * kFillWords) {
    const int q = threadIdx.x / kFillWords, w = threadIdx.x - q * kFillWords;
    unsigned int bits = S.need[q][w];
    int pos = S.base[q][w];
    while (bits) {
      const int c = 32 * w + __ffs(bits) - 1;
      bits &= bits - 1;
      S.list[pos++] = (unsigned short)((q + 1) * kFillPitch + c + 1);
    }
  }
  __syncthreads();
  double x[kFillPer], r[kFillPer], p[kFillPer], s[kFillPer], w[kFillPer], b[kFillPer];
  int at[kFillPer];
  float deg[kFillPer];
  double bb = 0.0;
#pragma unroll
  for (int q = 0; q < kFillPer; ++q) {
    const int l = threadIdx.x + q * kFillThreads;
    at[q] = 0;
    x[q] = r[q] = p[q] = s[q] = w[q] = b[q] = 0.0;
    deg[q] = 0.f;
    if (l < cnt) {
      at[q] = S.list[l];
      const int rj = at[q] / kFillPitch - 1, rc = at[q] - (rj + 1) * kFillPitch - 1;
      const int i = ox + rc, j = oy + rj;
      auto unknown = [&](int jj, int ii) { return (int)(S.unk[jj][ii >> 5] >> (ii & 31) & 1u); };
      // inside the region the bits tell; beyond its edge there is no grid
      // (a needed node there would be open)
      const int dg = (i > 0) + (i < M - 1) + (j > 0) + (j < N - 1);
      int uc = 0;
      if (rc > 0) uc += unknown(rj, rc - 1);
      if (rc < kFillReg - 1) uc += unknown(rj, rc + 1);
      if (rj > 0) uc += unknown(rj - 1, rc);
      if (rj < kFillReg - 1) uc += unknown(rj + 1, rc);
      b[q] = A.b[f * n + (long long)j * M + i];
      deg[q] = (float)dg;
      x[q] = dg > uc ? b[q] / (dg - uc) : 0.0;
      S.r[at[q]] = x[q];
      bb += b[q] * b[q];
    }
  }
  __syncthreads();
  // y = A v at this thread's nodes, v in S.r (0 at every node that is not needed)
  auto apply = [&](const double *v, double *y) {
#pragma unroll
    for (int q = 0; q < kFillPer; ++q)
      if (q * kFillThreads < cnt && threadIdx.x + q * kFillThreads < cnt) {
        const double *c = S.r + at[q];
        y[q] = (double)deg[q] * v[q] - ((c[-1] + c[1]) + (c[-kFillPitch] + c[kFillPitch]));
      }
  };
  int par = 0;
  double tot[3];
  auto reduce = [&](double a0, double a1, double a2) {
    a0 = warp_sum(a0);
    a1 = warp_sum(a1);
    a2 = warp_sum(a2);
    if (lane == 0) {
      S.red[par][wid][0] = a0;
      S.red[par][wid][1] = a1;
      S.red[par][wid][2] = a2;
    }
    __syncthreads();
    tot[0] = tot[1] = tot[2] = 0.0;
#pragma unroll
    for (int k = 0; k < kFillThreads / 32; ++k) {
      tot[0] += S.red[par][k][0];
      tot[1] += S.red[par][k][1];
      tot[2] += S.red[par][k][2];
    }
    par ^= 1;
  };
  apply(x, w);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kFillPer; ++q)
    if (threadIdx.x + q * kFillThreads < cnt) {
      r[q] = b[q] - w[q];
      S.r[at[q]] = r[q];
    }
  __syncthreads();
  double alpha = 0.0, beta = 0.0, gi = 0.0, ai = 0.0, bnorm = 0.0;
  bool done = false;
  int it = 0;
  for (; it < kFillMaxit; ++it) {
    apply(r, w);
    double a0 = 0.0, a1 = 0.0;
#pragma unroll
    for (int q = 0; q < kFillPer; ++q) {
      a0 += r[q] * r[q];
      a1 += w[q] * r[q];
    }
    reduce(a0, a1, it == 0 ? bb : 0.0);
    if (it == 0) bnorm = tot[2];
    // a tenth of the grid solver's tolerance: the norm is the tile's, not the grid's
    if (!(tot[0] > 0.01 * A.rtol * A.rtol * bnorm)) {
      done = true;
      break;
    }
    // gi, ai: 1 / gamma and 1 / alpha of the iteration before, formed beside its
    // alpha, so one division is in the chain
    beta = it == 0 ? 0.0 : tot[0] * gi;
    const double t = tot[1] - beta * tot[0] * ai;
    alpha = tot[0] / t;
    gi = 1.0 / tot[0];
    ai = t * gi;
#pragma unroll
    for (int q = 0; q < kFillPer; ++q)
      if (q * kFillThreads < cnt) {
        p[q] = r[q] + beta * p[q];
        s[q] = w[q] + beta * s[q];
        x[q] += alpha * p[q];
        r[q] -= alpha * s[q];
        if (threadIdx.x + q * kFillThreads < cnt) S.r[at[q]] = r[q];
      }
    __syncthreads();
  }
  if (!done) {
    if (threadIdx.x == 0) atomicExch(A.gate, 1);
    return;
  }
  if (threadIdx.x == 0) atomicMax(A.iters, it);
#pragma unroll
  for (int q = 0; q < kFillPer; ++q)
    if (threadIdx.x + q * kFillThreads < cnt) {
      const int rj = at[q] / kFillPitch - 1, rc = at[q] - (rj + 1) * kFillPitch - 1;
      if (rj < kFillHalo || rj >= kFillHalo + kFillTile || rc < kFillHalo || rc >= kFillHalo + kFillTile)
        continue;
      const long long k = (long long)(oy + rj) * M + ox + rc;
      A.x[f * n + k] = x[q];
      A.vals.p[f][k * A.vals.stride[f]] = x[q];
    }
}

// Chebyshev coefficients for eigenvalues in 1 +- kFitRho (Saad, Iterative
// Methods for Sparse Linear Systems, 2nd ed., Algorithm 12.1)
void fit_coefficients(double *ca, double *cb) {
  double rho = kFitRho;
  ca[0] = 0.0;
  cb[0] = 1.0;
  for (int k = 1; k < kFitSteps; ++k) {
    const double next = 1.0 / (2.0 / kFitRho - rho);
    ca[k] = next * rho;
    cb[k] = 2.0 * next / kFitRho;
    rho = next;
  }
}

}  // namespace

int fit_tiles(GridWork &w, int M, int N, int nf, const FieldMap &in, const FieldMap &out,
              const int *bad, const FieldMap *guess, double lam2, double rtol, bool conv,
              cudaStream_t st) {
  FitArgs A;
  A.in = in;
  A.out = out;
  A.guess = guess ? *guess : FieldMap{};
  A.bad = bad;
  A.b = w.b; A.x = w.x; A.mask = w.mask;
  A.part = w.r;  // k_pcg overwrites it only once the gate is set
  A.gate = w.gate; A.iters = w.iters_out; A.bar = w.bar;
  A.lam2 = lam2; A.rtol = rtol;
  fit_coefficients(A.ca, A.cb);
  for (int k = 0; k < 18; ++k) {
    const int nx = k / 3 % 3, ny = k % 3;
    const double d = k / 9 + lam2 * ((nx + ny) + 0.5 * (nx * ny));
    A.dg[k / 9][nx][ny] = d;
    A.di[k / 9][nx][ny] = d > 0.0 ? 1.0 / d : 0.0;
  }
  A.M = M; A.N = N; A.nf = nf;
  const long long tiles = (long long)((M + kFitTile - 1) / kFitTile) * ((N + kFitTile - 1) / kFitTile);
  const dim3 grid((unsigned)tiles, nf);
  const int smem = 2 * kFitPitch * kFitPitch * sizeof(double);
  auto *fn = conv ? k_fit_tile<true> : k_fit_tile<false>;
  ALDIC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  fn<<<grid, kFitThreads, smem, st>>>(A);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

int fill_tiles(GridWork &w, int M, int N, int nf, const FieldMap &vals, const unsigned char *bad,
               double rtol, cudaStream_t st) {
  FillArgs A;
  A.vals = vals;
  A.bad = bad;
  A.b = w.b; A.x = w.x; A.mask = w.mask;
  A.gate = w.gate; A.iters = w.iters_out; A.bar = w.bar;
  A.rtol = rtol;
  A.M = M; A.N = N; A.nf = nf;
  const long long n = (long long)M * N;
  const long long tiles = (long long)((M + kFillTile - 1) / kFillTile) * ((N + kFillTile - 1) / kFillTile);
  const dim3 grid((unsigned)tiles, nf);
  long long lb = (n + 255) / 256;
  if (lb > 592) lb = 592;
  k_fill_load<<<dim3((unsigned)lb, nf), 256, 0, st>>>(A);
  ALDIC_CUDA(cudaFuncSetAttribute(k_fill_tile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(FillShared)));
  k_fill_tile<<<grid, kFillThreads, sizeof(FillShared), st>>>(A);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

}  // namespace aldic
