// fdm.cu -- direct solve of the uniform-mesh Subproblem 2 by fast
// diagonalisation (Lynch, Rice and Thomas, "Direct solution of partial
// difference equations by tensor product methods", Numer. Math. 6, 1964).
//
// On the M x N node grid of MeshSetUp.m both Subproblem 2 operators are
// Kronecker sums of 1-D operators, one per grid direction:
//
//   FE (Subpb2.m:100-195, bilinear squares of side h, 3x3 Gauss -- exact for
//   these integrands, natural boundaries):
//       A = beta (Kx (x) My + Mx (x) Ky) + mu Mx (x) My
//   with the 1-D linear-element stiffness K = (1/h) tridiag(-1, 2, -1)
//   (corner entries 1) and mass M = (h/6) tridiag(1, 4, 1) (corner entries 2);
//
//   FD (funDerivativeOp.m on the (M-2) x (N-2) interior, main_ALDIC.m:243-259):
//       A = beta (I (x) Gx + Gy (x) I) + mu I
//   with G = d'd, d the 1-D difference of funDerivativeOp (central / 2h inside,
//   one-sided with doubled weights at the two ends).
//
// With the generalised eigenbases K V = M V Lambda, V' M V = I of each
// direction, A^-1 = (Vx (x) Vy) D^-1 (Vx (x) Vy)', D = beta (lx_p + ly_q) + mu,
// so a solve is four dense products per field (two per direction) and a
// diagonal scale: C = Vy' B Vx, C ./= D, X = Vy C Vx'.  The 1-D bases are
// computed once per geometry on the host in FP64 (Cholesky M = L L',
// Householder tridiagonalisation and implicit symmetric QR steps with
// Wilkinson shifts of L^-1 K L^-T -- Golub and Van Loan, Matrix
// Computations, 4th ed., algorithms 8.3.1 and 8.3.2) and kept on the device;
// the products run as tiles on the FP64 tensor instruction.  The solution is exact up to
// rounding (about 1e-13 relative), where an iterative solve stops at a
// residual of 1e-11.
#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/aldic_b200.h"
#include "aldic_internal.cuh"
#include "fe_node.cuh"
#include "kernels.cuh"

namespace aldic {

namespace {

// ---------------------------------------------------------------- host: 1-D operators
// assembled 1-D linear-element stiffness K and mass M of n nodes at spacing h
// (natural boundaries), dense row-major
void fe_stiffness_mass(int n, double h, std::vector<double> &K, std::vector<double> &Mm) {
  K.assign((size_t)n * n, 0.0);
  Mm.assign((size_t)n * n, 0.0);
  for (int e = 0; e + 1 < n; ++e) {  // element (e, e+1)
    const int a = e, b = e + 1;
    K[(size_t)a * n + a] += 1.0 / h;
    K[(size_t)b * n + b] += 1.0 / h;
    K[(size_t)a * n + b] -= 1.0 / h;
    K[(size_t)b * n + a] -= 1.0 / h;
    Mm[(size_t)a * n + a] += 2.0 * h / 6.0;
    Mm[(size_t)b * n + b] += 2.0 * h / 6.0;
    Mm[(size_t)a * n + b] += h / 6.0;
    Mm[(size_t)b * n + a] += h / 6.0;
  }
}

// G = d'd with d the n x n difference of funDerivativeOp.m:25-35 along one line
void fd_gram(int n, double h, std::vector<double> &G) {
  std::vector<double> d((size_t)n * n, 0.0);
  const double s = 1.0 / (2.0 * h);
  for (int t = 0; t < n && n > 1; ++t) {
    if (t == 0) {
      d[(size_t)t * n + 1] += 2 * s;
      d[(size_t)t * n + 0] -= 2 * s;
    } else if (t == n - 1) {
      d[(size_t)t * n + n - 1] += 2 * s;
      d[(size_t)t * n + n - 2] -= 2 * s;
    } else {
      d[(size_t)t * n + t + 1] += s;
      d[(size_t)t * n + t - 1] -= s;
    }
  }
  G.assign((size_t)n * n, 0.0);
  for (int i = 0; i < n; ++i)
    for (int j = std::max(0, i - 2); j <= std::min(n - 1, i + 2); ++j) {
      double v = 0.0;
      for (int t = std::max(0, i - 1); t <= std::min(n - 1, i + 1); ++t)
        v += d[(size_t)t * n + i] * d[(size_t)t * n + j];
      G[(size_t)i * n + j] = v;
    }
}

// ---------------------------------------------------------------- host: symmetric eigenproblem
// Householder reduction of the symmetric A (n x n, row-major, destroyed) to
// tridiagonal form T = Q' A Q: diag d, sub-diagonal e (e[k] = T[k+1][k]);
// returns Qt = Q' (row k of Qt is column k of Q).
void tridiagonalise(int n, std::vector<double> &A, std::vector<double> &d, std::vector<double> &e,
                    std::vector<double> &Qt) {
  d.assign(n, 0.0);
  e.assign(n > 1 ? n - 1 : 0, 0.0);
  Qt.assign((size_t)n * n, 0.0);
  for (int i = 0; i < n; ++i) Qt[(size_t)i * n + i] = 1.0;
  std::vector<double> v(n), p(n), w(n), sc(n);
  for (int k = 0; k + 2 < n; ++k) {
    // x = A[k+1:, k]
    const int m = n - k - 1;
    double sig = 0.0;
    for (int i = 1; i < m; ++i) sig += A[(size_t)(k + 1 + i) * n + k] * A[(size_t)(k + 1 + i) * n + k];
    const double x0 = A[(size_t)(k + 1) * n + k];
    if (sig == 0.0) {  // already tridiagonal in this column
      e[k] = x0;
      continue;
    }
    const double nx = std::sqrt(x0 * x0 + sig);
    const double alpha = x0 >= 0 ? -nx : nx;  // H x = alpha e1
    // v = x - alpha e1, H = I - tau v v', tau = 2 / v'v
    v[0] = x0 - alpha;
    for (int i = 1; i < m; ++i) v[i] = A[(size_t)(k + 1 + i) * n + k];
    const double tau = 2.0 / (v[0] * v[0] + sig);
    // p = tau A22 v ; w = p - (tau p'v / 2) v ; A22 -= v w' + w v'
    for (int i = 0; i < m; ++i) {
      const double *row = &A[(size_t)(k + 1 + i) * n + k + 1];
      double s = 0.0;
      for (int j = 0; j < m; ++j) s += row[j] * v[j];
      p[i] = tau * s;
    }
    double pv = 0.0;
    for (int i = 0; i < m; ++i) pv += p[i] * v[i];
    const double kk = 0.5 * tau * pv;
    for (int i = 0; i < m; ++i) w[i] = p[i] - kk * v[i];
    for (int i = 0; i < m; ++i) {
      double *row = &A[(size_t)(k + 1 + i) * n + k + 1];
      for (int j = 0; j < m; ++j) row[j] -= v[i] * w[j] + w[i] * v[j];
    }
    e[k] = alpha;
    // Q <- Q H on columns k+1..: Qt rows k+1.. <- H Qt rows (H symmetric),
    // as row sweeps: sc = v' Qt[k+1:], then Qt[k+1+i] -= tau v_i sc
    std::fill(sc.begin(), sc.end(), 0.0);
    for (int i = 0; i < m; ++i) {
      const double *row = &Qt[(size_t)(k + 1 + i) * n];
      const double vi = v[i];
      for (int c = 0; c < n; ++c) sc[c] += vi * row[c];
    }
    for (int i = 0; i < m; ++i) {
      double *row = &Qt[(size_t)(k + 1 + i) * n];
      const double tv = tau * v[i];
      for (int c = 0; c < n; ++c) row[c] -= tv * sc[c];
    }
  }
  for (int i = 0; i < n; ++i) d[i] = A[(size_t)i * n + i];
  if (n >= 2) e[n - 2] = A[(size_t)(n - 1) * n + n - 2];
}

// implicit symmetric QR steps with Wilkinson shifts on (d, e) until every
// off-diagonal is negligible; each rotation R of rows k, k+1 (T <- R T R')
// is applied to rows k, k+1 of Qt as well, so with Qt = Q' from
// tridiagonalise the original matrix is Qt' diag(d) Qt on return: row p of
// Qt is the eigenvector of eigenvalue d[p].
int tridiagonal_qr(int n, std::vector<double> &d, std::vector<double> &e, std::vector<double> &Qt) {
  const double eps = 2.220446049250313e-16;
  int hi = n - 1, sweeps = 0;
  while (hi > 0) {
    if (std::fabs(e[hi - 1]) <= eps * (std::fabs(d[hi - 1]) + std::fabs(d[hi]))) {
      e[hi - 1] = 0.0;
      --hi;
      continue;
    }
    int lo = hi - 1;
    while (lo > 0 && std::fabs(e[lo - 1]) > eps * (std::fabs(d[lo - 1]) + std::fabs(d[lo]))) --lo;
    if (++sweeps > 60 * n) return E_STATE;
    // Wilkinson shift from the trailing 2 x 2 block
    const double dd = 0.5 * (d[hi - 1] - d[hi]);
    const double eh = e[hi - 1];
    const double den = dd + (dd >= 0 ? 1.0 : -1.0) * std::hypot(dd, eh);
    const double shift = d[hi] - eh * eh / den;
    double x = d[lo] - shift, z = e[lo];
    for (int k = lo; k < hi; ++k) {
      // rotation R (rows k, k+1): [c s; -s c] (x, z)' = (r, 0)'
      const double r = std::hypot(x, z);
      const double c = r == 0.0 ? 1.0 : x / r, s = r == 0.0 ? 0.0 : z / r;
      if (k > lo) e[k - 1] = r;
      const double a = d[k], b = e[k], dn = d[k + 1];
      d[k] = c * c * a + 2 * c * s * b + s * s * dn;
      d[k + 1] = s * s * a - 2 * c * s * b + c * c * dn;
      e[k] = c * s * (dn - a) + (c * c - s * s) * b;
      if (k + 1 < hi) {  // the bulge moves to (k+2, k)
        const double f = e[k + 1];
        x = e[k];
        z = s * f;
        e[k + 1] = c * f;
      }
      double *qa = &Qt[(size_t)k * n], *qb = &Qt[(size_t)(k + 1) * n];
      for (int j = 0; j < n; ++j) {
        const double u = qa[j], w = qb[j];
        qa[j] = c * u + s * w;
        qb[j] = -s * u + c * w;
      }
    }
  }
  return OK;
}

// ---------------------------------------------------------------- device: FP64 products
// TILE x TILE outputs a CTA on the FP64 tensor instruction (m8n8k4), a warp
// 16 x 8 (TILE 32) or 32 x 16 (TILE 64).  K runs in chunks
// of 32 through a ring of three buffers filled by cp.async; an operand lies in
// shared memory the way it does in global memory (k fast or row/column fast),
// lines of TILE or 32 doubles 4 further apart than they are long, so that the
// 4 x 4 doubles a half warp reads of a fragment are in 16 different bank pairs.
//
// What bounds it: these products are small (243 x 243 x 243 and two fields in a
// frame), so the time goes to filling the chip and to latency, not to the 64
// multiply-adds a cycle and SM.  32 x 32 tiles make 128 CTAs of that product
// where 64 x 64 ones made 32, which had K split four ways and a second launch
// to add the slices.  A product of 243 x 243 and two fields takes 9 us against
// 16 with its sum; the fragments need 3 shared loads for 512 multiply-adds a
// warp where a 4 x 4 register tile needs 8.  Addresses are stepped, not formed
// from (line, k) at every copy: that alone was 18 us a product.
constexpr int KC = 32, GT = 256, kFdmStages = 3;
// 64 x 64 tiles, which read half the operand bytes a multiply-add, from two
// full waves of them on
constexpr int kFdmBig = 296;
constexpr int kFdmCluster = 8, kFdmChainTiles = 8;
template <int TILE> struct FdmTile {
  static constexpr int mi = TILE / 16, ni = TILE / 32;  // m8 and n8 fragments a warp
  static constexpr int LT = TILE + 4, LK = KC + 4; // line pitch: row/column fast, k fast
  static constexpr int oper = TILE * LK > KC * LT ? TILE * LK : KC * LT;  // doubles an operand
  static constexpr int smem = kFdmStages * 2 * oper * (int)sizeof(double);
};

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

struct GemmArgs {
  const double *A, *B;
  double *C;
  long long sab, sar, sak;  // element (r, k) of batch b of A at A[b sab + r sar + k sak]
  long long sbb, sbk, sbc;  // element (k, c) of batch b of B
  long long scb, scr, scc;  // element (r, c) of batch b of C
  int R, Cn, K;
  // epilogue 1: C /= beta_b (lr[r] + lc[c]) + mu
  int scale;
  const double *lr, *lc;
  double mu;
  double beta[12];
  const double *beta_ptr;  // if set, beta = *beta_ptr for every batch entry
};

// One operand's TILE lines (line l, k at src[l sl + k sk]) on their way to
// shared memory, KC of k at a time; fast: the lines are adjacent in memory.  A
// thread copies the same TILE KC / 256 places of every chunk, zeros beyond the
// operand.
template <int TILE>
struct Stage {
  using T = FdmTile<TILE>;
  static constexpr int each = TILE * KC / GT;
  const double *src;    // of its first place
  long long next, adv;  // to its next place, to the next chunk
  int l, k, dl, dk, dst, dnext;
  __device__ __forceinline__ Stage(const double *base, long long sl, long long sk, int l0, bool fast) {
    const int t = threadIdx.x;
    const int ll = fast ? t % TILE : t / KC;
    k = fast ? t / TILE : t % KC;
    l = l0 + ll;
    dl = fast ? 0 : GT / KC;
    dk = fast ? GT / TILE : 0;
    dst = fast ? k * T::LT + ll : ll * T::LK + k;
    dnext = fast ? dk * T::LT : dl * T::LK;
    src = base + l * sl + k * sk;
    next = dl * sl + dk * sk;
    adv = KC * sk;
  }
  __device__ __forceinline__ void copy(double *buf, int lines, int K) {
    const unsigned to = (unsigned)__cvta_generic_to_shared(buf + dst);
#pragma unroll
    for (int i = 0; i < each; ++i) {
      const bool in = l + i * dl < lines && k + i * dk < K;
      const double *p = in ? src + i * next : src0;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(to + 8u * (unsigned)(i * dnext)), "l"(p),
                   "r"(in ? 8 : 0)
                   : "memory");
    }
    src += adv;
    k += KC;
  }
  const double *src0 = nullptr;  // a valid address, not read
};

template <int TILE>
__device__ __forceinline__ void fdm_tile(const GemmArgs &g, int b, int r0, int c0, double *sm) {
  using T = FdmTile<TILE>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double *A = g.A + (long long)b * g.sab;
  const double *B = g.B + (long long)b * g.sbb;
  const bool af = g.sar <= g.sak, bf = g.sbc <= g.sbk;
  const int nch = (g.K + KC - 1) / KC;
  Stage<TILE> sa(A, g.sar, g.sak, r0, af), sb(B, g.sbc, g.sbk, c0, bf);
  sa.src0 = A;
  sb.src0 = B;
  auto stage = [&](int ch) {
    if (ch < nch) {
      double *buf = sm + (ch % kFdmStages) * 2 * T::oper;
      sa.copy(buf, g.R, g.K);
      sb.copy(buf + T::oper, g.Cn, g.K);
    }
    cp_async_commit();
  };
  // the warp's part of the tile; a lane's row/column (lane / 4) and k (lane % 4) of a fragment
  const int wr = (warp >> 2) * (TILE / 2), wc = (warp & 3) * (TILE / 4);
  const int al = af ? 1 : T::LK, ak = af ? T::LT : 1, bl = bf ? 1 : T::LK, bk = bf ? T::LT : 1;
  const int oa = (wr + (lane >> 2)) * al + (lane & 3) * ak, ob = (wc + (lane >> 2)) * bl + (lane & 3) * bk;
  double acc[T::mi][T::ni][2] = {};
#pragma unroll
  for (int ch = 0; ch < kFdmStages - 1; ++ch) stage(ch);
  for (int ch = 0; ch < nch; ++ch) {
    cp_async_wait<kFdmStages - 2>();
    __syncthreads();  // chunk ch is in; the buffer of chunk ch - 1 is free
    stage(ch + kFdmStages - 1);
    const double *As = sm + (ch % kFdmStages) * 2 * T::oper + oa, *Bs = As - oa + T::oper + ob;
#pragma unroll
    for (int kk = 0; kk < KC; kk += 4) {
      double fa[T::mi], fb[T::ni];
#pragma unroll
      for (int i = 0; i < T::mi; ++i) fa[i] = As[8 * i * al + kk * ak];
#pragma unroll
      for (int j = 0; j < T::ni; ++j) fb[j] = Bs[8 * j * bl + kk * bk];
#pragma unroll
      for (int i = 0; i < T::mi; ++i)
#pragma unroll
        for (int j = 0; j < T::ni; ++j) mma_f64(acc[i][j], fa[i], fb[j]);
    }
  }
  const double beta = g.beta_ptr ? *g.beta_ptr : g.beta[b < 12 ? b : 11];
  double *C = g.C + (long long)b * g.scb;
#pragma unroll
  for (int i = 0; i < T::mi; ++i) {
    const int r = r0 + wr + 8 * i + (lane >> 2);
    if (r >= g.R) continue;
#pragma unroll
    for (int j = 0; j < T::ni; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c0 + wc + 8 * j + 2 * (lane & 3) + e;
        if (c >= g.Cn) continue;
        double v = acc[i][j][e];
        if (g.scale) v /= beta * (g.lr[r] + g.lc[c]) + g.mu;
        C[(long long)r * g.scr + (long long)c * g.scc] = v;
      }
  }
}

template <int TILE>
__global__ void __launch_bounds__(GT) k_fdm_gemm(const __grid_constant__ GemmArgs g) {
  extern __shared__ double sm[];
  fdm_tile<TILE>(g, blockIdx.z, blockIdx.y * TILE, blockIdx.x * TILE, sm);
}

// The four products of a small solve in one launch, and before them the
// right-hand side of the finite-element step: a cluster of eight CTAs takes the
// nodes, then the 32 x 32 tiles of each product in turn and meets at the cluster's
// barrier (a few hundred cycles, where a launch costs some 2 us).
struct FdmChain {
  GemmArgs g[4];
  int batch;
  // the right-hand side's inputs (null U: it is there), two fields of M N at b
  const double *U, *F, *ud, *vd;
  double *b;
  double h;
};
__global__ void __launch_bounds__(GT) __cluster_dims__(kFdmCluster, 1, 1)
    k_fdm_chain(const __grid_constant__ FdmChain ch) {
  extern __shared__ double sm[];
  auto meet = []() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  };
  if (ch.U) {
    const int M = ch.g[0].Cn, N = ch.g[0].R, n = M * N;
    const double beta = ch.g[0].beta_ptr ? *ch.g[0].beta_ptr : ch.g[0].beta[0], mu = ch.g[0].mu;
    for (int k = blockIdx.x * GT + threadIdx.x; k < n; k += kFdmCluster * GT) {
      const FeParts p = fe_rhs_node(M, N, ch.h, k % M, k / M, ch.U, ch.F, ch.ud, ch.vd);
      ch.b[k] = beta * p.ku + mu * p.mu;
      ch.b[n + k] = beta * p.kv + mu * p.mv;
    }
    meet();
  }
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    const GemmArgs &g = ch.g[q];
    const int tc = (g.Cn + 31) / 32, tr = (g.R + 31) / 32;
    for (int t = blockIdx.x; t < tc * tr * ch.batch; t += kFdmCluster) {
      fdm_tile<32>(g, t / (tc * tr), t % (tc * tr) / tc * 32, t % tc * 32, sm);
      __syncthreads();  // the ring is refilled
    }
    meet();
  }
}

// the kernels' dynamic shared memory (above the 48 KB default) on the current
// device; set by fdm_ensure, ahead of any stream capture
int gemm_setup() {
  ALDIC_CUDA(cudaFuncSetAttribute(k_fdm_gemm<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, FdmTile<32>::smem));
  ALDIC_CUDA(cudaFuncSetAttribute(k_fdm_gemm<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, FdmTile<64>::smem));
  ALDIC_CUDA(cudaFuncSetAttribute(k_fdm_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, FdmTile<32>::smem));
  return OK;
}

template <int TILE>
int gemm_tile(const GemmArgs &g, int batch, cudaStream_t st) {
  const dim3 grid((unsigned)((g.Cn + TILE - 1) / TILE), (unsigned)((g.R + TILE - 1) / TILE), (unsigned)batch);
  k_fdm_gemm<TILE><<<grid, GT, FdmTile<TILE>::smem, st>>>(g);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}
long long gemm_tiles(int R, int Cn, int batch, int tile) {
  return (long long)((Cn + tile - 1) / tile) * ((R + tile - 1) / tile) * batch;
}
int gemm(const GemmArgs &g, int batch, cudaStream_t st) {
  return gemm_tiles(g.R, g.Cn, batch, 64) >= kFdmBig ? gemm_tile<64>(g, batch, st) : gemm_tile<32>(g, batch, st);
}

}  // namespace

// V (n x n row-major, column p = eigenvector p) and lam (n) of the 1-D
// pencil (K, M) of `type` (FDM_FE: linear-element stiffness and mass;
// FDM_FD: funDerivativeOp's d'd with M = I), V' M V = I.
int fdm_basis_1d(int type, int n, double h, double *V, double *lam) {
  ALDIC_CHECK(n >= 1 && n <= 16384 && h > 0 && V && lam && (type == FDM_FE || type == FDM_FD), E_ARG,
              "fdm basis: bad arguments");
  std::vector<double> K, Mm;
  if (type == FDM_FE) {
    fe_stiffness_mass(n, h, K, Mm);
  } else {
    fd_gram(n, h, K);
  }
  if (n == 1) {  // a single node: K = 0 (FE) / G = 0 (FD)
    lam[0] = 0.0;
    V[0] = type == FDM_FE ? 1.0 / std::sqrt(Mm[0] > 0 ? Mm[0] : 1.0) : 1.0;
    return OK;
  }
  // C = L^-1 K L^-T with M = L L' (L lower bidiagonal: diag l, sub m); FD: L = I
  std::vector<double> l(n, 1.0), m(n, 0.0);
  std::vector<double> C = K;
  if (type == FDM_FE) {
    for (int i = 0; i < n; ++i) {
      const double t = Mm[(size_t)i * n + i] - (i ? m[i] * m[i] : 0.0);
      ALDIC_CHECK(t > 0, E_STATE, "fdm basis: mass matrix not positive definite");
      l[i] = std::sqrt(t);
      if (i + 1 < n) m[i + 1] = Mm[(size_t)(i + 1) * n + i] / l[i];
    }
    // X = L^-1 K (rows), then C = L^-1 X' (= L^-1 K L^-T, K symmetric)
    std::vector<double> X((size_t)n * n);
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j)
        X[(size_t)i * n + j] = (K[(size_t)i * n + j] - (i ? m[i] * X[(size_t)(i - 1) * n + j] : 0.0)) / l[i];
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j)
        C[(size_t)i * n + j] = (X[(size_t)j * n + i] - (i ? m[i] * C[(size_t)(i - 1) * n + j] : 0.0)) / l[i];
    for (int i = 0; i < n; ++i)  // symmetrise the rounding
      for (int j = 0; j < i; ++j) {
        const double s = 0.5 * (C[(size_t)i * n + j] + C[(size_t)j * n + i]);
        C[(size_t)i * n + j] = C[(size_t)j * n + i] = s;
      }
  }
  std::vector<double> d, e, Qt;
  tridiagonalise(n, C, d, e, Qt);
  const int rc = tridiagonal_qr(n, d, e, Qt);
  ALDIC_CHECK(rc == OK, E_STATE, "fdm basis: the QR iteration did not converge");
  // V = L^-T Q: back substitution L' V = Q, Q[i][p] = Qt[p][i]
  for (int i = n - 1; i >= 0; --i)
    for (int p = 0; p < n; ++p) {
      double q = Qt[(size_t)p * n + i];
      if (i + 1 < n) q -= m[i + 1] * V[(size_t)(i + 1) * n + p];
      V[(size_t)i * n + p] = q / l[i];
    }
  for (int p = 0; p < n; ++p) lam[p] = d[p];
  return OK;
}

int fdm_ensure(FdmBasis &B, int type, int M, int N, double h, cudaStream_t st) {
  if (B.type == type && B.M == M && B.N == N && B.h == h && B.buf.p) return OK;
  ALDIC_CHECK(M >= 1 && N >= 1, E_ARG, "fdm: empty grid");
  std::vector<double> host((size_t)M * M + (size_t)N * N + M + N);
  double *Vx = host.data(), *Vy = Vx + (size_t)M * M, *lx = Vy + (size_t)N * N, *ly = lx + M;
  int rc;
  if ((rc = gemm_setup())) return rc;
  if ((rc = fdm_basis_1d(type, M, h, Vx, lx))) return rc;
  if ((rc = fdm_basis_1d(type, N, h, Vy, ly))) return rc;
  B.type = -1;
  if ((rc = B.buf.ensure(sizeof(double) * host.size()))) return rc;
  ALDIC_CUDA(cudaMemcpyAsync(B.buf.p, host.data(), sizeof(double) * host.size(),
                             cudaMemcpyHostToDevice, st));
  ALDIC_CUDA(cudaStreamSynchronize(st));  // the host vector goes out of scope
  double *d = B.buf.as<double>();
  B.Vx = d;
  B.Vy = d + (size_t)M * M;
  B.lx = B.Vy + (size_t)N * N;
  B.ly = B.lx + M;
  B.type = type;
  B.M = M;
  B.N = N;
  B.h = h;
  return OK;
}

namespace {

// the products of fdm_solve
FdmChain solve_chain(const FdmBasis &B, int nrhs, const double *b, double *x, double *tmp, double mu, double beta,
                     const double *beta_each, const double *beta_ptr, double *inter) {
  const int M = B.M, N = B.N;
  const long long n = (long long)M * N;
  FdmChain ch{};
  ch.batch = nrhs;
  GemmArgs &g = ch.g[0];
  g.mu = mu;
  for (int f = 0; f < 12; ++f) g.beta[f] = (beta_each && f < nrhs) ? beta_each[f] : beta;
  g.beta_ptr = beta_ptr;
  g.R = N; g.Cn = M;
  for (int q = 1; q < 4; ++q) ch.g[q] = g;
  // field f as an N x M matrix (row j = node row y, column i = x): B_f[j][i] = b[f n + j M + i]
  auto set = [&](int q, const double *A, long long sab, long long sar, long long sak, const double *Bm,
                 long long sbb, long long sbk, long long sbc, double *C, int K) {
    GemmArgs &p = ch.g[q];
    p.A = A; p.sab = sab; p.sar = sar; p.sak = sak;
    p.B = Bm; p.sbb = sbb; p.sbk = sbk; p.sbc = sbc;
    p.C = C; p.scb = n; p.scr = M; p.scc = 1;
    p.K = K;
  };
  set(0, b, n, M, 1, B.Vx, 0, M, 1, tmp, M);     // T = B_f Vx
  set(1, B.Vy, 0, 1, N, tmp, n, M, 1, x, N);     // C = Vy' T, C[q][p] /= beta (ly[q] + lx[p]) + mu
  ch.g[1].scale = 1; ch.g[1].lr = B.ly; ch.g[1].lc = B.lx;
  set(2, x, n, M, 1, B.Vx, 0, 1, M, tmp, M);     // S = C Vx'
  set(3, B.Vy, 0, N, 1, tmp, n, M, 1, x, N);     // X = Vy S
  if (inter) {
    ch.g[3].C = inter;
    ch.g[3].scb = 1; ch.g[3].scr = (long long)nrhs * M; ch.g[3].scc = nrhs;
  }
  return ch;
}

bool one_launch(const FdmBasis &B, int nrhs) {
  // One launch while the cluster has a tile a CTA: a whole aldic_subpb2 at 43 x 43
  // takes 38.8 us this way and 58 us with five launches; with two rounds of
  // tiles (61 x 97, 55.4 us) it is no faster than four launches of 128 x 128
  // (53.7 us).
  return gemm_tiles(B.N, B.M, nrhs, 32) <= kFdmChainTiles;
}

int run_chain(const FdmChain &ch, cudaStream_t st) {
  k_fdm_chain<<<kFdmCluster, GT, FdmTile<32>::smem, st>>>(ch);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

}  // namespace

int fdm_solve(const FdmBasis &B, int nrhs, const double *b, double *x, double *tmp, double mu,
              double beta, const double *beta_each, const double *beta_ptr, cudaStream_t st,
              double *inter) {
  ALDIC_CHECK(B.buf.p && nrhs >= 1 && nrhs <= 12, E_ARG, "fdm solve: bad arguments");
  const FdmChain ch = solve_chain(B, nrhs, b, x, tmp, mu, beta, beta_each, beta_ptr, inter);
  if (one_launch(B, nrhs)) return run_chain(ch, st);
  for (int q = 0; q < 4; ++q) {
    const int rc = gemm(ch.g[q], nrhs, st);
    if (rc) return rc;
  }
  return OK;
}

int fe_solve(const FdmBasis &B, GridWork &w, double h, double beta, double mu, const double *beta_ptr,
             const double *U, const double *F, const double *ud, const double *vd, double *Uhat, cudaStream_t st) {
  ALDIC_CHECK(B.buf.p && B.type == FDM_FE, E_ARG, "fe solve: no basis");
  FdmChain ch = solve_chain(B, 2, w.b, w.x, w.r, mu, beta, nullptr, beta_ptr, Uhat);
  if (one_launch(B, 2)) {
    ch.U = U; ch.F = F; ch.ud = ud; ch.vd = vd;
    ch.b = w.b;
    ch.h = h;
    return run_chain(ch, st);
  }
  const int rc = fe_rhs(w, B.M, B.N, h, beta, mu, U, F, ud, vd, st, beta_ptr, 0);
  return rc ? rc : fdm_solve(B, 2, w.b, w.x, w.r, mu, beta, nullptr, beta_ptr, st, Uhat);
}

// The beta sweep's eigen-domain solutions from the two transformed
// right-hand-side parts C4 (fields 0-1 beta part, 2-3 mu part; entry
// (q, p) at q M + p): X field 2k + c = (beta_k F_c + mu U_c) /
// (beta_k (ly[q] + lx[p]) + mu), the divisor of the one-system epilogue.
struct SweepBetas {
  double v[6];
};
__global__ void k_fdm_sweep_combine(int M, int N, const double *__restrict__ ly,
                                    const double *__restrict__ lx, SweepBetas be, double mu,
                                    const double *__restrict__ C4, double *__restrict__ X) {
  const long long n = (long long)M * N;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    const int q = (int)(idx / M), p = (int)(idx - (long long)q * M);
    const double lam = ly[q] + lx[p];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double F = C4[c * n + idx], U = C4[(2 + c) * n + idx];
#pragma unroll
      for (int k = 0; k < 6; ++k)
        X[(2 * k + c) * n + idx] = (be.v[k] * F + mu * U) / (be.v[k] * lam + mu);
    }
  }
}

int fdm_solve_sweep(const FdmBasis &B, const double beta[6], const double *b, double *x,
                    double *tmp, double mu, cudaStream_t st) {
  ALDIC_CHECK(B.buf.p, E_ARG, "fdm sweep: no basis");
  const int M = B.M, N = B.N;
  const long long n = (long long)M * N;
  GemmArgs g{};
  g.mu = mu;
  int rc;
  // 1. T = B_f Vx for the two parts (4 fields) -> tmp fields 0-3
  g.A = b; g.sab = n; g.sar = M; g.sak = 1;
  g.B = B.Vx; g.sbb = 0; g.sbk = M; g.sbc = 1;
  g.C = tmp; g.scb = n; g.scr = M; g.scc = 1;
  g.R = N; g.Cn = M; g.K = M; g.scale = 0;
  if ((rc = gemm(g, 4, st))) return rc;
  // 2. C = Vy' T, unscaled -> tmp fields 4-7
  g.A = B.Vy; g.sab = 0; g.sar = 1; g.sak = N;
  g.B = tmp; g.sbb = n; g.sbk = M; g.sbc = 1;
  g.C = tmp + 4 * n; g.scb = n; g.scr = M; g.scc = 1;
  g.R = N; g.Cn = M; g.K = N; g.scale = 0;
  if ((rc = gemm(g, 4, st))) return rc;
  // the six systems' scaled eigen-domain solutions -> x fields 0-11
  SweepBetas be;
  for (int k = 0; k < 6; ++k) be.v[k] = beta[k];
  const long long nb = (n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8;
  k_fdm_sweep_combine<<<(unsigned)nb, 256, 0, st>>>(M, N, B.ly, B.lx, be, mu, tmp + 4 * n, x);
  ALDIC_CUDA(cudaGetLastError());
  // 3. S = C Vx' -> tmp (12 fields)
  g.A = x; g.sab = n; g.sar = M; g.sak = 1;
  g.B = B.Vx; g.sbb = 0; g.sbk = 1; g.sbc = M;
  g.C = tmp; g.scb = n; g.scr = M; g.scc = 1;
  g.R = N; g.Cn = M; g.K = M; g.scale = 0;
  if ((rc = gemm(g, 12, st))) return rc;
  // 4. X = Vy S -> x
  g.A = B.Vy; g.sab = 0; g.sar = N; g.sak = 1;
  g.B = tmp; g.sbb = n; g.sbk = M; g.sbc = 1;
  g.C = x; g.scb = n; g.scr = M; g.scc = 1;
  g.R = N; g.Cn = M; g.K = N; g.scale = 0;
  return gemm(g, 12, st);
}

}  // namespace aldic

extern "C" ALDIC_API int aldic_fdm_basis(int type, int n, double h, double *V, double *lam) {
  return aldic::fdm_basis_1d(type, n, h, V, lam);
}
