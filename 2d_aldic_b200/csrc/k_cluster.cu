// k_cluster.cu -- the pipelined conjugate gradients of k_pcg (k_grid.cu) for
// systems of up to 32768 nodes, a cluster of 16 CTAs a right-hand side.
//
// What bounds such a solve is latency: tens to a hundred iterations of a few
// thousand rows each.  In the grid-wide kernel an iteration is a chain through
// L2 -- row pointer, column, direction of every entry, ten vectors, block
// partials, a barrier over all CTAs -- of 8 us for two fields and 18 us for
// six.  Here a thread keeps its rows' iterates in registers, the matrix rows lie
// in shared memory, the direction vector is read from the other CTAs'
// memory, and the barrier is the cluster's: 2 us an iteration, and the fields
// run side by side, each to its own end.  Quadtree frame, 16805 nodes: the
// refills (74 iterations of 2 fields, 129 of 6) and three solves (20 iterations
// of 2, 6 and 2 fields) took 3.6 ms, 0.74 ms so.  With each CTA's own
// unknowns as its rows, not equal runs of all, the refills of a hole's rim took
// 3.3 us an iteration.
//
// The operator is applied as y = s x_k + sum_c a_c (x_c - x_k), s the row's sum:
// the differences keep the digits that a Laplacian's entries would cancel.
#include <algorithm>

#include "aldic_internal.cuh"
#include "kernels.cuh"

namespace aldic {

namespace {

constexpr int CL = 16;                  // CTAs of a cluster
constexpr int CT = 512, CW = CT / 32;   // threads, warps
constexpr int kClMaxRows = 4;           // rows a thread at most
constexpr size_t kClSmem = 216 * 1024;  // dynamic shared memory, at 1 CTA an SM

struct ClArgs {
  int n, chunk;  // nodes; nodes a CTA
  int cap;       // matrix entries its shared memory holds
  const double *b;
  double *x;
  const unsigned char *mask;
  CsrOp csr;
  double beta[6], mu;
  // scattered gridfit: A'A (9 coefficients a node), springs lam2 on an M x N grid
  const double *ata;
  int M, N;
  double lam2;
  double rtol;
  int maxit;
  int *iters_out, *err;
};

// Entry p of row k of the system, p from first to last: its column (-1: none) and
// its value.
struct CsrRows {
  static constexpr bool masked = true;
  static __device__ __forceinline__ int first(const ClArgs &A, int k) { return A.csr.row[k]; }
  static __device__ __forceinline__ int last(const ClArgs &A, int k) { return A.csr.row[k + 1]; }
  static __device__ __forceinline__ int col(const ClArgs &A, int, int p) { return A.csr.col[p]; }
  static __device__ __forceinline__ double val(const ClArgs &A, int f, int, int p) {
    return A.csr.valM ? A.beta[f] * A.csr.val[p] + A.mu * A.csr.valM[p] : A.csr.val[p];
  }
  // its share of the row's sum
  static __device__ __forceinline__ double share(const ClArgs &, int, int, double v) { return v; }
  static __device__ __forceinline__ double diag(const ClArgs &A, int f, int k) {
    return A.csr.valM ? A.beta[f] * A.csr.diag[k] + A.mu * A.csr.diagM[k] : A.csr.diag[k];
  }
};
struct AtaRows {
  static constexpr bool masked = false;
  static __device__ __forceinline__ int first(const ClArgs &, int) { return 0; }
  static __device__ __forceinline__ int last(const ClArgs &, int) { return 9; }
  static __device__ __forceinline__ int col(const ClArgs &A, int k, int p) {
    const int di = p % 3 - 1, dj = p / 3 - 1, i = k % A.M + di, j = k / A.M + dj;
    return i < 0 || i >= A.M || j < 0 || j >= A.N ? -1 : i + j * A.M;
  }
  static __device__ __forceinline__ double spring(const ClArgs &A, int p) {
    return p == 4 ? 0.0 : A.lam2 * (p & 1 ? 1.0 : 0.5);
  }
  static __device__ __forceinline__ double val(const ClArgs &A, int, int k, int p) {
    return A.ata[9LL * k + p] - spring(A, p);
  }
  // the springs' entries sum to nothing
  static __device__ __forceinline__ double share(const ClArgs &A, int k, int p, double) { return A.ata[9LL * k + p]; }
  static __device__ __forceinline__ double diag(const ClArgs &A, int, int k) {
    double d = A.ata[9LL * k + 4];
    for (int p = 0; p < 9; ++p)
      if (col(A, k, p) >= 0) d += spring(A, p);
    return d;
  }
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(const void *p, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ double cluster_load(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void cluster_store(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ unsigned short cluster_load16(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void cluster_store32(uint32_t a, int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// v / d for v below 2^16 and d from 2 to 2^12 by its ceil(2^32 / d): v times what that
// exceeds 2^32 / d by is below 2^16, less than 2^32 / d, a quotient's least step
__device__ __forceinline__ uint32_t split_by(int d) { return d == 1 ? 0u : 0xffffffffu / (uint32_t)d + 1u; }
__device__ __forceinline__ int split(int v, uint32_t m) { return m ? (int)__umulhi((uint32_t)v, m) : v; }

struct ClShared {
  double warp_part[CW][4];
  double part[2][CL][4];
  int warp_count[CW];
  int count[CL];  // unknowns of each CTA's nodes
};
constexpr unsigned short kKnown = 0xffff;

template <typename Rows, int K>
__global__ void __launch_bounds__(CT, 1) k_pcg_cluster(const __grid_constant__ ClArgs A) {
  __shared__ ClShared S;
  extern __shared__ __align__(16) unsigned char sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = blockIdx.x / CL, rank = blockIdx.x % CL;
  const int base = rank * A.chunk, cnt = max(0, min(A.chunk, A.n - base));
  double *const mb = (double *)sm;  // the direction vector, two buffers of chunk
  double *const val = mb + 2 * A.chunk;
  uint32_t *const adr = (uint32_t *)(val + A.cap);
  int *const list = (int *)(adr + A.cap);                               // the rows: their nodes
  unsigned short *const slot = (unsigned short *)(list + A.chunk);      // of its nodes: the number among their unknowns
  const long long fo = (long long)f * A.n;
  const double *b = A.b + fo;
  double *X = A.x + fo;
  const unsigned char *mask = A.mask + fo;
  const uint32_t other = 8u * (uint32_t)A.chunk;  // from buffer 0 to buffer 1

  // every CTA of the cluster runs before its shared memory is written from another
  cluster_sync();
  // value of every thread scanned over the block: the sum before it, and in all
  auto scan = [&](int v, int *total) {
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    __syncthreads();  // warp_count is free
    if (lane == 31) S.warp_count[warp] = inc;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < CW; ++w) {
      const int t = S.warp_count[w];
      before += w < warp ? t : 0;
      all += t;
    }
    *total = all;
    return before + inc - v;
  };
  // sums over the cluster, the same bits in every thread; orders all shared
  // memory of the cluster
  auto reduce = [&](double (&v)[4], int nv, int buf) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c < nv) {
        v[c] = warp_sum(v[c]);
        if (lane == 0) S.warp_part[warp][c] = v[c];
      }
    __syncthreads();
    if (warp == 0) {
      const uint32_t to = cluster_addr(&S.part[buf][rank][0], lane & (CL - 1));
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (c < nv) {
          double t = S.warp_part[lane & (CW - 1)][c];
#pragma unroll
          for (int o = CW / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          if (lane < CL) cluster_store(to + 8 * c, t);
        }
    }
    cluster_sync();
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c < nv) {
        double t = S.part[buf][lane & (CL - 1)][c];
#pragma unroll
        for (int o = CL / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        v[c] = t;
      }
  };

  // ---- the unknowns among this CTA's nodes, numbered in order; then dealt to the
  // CTAs in equal runs (a refill's lie close together)
  int mine = 0;
  double bb = 0.0;
  for (int i0 = 0; i0 < A.chunk; i0 += CT) {
    const int i = i0 + tid;
    const bool in = i < cnt, act = in && (!Rows::masked || mask[base + i]);
    if (in) bb += b[base + i] * b[base + i];
    int total;
    const int at = mine + scan(act ? 1 : 0, &total);
    if (i < A.chunk) slot[i] = act ? (unsigned short)at : kKnown;
    mine += total;
  }
  if (tid < CL) cluster_store32(cluster_addr(&S.count[rank], tid), mine);
  cluster_sync();
  int all = 0, before = 0;
#pragma unroll
  for (int r = 0; r < CL; ++r) {
    before += r < rank ? S.count[r] : 0;
    all += S.count[r];
  }
  const int per = max(1, (all + CL - 1) / CL), nact = max(0, min(per, all - rank * per));
  const uint32_t perM = split_by(per), chunkM = split_by(A.chunk);
  for (int i = tid; i < cnt; i += CT)
    if (slot[i] != kKnown) {
      const int u = before + slot[i];
      cluster_store32(cluster_addr(list + (u - split(u, perM) * per), split(u, perM)), base + i);
    }
  __syncthreads();  // the scans' reads
  if (tid == 0) {  // counts to offsets
    int o = 0;
    for (int r = 0; r < CL; ++r) {
      const int t = S.count[r];
      S.count[r] = o;
      o += t;
    }
  }
  cluster_sync();
  // the number of node c among all unknowns, or -1
  auto unknown = [&](int c) {
    const int r = split(c, chunkM);
    const unsigned short t = cluster_load16(cluster_addr(slot + (c - r * A.chunk), r));
    return t == kKnown ? -1 : S.count[r] + t;
  };
  // ---- their rows; r = b - A x, u = r / diag
  int start[K], len[K];
  double xs[K], rs[K], us[K], ws[K], zs[K], qs[K], ss[K], ps[K], di[K], s0[K], ms[K];
  int used = 0;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int it = q * CT + tid;
    const bool in = it < nact;
    const int k = in ? list[it] : 0;
    len[q] = start[q] = 0;
    xs[q] = rs[q] = us[q] = ws[q] = zs[q] = qs[q] = ss[q] = ps[q] = di[q] = s0[q] = ms[q] = 0.0;
    if (q * CT >= nact) continue;  // the whole block
    const int p0 = in ? Rows::first(A, k) : 0, p1 = in ? Rows::last(A, k) : 0;
    int total;
    start[q] = used + scan(p1 - p0, &total);
    used += total;
    if (start[q] + p1 - p0 > A.cap) start[q] = -1;  // stays in global memory
    if (in) {
      const double x = X[k];
      double y = 0.0, sum = 0.0;
      int at = start[q];
      for (int p = p0; p < p1; p += 8) {
        int c[8], u[8];
        double v[8], xc[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          c[e] = p + e < p1 ? Rows::col(A, k, p + e) : -1;
          v[e] = c[e] >= 0 ? Rows::val(A, f, k, p + e) : 0.0;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          u[e] = c[e] >= 0 ? unknown(c[e]) : -1;
          xc[e] = u[e] >= 0 ? X[c[e]] : 0.0;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (u[e] < 0) continue;
          sum += Rows::share(A, k, p + e, v[e]);
          if (c[e] == k) continue;
          y += v[e] * (xc[e] - x);
          if (at >= 0) {
            val[at] = v[e];
            adr[at++] = cluster_addr(mb + (u[e] - split(u[e], perM) * per), split(u[e], perM));
          }
        }
      }
      if (at >= 0) len[q] = at - start[q];
      s0[q] = sum;
      xs[q] = x;
      rs[q] = b[k] - (y + sum * x);
      di[q] = 1.0 / Rows::diag(A, f, k);
      us[q] = rs[q] * di[q];
      mb[it] = us[q];
    }
  }
  // y = A v at this thread's row q, v in buffer buf of the cluster, vk its own
  auto apply = [&](int q, int buf, double vk) {
    const uint32_t o = buf ? other : 0u;
    double y = 0.0;
    if (start[q] >= 0) {
      const int p0 = start[q], p1 = p0 + len[q];
      for (int p = p0; p < p1; p += 8) {
        double v[8], a[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const bool in = p + e < p1;
          v[e] = vk;
          a[e] = in ? val[p + e] : 0.0;
          if (in) v[e] = cluster_load(adr[p + e] + o);
        }
        double y0 = 0.0;
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          y += a[e] * (v[e] - vk);
          y0 += a[e + 1] * (v[e + 1] - vk);
        }
        y += y0;
      }
    } else {
      const int k = list[q * CT + tid], p1 = Rows::last(A, k);
      for (int p = Rows::first(A, k); p < p1; ++p) {
        const int c = Rows::col(A, k, p), u = c >= 0 && c != k ? unknown(c) : -1;
        if (u >= 0) y += Rows::val(A, f, k, p) * (cluster_load(cluster_addr(mb + (u - split(u, perM) * per), split(u, perM)) + o) - vk);
      }
    }
    return y + s0[q] * vk;
  };
  cluster_sync();
  double sums[4] = {0.0, 0.0, 0.0, bb};
#pragma unroll
  for (int q = 0; q < K; ++q) {
    if (q * CT + tid >= nact) continue;
    ws[q] = apply(q, 0, us[q]);
    ms[q] = ws[q] * di[q];
    mb[A.chunk + q * CT + tid] = ms[q];
    sums[0] += rs[q] * us[q];
    sums[1] += ws[q] * us[q];
    sums[2] += rs[q] * rs[q];
  }
  reduce(sums, 4, 0);
  double alpha = sums[0] / sums[1], beta = 0.0;
  double gi = 1.0 / sums[0], ai = sums[1] / sums[0];  // of gamma and alpha, ahead of the next sums
  const double goal = A.rtol * A.rtol * sums[3];
  bool done = !(sums[2] > goal);
  int it = 0;
  for (; it < A.maxit && !done; ++it) {
    const int buf = (it & 1) ^ 1;  // holds m
    sums[0] = sums[1] = sums[2] = 0.0;
#pragma unroll
    for (int q = 0; q < K; ++q) {
      if (q * CT + tid >= nact) continue;
      const double nv = apply(q, buf, ms[q]);
      zs[q] = nv + beta * zs[q];
      qs[q] = ms[q] + beta * qs[q];
      ss[q] = ws[q] + beta * ss[q];
      ps[q] = us[q] + beta * ps[q];
      xs[q] += alpha * ps[q];
      rs[q] -= alpha * ss[q];
      us[q] -= alpha * qs[q];
      ws[q] -= alpha * zs[q];
      ms[q] = ws[q] * di[q];
      mb[(buf ^ 1) * A.chunk + q * CT + tid] = ms[q];
      sums[0] += rs[q] * us[q];
      sums[1] += ws[q] * us[q];
      sums[2] += rs[q] * rs[q];
    }
    reduce(sums, 3, buf);
    beta = sums[0] * gi;
    const double t = sums[1] - beta * sums[0] * ai;
    alpha = sums[0] / t;
    gi = 1.0 / sums[0];
    ai = t * gi;
    done = !(sums[2] > goal);
  }
#pragma unroll
  for (int q = 0; q < K; ++q)
    if (q * CT + tid < nact) X[list[q * CT + tid]] = xs[q];
  if (rank == 0 && tid == 0) {
    atomicMax(A.iters_out, it);
    if (!done) atomicExch(A.err, 2);  // not converged within maxit
  }
  cluster_sync();  // no CTA leaves while another may read its shared memory
}

template <typename Rows, int K>
int launch_k(ClArgs &A, int nrhs, cudaStream_t st, bool *ran) {
  auto fn = k_pcg_cluster<Rows, K>;
  // an entry is 12 bytes; a node 16 of direction, 4 of the list, 2 of its number
  A.cap = (int)((kClSmem - 22 * (size_t)A.chunk - 64) / 12) & ~3;
  ALDIC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmem));
  ALDIC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(CL * nrhs));
  cfg.blockDim = dim3(CT);
  cfg.dynamicSmemBytes = kClSmem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = CL;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int clusters = 0;
  ALDIC_CUDA(cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg));
  if (clusters < 1) return OK;  // no room for 16 neighbouring CTAs on this device
  ALDIC_CUDA(cudaLaunchKernelEx(&cfg, fn, A));
  *ran = true;
  return OK;
}

template <typename Rows>
int launch(ClArgs &A, long long n, int nrhs, cudaStream_t st, bool *ran) {
  *ran = false;
  if (n > (long long)CL * CT * kClMaxRows || nrhs > 6) return OK;
  A.n = (int)n;
  A.chunk = (int)((n + CL - 1) / CL);
  if (A.chunk <= CT) return launch_k<Rows, 1>(A, nrhs, st, ran);
  if (A.chunk <= 2 * CT) return launch_k<Rows, 2>(A, nrhs, st, ran);
  if (A.chunk <= 3 * CT) return launch_k<Rows, 3>(A, nrhs, st, ran);
  return launch_k<Rows, 4>(A, nrhs, st, ran);
}

}  // namespace

int cluster_csr(GridWork &w, const CsrOp &op, long long n, int nrhs, double rtol, int maxit,
                const double *beta_each, double mu, cudaStream_t st, bool *ran) {
  ClArgs A{};
  A.b = w.b; A.x = w.x; A.mask = w.mask;
  A.csr = op;
  for (int f = 0; f < 6 && f < nrhs; ++f) A.beta[f] = beta_each ? beta_each[f] : 0.0;
  A.mu = mu;
  A.rtol = rtol; A.maxit = maxit;
  A.iters_out = w.iters_out; A.err = w.err;
  return launch<CsrRows>(A, n, nrhs, st, ran);
}

int cluster_ata(GridWork &w, const double *ata, int M, int N, int nrhs, double lam2, double rtol, int maxit,
                cudaStream_t st, bool *ran) {
  ClArgs A{};
  A.b = w.b; A.x = w.x; A.mask = w.mask;
  A.ata = ata; A.M = M; A.N = N; A.lam2 = lam2;
  A.rtol = rtol; A.maxit = maxit;
  A.iters_out = w.iters_out; A.err = w.err;
  return launch<AtaRows>(A, (long long)M * N, nrhs, st, ran);
}

}  // namespace aldic
