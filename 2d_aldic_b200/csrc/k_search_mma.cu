// k_search_mma.cu -- the whole-field integer search of 8- and 16-bit images a
// grid point at a time, its correlation on the tensor cores (tcgen05 kind::i8,
// exact 32-bit sums).
//
// For one template row y the sums over shifts (a along x, b along y) are a
// product of two matrices,
//   D[a, b] += sum_k T_y[a, k] G[y + b, k],   T_y[a, k] = f[y][k - a],
// T_y a banded Toeplitz matrix of the template row, G the search region.  The
// region stays in shared memory once a point (K-major, 128-byte swizzle; rows
// y .. y + cc start y rows further down), the Toeplitz rows are built in
// registers and written to tensor memory, 128 lanes at once, so that the
// product reads one operand only from shared memory.  16-bit pixels are two
// byte planes: the lanes hold 64 shifts of the template's high bytes and 64 of
// its low bytes, the region's rows alternate between high and low bytes, and
// the four sums of a shift combine to the exact 64-bit one.
//
// A point (32 px subset, +-24 px, 16 bit: 33 rows x 3 K steps of 128 x 112 x 32)
// takes 99 products of 56 cycles; most of their work is zeros of the band
// (the sums need 11.3 M byte products, the tensor cores do 45 M), which is
// still 20 times the rate of the 16-bit dot products on the integer pipe.
//
// What bounds it: of a CTA's 33 k cycles a point, the building of the Toeplitz
// rows takes 14 k (funnel shifts and tensor memory writes of two warps a
// scheduler, the products 5.5 k beneath them), the estimates of the 2601
// entries 5.5 k, staging 5 k; two CTAs an SM overlap one's products and peak
// with the other's staging.  2048 x 2048, 13924 points, this geometry: 0.93 ms
// against 5.4 ms of a kernel of 16-bit dot products; 8 bit, subset 20, step
// 10, +-20 (2304 points): 0.092 ms against 0.27.  One template row a handover between
// builders and issuer was 1.2 ms, window sums in the kernel instead of the
// table 1.3 ms.
//
// Warps 0-3 and 4-7 build Toeplitz rows in turn, 8-11 meanwhile the sums of the
// template and of the windows that reach beyond the region (the map's outer
// ring; the others come from the window table), 12 issues the products.  0-11
// stage a point, read the sums back and estimate each correlation coefficient
// in FP32 from the exact integers (|error| < kMmaEps); those that can be the
// maximum go through a queue to warp 13, which evaluates them with ncc_combine,
// findpeak's 3 x 3 neighbourhood likewise, so the results are those of the
// full map, bit for bit; it does so while the others are at the next point.
#include <algorithm>
#include <type_traits>

#include "aldic_internal.cuh"
#include "kernels.cuh"
#include "ncc.cuh"
#include "search.cuh"
#include "tc.cuh"

namespace aldic {

namespace {

constexpr int kMmaWarps = 12, kMmaThreads = 32 * kMmaWarps, kMmaBlock = kMmaThreads + 64;
constexpr int kIssuer = kMmaWarps, kPeak = kMmaWarps + 1;
constexpr int kMmaQueue = 512;
constexpr float kMmaEps = 1e-5f;
constexpr size_t kMmaStatic = 8192;  // MmaShared, rounded up
constexpr int kMmaSlots = 2, kMmaMaxRows = 6;  // Toeplitz buffers, one a builder group; template rows of one at most

// Sizes of one geometry.  PL byte planes; a pass covers `lanes` shifts along x
// and `nb` along y.
struct MmaPlan {
  int pl, lanes, nb, px, py;  // passes along x and y: px, py
  int kb;                     // bytes of K (a multiple of 32)
  int ncol;                   // columns of the accumulator
  int nblk, rows;             // region: 128-byte blocks, rows of a block
  int fp;                     // bytes of a padded template row
  int trows, tcols;           // template rows of a Toeplitz buffer; tensor memory columns to allocate
  int gB, fB, ringB, ring2B, mapB, tabB, total;  // shared memory offsets
  int lineN;                  // entries of a line's prefix sums
  int ctas;                   // per SM
  bool fits;
};

__host__ __device__ inline int up(int v, int m) { return (v + m - 1) / m * m; }

MmaPlan mma_plan(const SearchGeom &G, int pl) {
  MmaPlan P{};
  P.pl = pl;
  P.lanes = 128 / pl;
  P.px = (G.cr + P.lanes - 1) / P.lanes;
  const int most = 256 / pl;
  P.py = (G.cc + most - 1) / most;
  P.nb = (G.cc + P.py - 1) / P.py;
  P.ncol = up(pl * P.nb, 16);
  P.kb = up(std::min(P.lanes, G.cr) + G.tw - 1, 32);
  P.nblk = ((P.px - 1) * P.lanes + P.kb + 127) / 128;
  P.rows = up(std::max(pl * G.dph, pl * (G.tw - 1 + (P.py - 1) * P.nb) + P.ncol), 8);
  P.fp = P.lanes + P.kb + 8;
  // as many template rows a buffer as tensor memory has room for beside the sums:
  // a handover between builders, issuer and back costs some 600 cycles
  const int row = P.kb / 4, need = P.ncol + kMmaSlots * row;
  P.tcols = need + kMmaSlots * row <= 256 ? 256 : 512;
  P.trows = std::min({kMmaMaxRows, G.tw, (P.tcols - P.ncol) / (kMmaSlots * row)});
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = (o + bytes + 127) & ~(size_t)127;
    return (int)at;
  };
  P.gB = take((size_t)P.nblk * P.rows * 128);
  P.fB = take((size_t)pl * G.tw * P.fp);
  const int line = std::max(G.dw, G.dh) + 3;  // prefix sums of the four lines the ring needs
  P.lineN = line;
  P.ringB = take(sizeof(int) * 4 * (size_t)line);
  P.ring2B = take((pl == 1 ? 4 : 8) * 4 * (size_t)line);
  P.mapB = take((pl == 1 ? 4 : 8) * (size_t)G.cr * G.cc);
  // two CTAs an SM where shared and tensor memory have the room; the point's
  // window table entries come along where they leave it
  auto fits = [&](size_t bytes, int ctas) { return ctas * (bytes + 1024 + kMmaStatic + 1024) <= kSmemMax + 1024; };
  const size_t core = o;
  const size_t table = sizeof(uint4) * (size_t)(G.cr - 2) * (G.cc - 2);
  P.ctas = P.tcols <= 256 && fits(core, 2) ? 2 : 1;
  P.tabB = -1;
  if (fits(core + table + 128, P.ctas)) P.tabB = take(table);
  P.total = (int)std::min<size_t>(o, 1 << 30);
  // sums below 2^31 in the accumulators, 64-bit products of the window sums
  P.fits = need <= 512 && fits(core, 1) && G.tw <= 128;
  return P;
}

struct MmaShared {
  uint64_t full[kMmaSlots], empty[kMmaSlots], done, drained;
  long long st, st2;
  long long part[4][2];            // a warp's share of st, st2
  int edge[4];                     // template sums: columns 0, tw - 1, rows 0, tw - 1
  int corner[2][2];                // its corner pixels [row][column]
  uint32_t tmem;
  unsigned int top;                // fkey of the largest estimate
  int nq, failed;
  int qi[kMmaQueue];
  float qe[kMmaQueue];
};

// kind::i8 instruction descriptor: D S32, A and B U8, both K-major
__device__ __forceinline__ constexpr uint32_t idesc_u8(int n) {
  return (2u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
}
__device__ __forceinline__ void mma_u8_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t id,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(db), "r"(id), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0));
}

// Four consecutive pixels from any address, read as aligned words
template <typename T>
struct Four {
  uint32_t w[2];  // the pixels, packed (8 bit: w[0])
  // skip: the first pixel is not wanted and its word not read unless it holds
  // the second one too
  __device__ __forceinline__ void load(const T *p, bool skip) {
    const uintptr_t a = (uintptr_t)p;
    const uint32_t *q = (const uint32_t *)(a & ~(uintptr_t)3);
    const uint32_t sh = 8 * (uint32_t)(a & 3);
    const bool first = !(skip && ((a + sizeof(T)) & 3) == 0);
    const uint32_t v0 = first ? q[0] : 0u, v1 = q[1];
    if (sizeof(T) == 1) {
      w[0] = __funnelshift_r(v0, v1, sh);
    } else {
      const uint32_t v2 = q[2];
      w[0] = __funnelshift_r(v0, v1, sh);
      w[1] = __funnelshift_r(v1, v2, sh);
    }
  }
  __device__ __forceinline__ uint32_t high() const { return sizeof(T) == 1 ? w[0] : __byte_perm(w[0], w[1], 0x7531); }
  __device__ __forceinline__ uint32_t low() const { return __byte_perm(w[0], w[1], 0x6420); }
};

// The outer ring of the map: entries of rows 0 and cc - 1, then of columns 0 and
// cr - 1 between them
__device__ __forceinline__ void ring_entry(int r, int cr, int cc, int *a, int *b) {
  if (r < 2 * cr) {
    *a = r < cr ? r : r - cr;
    *b = r < cr ? 0 : cc - 1;
  } else {
    r -= 2 * cr;
    *a = r < cc - 2 ? 0 : cr - 1;
    *b = (r < cc - 2 ? r : r - (cc - 2)) + 1;
  }
}

__device__ __forceinline__ void named_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// list: null, or {count, points...}
template <typename T>
__global__ void __launch_bounds__(kMmaBlock, 2)
    k_search_mma(const T *__restrict__ f, const T *__restrict__ g, const SearchGeom G, const MmaPlan P,
                 const uint4 *__restrict__ tab, const int *__restrict__ list, double *__restrict__ ox,
                 double *__restrict__ oy, double *__restrict__ ou, double *__restrict__ ov,
                 double *__restrict__ occ, int *__restrict__ err, const uint32_t tries) {
  constexpr int PL = sizeof(T);
  using Wide = typename std::conditional<PL == 1, int, long long>::type;  // sums of products
  extern __shared__ unsigned char mma_raw[];
  unsigned char *sm = (unsigned char *)(((uintptr_t)mma_raw + 1023) & ~(uintptr_t)1023);
  unsigned char *const Gs = sm + P.gB, *const Fs = sm + P.fB;
  int *const R1 = (int *)(sm + P.ringB);
  Wide *const R2 = (Wide *)(sm + P.ring2B), *const map = (Wide *)(sm + P.mapB);
  __shared__ MmaShared S;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int npts = list ? list[0] : G.nx * G.ny;
  if ((int)blockIdx.x >= npts) return;
  // a warp of a builder group holds 32 / PL shifts of every plane
  constexpr int kPer = 32 / PL;
  const int group = warp >> 2, plane = PL == 2 ? lane >> 4 : 0;
  const int d0 = kPer * (warp & 3), d = d0 + (lane & (kPer - 1));
  const int shifts = min(P.lanes, G.cr);  // of the first (widest) pass
  const bool builds = group < 2 && d0 < shifts;
  if (warp == 0) tmem_alloc(&S.tmem, P.tcols);
  if (tid == 0) {
    for (int s = 0; s < kMmaSlots; ++s) {
      bar_init(&S.full[s], (shifts + kPer - 1) / kPer);
      bar_init(&S.empty[s], 1);
    }
    bar_init(&S.done, 1);
    bar_init(&S.drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    S.top = 0u;
    S.nq = S.failed = 0;
  }
  // bytes outside the region and the template read 0 at every point
  for (int q = tid; q < P.nblk * P.rows * 32; q += kMmaBlock) ((uint32_t *)Gs)[q] = 0u;
  for (int q = tid; q < PL * G.tw * P.fp; q += kMmaBlock) Fs[q] = 0;
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const uint32_t tD = S.tmem, tA = tD + P.ncol;
  const int acols = P.kb / 4, steps = P.kb / 32;
  const int npass = P.px * P.py;
  const int rounds = (G.tw + P.trows - 1) / P.trows;
  const long long mn = (long long)G.tw * G.tw;
  const double mu = *G.mu;
  auto wait = [&](uint64_t *bar, uint32_t parity) {
    const bool ok = !*(volatile int *)&S.failed && bar_wait(bar, parity, tries);
    if (!ok) S.failed = 1;
    return ok;
  };
  auto pix = [&](int y, int x) {  // pixel of the padded region
    int v = 0;
#pragma unroll
    for (int p = 0; p < PL; ++p) {
      const int r = PL * y + p;
      v = 256 * v + Gs[((x >> 7) * P.rows + r) * 128 + ((((x & 127) >> 4) ^ (r & 7)) << 4) + (x & 15)];
    }
    return v;
  };
  // the point's window table entry of map entry (1, 1)
  auto window = [&](int pt) {
    const int ii = G.gx1 + pt % G.nx * G.step, jj = G.gy1 + pt / G.nx * G.step;
    return tab + (long long)(jj - 1 - G.sy) * G.W + (ii - 1 - G.sx);
  };
  auto squares = [](const uint4 &t) {
    return PL == 1 ? (long long)t.y : (long long)(((unsigned long long)t.z << 32) | t.y);
  };
  // window sums of map entry (a, b): the table's, or in the outer ring those of
  // the nearest full window less the column and the row (P, prefix sums of
  // line 0: column tw, 1: column cr - 2, 2: row tw, 3: row cc - 2) that it has
  // and the ring's has not
  struct Sums {
    int sd, st_out, n_out;
    Wide sd2;
  };
  auto sums = [&](const uint4 *win, long long pitch, int a, int b) {
    int st_out = 0, n_out = 0;
    const int oc = a == 0 ? 0 : (a == G.cr - 1 ? 1 : -1), orow = b == 0 ? 0 : (b == G.cc - 1 ? 1 : -1);
    const int af = min(max(a, 1), G.cr - 2), bf = min(max(b, 1), G.cc - 2);
    const uint4 t = win[(bf - 1) * pitch + af - 1];
    int sd = (int)t.x;
    Wide sd2 = (Wide)squares(t);
    if (oc >= 0) {
      const int at = oc * P.lineN + bf;
      sd -= R1[at + G.tw] - R1[at];
      sd2 -= R2[at + G.tw] - R2[at];
      st_out += S.edge[oc];
      n_out += G.tw;
    }
    if (orow >= 0) {
      const int at = (2 + orow) * P.lineN + a;
      sd -= R1[at + G.tw] - R1[at];
      sd2 -= R2[at + G.tw] - R2[at];
      st_out += S.edge[2 + orow];
      n_out += G.tw;
      if (oc >= 0) {
        st_out -= S.corner[orow][oc];
        n_out -= 1;
      }
    }
    return Sums{sd, st_out, n_out, sd2};
  };
  auto exact = [&](const uint4 *win, long long pitch, int a, int b) {
    const Sums u = sums(win, pitch, a, b);
    return ncc_combine(mn, S.st, S.st2, map[b * G.cr + a], u.sd, u.sd2, u.st_out, u.n_out, mu);
  };
  // the point's windows: staged in shared memory, or the table itself
  const bool staged = P.tabB >= 0;
  uint4 *const tabS = (uint4 *)(sm + (staged ? P.tabB : 0));
  const long long pitch = staged ? G.cr - 2 : G.W;

  if (uniform(warp) == kIssuer) {
    const uint32_t id = idesc_u8(P.ncol), uD = uniform(tD), uA = uD + P.ncol;
    uint32_t rc = 0;  // rounds so far: buffer rc & 1, its use rc >> 1
    for (int k = blockIdx.x; k < npts; k += gridDim.x)
      for (int ps = 0; ps < npass; ++ps) {
        const int x0 = (ps % P.px) * P.lanes, b0 = (ps / P.px) * P.nb;
        const uint64_t base = sdesc(uniform(smem_u32(Gs)) + ((x0 >> 7) * P.rows + PL * b0) * 128 + (x0 & 127));
        // K steps from `wrap` on are in the next block
        const int wrap = (128 - (x0 & 127)) / 32;
        const uint32_t skip = (P.rows * 128 - 128) / 16;
        for (int r = 0; r < rounds; ++r, ++rc) {
          const int s = rc & 1, y0 = r * P.trows;
          if (!__all_sync(0xffffffffu, wait(&S.full[s], (rc >> 1) & 1))) break;  // no more products
          tc_after_sync();
          // the rows' descriptors: 8 PL further (16-byte units) a template row, 2
          // a K step, another block after 128 bytes
          uint64_t db = base + (uint64_t)(PL * 8 * y0);
          uint32_t a = uA + s * P.trows * acols;
          if (elect_one()) {
            for (int h = 0; h < P.trows && y0 + h < G.tw; ++h, db += PL * 8, a += acols) {
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                if (q >= steps) break;
                mma_u8_ta(uD, a + 8 * q, db + 2 * q + (q >= wrap ? skip : 0u), id, y0 + h > 0 || q > 0);
              }
            }
            mma_commit(&S.empty[s]);
            if (r == rounds - 1) mma_commit(&S.done);
          }
          __syncwarp();
        }
      }
  } else if (warp == kPeak) {
    for (int k = blockIdx.x; k < npts; k += gridDim.x) {
      named_sync(4, kMmaThreads + 32);  // the queue is complete
      const int pt = list ? list[1 + k] : k;
      const uint4 *win = staged ? tabS : window(pt);
      const bool flat = mn * S.st2 - S.st * S.st == 0;
      double best = -1e300;
      int bi = 0;
      auto take = [&](int i) {
        const double v = exact(win, pitch, i % G.cr, i / G.cr);
        if (v > best || (v == best && i < bi)) {
          best = v;
          bi = i;
        }
      };
      auto reduce = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ob > best || (ob == best && oi < bi)) {
            best = ob;
            bi = oi;
          }
        }
      };
      const int nq = S.nq;
      const float top = fkey_inv(S.top);
      if (!flat) {
        if (nq <= kMmaQueue) {
          for (int q = lane; q < nq; q += 32)
            if (S.qe[q] >= top - 2.f * kMmaEps) take(S.qi[q]);
          reduce();
        }
        // more near-ties than the queue holds, or an estimate that met
        // ncc_combine's clamp of |r| > 1: the whole map
        if (nq > kMmaQueue || best < (double)top - kMmaEps) {
          best = -1e300;
          bi = 0;
          for (int i = lane; i < G.cr * G.cc; i += 32) take(i);
          reduce();
        }
      }
      const int r = bi % G.cr, c = bi / G.cr;
      double rpk = r + 1, cpk = c + 1, mf = best;
      if (!flat && r > 0 && r < G.cr - 1 && c > 0 && c < G.cc - 1) {
        double u9[9];
        const double mine = lane < 9 ? exact(win, pitch, r + lane % 3 - 1, c + lane / 3 - 1) : 0.0;
#pragma unroll
        for (int q = 0; q < 9; ++q) u9[q] = __shfl_sync(0xffffffffu, mine, q);
        findpeak_fit9(u9, r, c, &rpk, &cpk, &mf);
      }
      if (lane == 0) {
        // normxcorr2 rejects a constant template (funIntegerSearch.m:153-157)
        const bool none = flat || *(volatile int *)&S.failed;
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        const int ix = pt % G.nx, iy = pt / G.nx;
        const int ii = G.gx1 + ix * G.step, jj = G.gy1 + iy * G.step;
        const long long o = (long long)iy + (long long)ix * G.ny;
        ox[o] = (ii + ii + G.w) / 2.0;
        oy[o] = (jj + jj + G.w) / 2.0;
        ou[o] = none ? nan : __dsub_rn(rpk, (double)(G.sx + 2));
        ov[o] = none ? nan : __dsub_rn(cpk, (double)(G.sy + 2));
        occ[o] = none ? nan : mf;
        S.top = 0u;
        S.nq = 0;
      }
      __syncwarp();
      if (k + (int)gridDim.x < npts) {  // the next point may overwrite the sums and the map
        named_arrive(5, 128 + 32);
        named_arrive(6, 256 + 32);
      }
    }
  } else {
    uint32_t rc = 0, passes = 0;
    if (group == 0 && builds) {  // K steps outside a warp's band stay 0
      const uint32_t z[8] = {};
      for (int s = 0; s < kMmaSlots * P.trows; ++s)
        for (int q = 0; q < steps; ++q) tmem_st8(tA + s * acols + 8 * q + ((uint32_t)(32 * warp) << 16), z);
      tmem_st_wait();
      tc_before_sync();
    }
    const int q0 = d0 / 32, q1 = min(steps, (d0 + kPer - 1 + G.tw - 1) / 32 + 1);  // its band
    const int words = (G.dw + 4) / 4;  // of pixels 0 .. dw of a padded row
    const int twords = (G.tw + 3) / 4;
    for (int k = blockIdx.x; k < npts; k += gridDim.x) {
      const int pt = list ? list[1 + k] : k;
      const int ii = G.gx1 + pt % G.nx * G.step, jj = G.gy1 + pt / G.nx * G.step;  // 1-based
      // ---- stage the region (one pixel of zeros around it) and the template,
      // several loads in flight a thread
      const T *trow0 = f + (long long)(jj - 1) * G.W + (ii - 1);
      const T *drow0 = g + (long long)(jj - 1 - G.sy) * G.W + (ii - 1 - G.sx) - 1;
      constexpr int kUn = 3;
      for (int q = tid; q < G.dh * words; q += kUn * kMmaThreads) {
        Four<T> px[kUn];
        int yy[kUn], ww[kUn];
#pragma unroll
        for (int i = 0; i < kUn; ++i) {
          const int qi = q + i * kMmaThreads;
          yy[i] = qi / words;
          ww[i] = qi - yy[i] * words;
          // the first word's first pixel is the border: nothing before the row is read
          if (yy[i] < G.dh) px[i].load(drow0 + (long long)yy[i] * G.W + 4 * ww[i], ww[i] == 0);
        }
#pragma unroll
        for (int i = 0; i < kUn; ++i) {
          if (yy[i] >= G.dh) continue;
          uint32_t m = ww[i] == 0 ? 0xffffff00u : 0xffffffffu;
          if (ww[i] == words - 1) m &= 0xffffffffu >> (8 * (4 * words - 1 - G.dw));
          const int byte = 4 * ww[i], r = PL * (yy[i] + 1);
          unsigned char *o = Gs + ((byte >> 7) * P.rows + r) * 128 + (byte & 15);
          const int c = (byte & 127) >> 4;
          *(uint32_t *)(o + ((c ^ (r & 7)) << 4)) = px[i].high() & m;
          if (PL == 2) *(uint32_t *)(o + 128 + ((c ^ ((r + 1) & 7)) << 4)) = px[i].low() & m;
        }
      }
      for (int q = tid; q < G.tw * twords; q += kMmaThreads) {
        const int y = q / twords, w4 = q - y * twords;
        Four<T> px;
        px.load(trow0 + (long long)y * G.W + 4 * w4, false);
        const uint32_t m = w4 == twords - 1 ? 0xffffffffu >> (8 * (4 * twords - G.tw)) : 0xffffffffu;
        uint32_t *o = (uint32_t *)(Fs + y * P.fp + P.lanes) + w4;
        *o = px.high() & m;
        if (PL == 2) o[G.tw * P.fp / 4] = px.low() & m;
      }
      smem_to_async();
      named_sync(1, kMmaThreads);
      if (group == 2) {
        if (k != (int)blockIdx.x) named_sync(5, 128 + 32);  // the last point's peak is found
        if (staged) {  // the point's part of the window table
          const uint4 *win = window(pt);
          for (int b = warp - 8; b < G.cc - 2; b += 4)
            for (int a = lane; a < G.cr - 2; a += 32)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(tabS + b * (G.cr - 2) + a)),
                           "l"(win + (long long)b * G.W + a)
                           : "memory");
        }
        {  // a warp a line: its prefix sums
          const int l = warp - 8, len = l < 2 ? G.dh + 2 : G.dw + 2;
          const int fix = l == 0 || l == 2 ? G.tw : (l == 1 ? G.cr - 2 : G.cc - 2);
          int c1 = 0;
          Wide c2 = 0;
          int *r1 = R1 + l * P.lineN;
          Wide *r2 = R2 + l * P.lineN;
          if (lane == 0) {
            r1[0] = 0;
            r2[0] = 0;
          }
          for (int x0 = 0; x0 < len; x0 += 32) {
            const int x = x0 + lane;
            const int v = x < len ? (l < 2 ? pix(x, fix) : pix(fix, x)) : 0;
            int s1 = v;
            Wide s2 = (Wide)v * v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int t1 = __shfl_up_sync(0xffffffffu, s1, o);
              const Wide t2 = __shfl_up_sync(0xffffffffu, s2, o);
              if (lane >= o) {
                s1 += t1;
                s2 += t2;
              }
            }
            if (x < len) {
              r1[x + 1] = c1 + s1;
              r2[x + 1] = c2 + s2;
            }
            c1 += __shfl_sync(0xffffffffu, s1, 31);
            c2 += __shfl_sync(0xffffffffu, s2, 31);
          }
        }
        {  // template sums: four pixels a word, then an edge a warp
          unsigned sh = 0, sl = 0, hh = 0, hl = 0, ll = 0;
          for (int q = tid - 256; q < G.tw * twords; q += 128) {
            const int y = q / twords;
            const uint32_t *o = (const uint32_t *)(Fs + y * P.fp + P.lanes) + (q - y * twords);
            const uint32_t h = o[0];
            sh = __dp4a(h, 0x01010101u, sh);
            hh = __dp4a(h, h, hh);
            if (PL == 2) {
              const uint32_t l = o[G.tw * P.fp / 4];
              sl = __dp4a(l, 0x01010101u, sl);
              hl = __dp4a(h, l, hl);
              ll = __dp4a(l, l, ll);
            }
          }
          const long long s1 = warp_sum_ll(PL == 2 ? 256ll * sh + sl : (long long)sh);
          const long long s2 = warp_sum_ll(PL == 2 ? 65536ll * hh + 512ll * hl + ll : (long long)hh);
          const int l = warp - 8;  // column 0, column tw - 1, row 0, row tw - 1
          int e = 0;
          for (int t = lane; t < G.tw; t += 32) {
            const int y = l < 2 ? t : (l == 2 ? 0 : G.tw - 1), x = l >= 2 ? t : (l == 0 ? 0 : G.tw - 1);
            const unsigned char *o = Fs + y * P.fp + P.lanes + x;
            const int v = PL == 2 ? 256 * o[0] + o[G.tw * P.fp] : o[0];
            e += v;
            if (l >= 2 && (t == 0 || t == G.tw - 1)) S.corner[l - 2][t != 0] = v;
          }
          e = __reduce_add_sync(0xffffffffu, e);
          if (lane == 0) {
            S.part[l][0] = s1;
            S.part[l][1] = s2;
            S.edge[l] = e;
          }
          named_sync(3, 128);
          if (tid == 256) {
            S.st = (S.part[0][0] + S.part[1][0]) + (S.part[2][0] + S.part[3][0]);
            S.st2 = (S.part[0][1] + S.part[1][1]) + (S.part[2][1] + S.part[3][1]);
          }
        }
        if (staged) asm volatile("cp.async.wait_all;" ::: "memory");
      }
      for (int ps = 0; ps < npass; ++ps, ++passes) {
        // ---- Toeplitz rows of this warp's shifts: byte k of a lane's row is
        // template byte k - d
        const unsigned char *Fp = Fs + plane * G.tw * P.fp;
        const int at = P.lanes - d, sh = 8 * (at & 3);
        for (int r = 0; r < rounds; ++r, ++rc) {
          if (!builds || (int)(rc & 1) != group) continue;
          const int s = rc & 1, y0 = r * P.trows;
          const uint32_t use = rc >> 1;
          if (use) wait(&S.empty[s], (use - 1) & 1);
          tc_after_sync();
          const uint32_t *wd = (const uint32_t *)(Fp + y0 * P.fp) + (at >> 2);
          uint32_t t = tA + s * P.trows * acols + ((uint32_t)(32 * (warp & 3)) << 16);
#pragma unroll 1
          for (int h = 0; h < P.trows && y0 + h < G.tw; ++h, wd += P.fp / 4, t += acols) {
            int q = q0;
            for (; q + 1 < q1; q += 2) {
              uint32_t v[17], o[16];
#pragma unroll
              for (int e = 0; e < 17; ++e) v[e] = wd[8 * q + e];
#pragma unroll
              for (int e = 0; e < 16; ++e) o[e] = __funnelshift_r(v[e], v[e + 1], sh);
              __syncwarp();
              tmem_st16(t + 8 * q, o);
            }
            if (q < q1) {
              uint32_t v[9], o[8];
#pragma unroll
              for (int e = 0; e < 9; ++e) v[e] = wd[8 * q + e];
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = __funnelshift_r(v[e], v[e + 1], sh);
              __syncwarp();
              tmem_st8(t + 8 * q, o);
            }
          }
          tmem_st_wait();
          tc_before_sync();
          __syncwarp();
          if (lane == 0) bar_arrive(&S.full[s]);
        }
        // ---- the pass's sums, a third of the rows a group: column PL b + plane
        // of the region, lanes as built
        if (ps == 0 && group < 2 && k != (int)blockIdx.x) named_sync(6, 256 + 32);
        wait(&S.done, passes & 1);
        tc_after_sync();
        const int a = (ps % P.px) * P.lanes + d, b0 = (ps / P.px) * P.nb;
        const int nb = min(P.nb, G.cc - b0);
        constexpr int kEach = 16 / PL;  // rows of the map a load covers
        for (int b = kEach * group; d0 < shifts && b < nb; b += 3 * kEach) {
          float raw[16];
          __syncwarp();
          tmem_ld16(tD + ((uint32_t)(32 * (warp & 3)) << 16) + PL * b, raw);
          if (PL == 1) {
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (b + e < nb && a < G.cr) map[(b0 + b + e) * G.cr + a] = (Wide)__float_as_uint(raw[e]);
          } else {
            // lanes below 16 (high template bytes) finish rows e, the others e + 1
#pragma unroll
            for (int e = 0; e < kEach; e += 2) {
              const uint32_t h0 = __float_as_uint(raw[2 * e]), l0 = __float_as_uint(raw[2 * e + 1]);
              const uint32_t h1 = __float_as_uint(raw[2 * e + 2]), l1 = __float_as_uint(raw[2 * e + 3]);
              const uint32_t oh = __shfl_xor_sync(0xffffffffu, plane ? h0 : h1, 16);
              const uint32_t ol = __shfl_xor_sync(0xffffffffu, plane ? l0 : l1, 16);
              // template high x region high, high x low, low x high, low x low
              const uint32_t hh = plane ? oh : h0, hl = plane ? ol : l0;
              const uint32_t lh = plane ? h1 : oh, ll = plane ? l1 : ol;
              const int be = b + e + plane;
              if (be < nb && a < G.cr)
                map[(b0 + be) * G.cr + a] =
                    (Wide)(((unsigned long long)hh << 16) + ((unsigned long long)(hl + lh) << 8) + ll);
            }
          }
        }
        tc_before_sync();
        named_sync(1, kMmaThreads);
      }
      // ---- estimates: the interior from the window table, then the ring
      const uint4 *win = staged ? tabS : window(pt);
      const float denf = (float)(mn * S.st2 - S.st * S.st), rt = rsqrtf(denf);
      const int st = (int)S.st;
      float least = -2.f;  // entries below it cannot be the maximum
      auto offer = [&](float e, int i) {  // all lanes of the warp; -3: no entry
        if (!__any_sync(0xffffffffu, e >= least)) return;
        const unsigned int best = __reduce_max_sync(0xffffffffu, fkey(e));
        unsigned int top = *(volatile unsigned int *)&S.top;
        if (best > top) {
          if (lane == 0) atomicMax(&S.top, best);
          top = best;
        }
        least = fkey_inv(top) - 2.f * kMmaEps;
        const bool keep = e >= least;
        const unsigned int m = __ballot_sync(0xffffffffu, keep);
        if (m) {
          int at = 0;
          if (lane == 0) at = atomicAdd(&S.nq, __popc(m));
          at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1));
          if (keep && at < kMmaQueue) {
            S.qi[at] = i;
            S.qe[at] = e;
          }
        }
      };
      for (int b = 1 + warp; b < G.cc - 1; b += kMmaWarps)
        for (int a = 1 + lane; a - lane < G.cr - 1; a += 32) {
          const bool in = a < G.cr - 1;
          const uint4 t = in ? win[(b - 1) * pitch + a - 1] : make_uint4(0, 0, 0, 0);
          const long long num = in ? mn * map[b * G.cr + a] - (long long)st * (int)t.x : 0;
          const float e = (float)num * (__uint_as_float(PL == 1 ? t.z : t.w) * rt);
          offer(in ? e : -3.f, b * G.cr + a);
        }
      for (int r0 = 32 * warp; r0 < 2 * (G.cr + G.cc) - 4; r0 += kMmaThreads) {
        const int r = r0 + lane;
        const bool in = r < 2 * (G.cr + G.cc) - 4;
        int a = 0, b = 0;
        ring_entry(in ? r : 0, G.cr, G.cc, &a, &b);
        const Sums u = sums(win, pitch, a, b);
        double num, den;
        ncc_parts(mn, S.st, map[b * G.cr + a], u.sd, u.sd2, u.st_out, u.n_out, mu, &num, &den);
        const float e = den > 0.0 ? (float)num * rsqrtf(denf * (float)den) : 0.f;
        offer(in ? e : -3.f, b * G.cr + a);
      }
      named_sync(4, kMmaThreads + 32);
    }
  }
  tc_before_sync();
  __syncthreads();
  if (S.failed) {  // the products under way end before the tensor memory goes
    if (uniform(warp) == kIssuer) {
      if (elect_one()) mma_commit(&S.drained);
      __syncwarp();
      bar_wait(&S.drained, 0);
    }
    if (tid == 0) atomicExch(err, 3);
    __syncthreads();
  }
  if (warp == 0) tmem_free(tD, P.tcols);
}

}  // namespace

bool search_mma_fits(const SearchGeom &G, int bytes) { return bytes <= 2 && mma_plan(G, bytes).fits; }

template <typename T>
int search_mma(const T *f, const T *g, const SearchGeom &G, const uint4 *tab, const int *list, double *x,
               double *y, double *u, double *v, double *cc, int *err, unsigned tries, cudaStream_t st) {
  const MmaPlan P = mma_plan(G, sizeof(T));
  const int smem = P.total + 1024;
  int dev = 0, sms = 148;
  ALDIC_CUDA(cudaGetDevice(&dev));
  ALDIC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  ALDIC_CUDA(cudaFuncSetAttribute(k_search_mma<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const long long npts = (long long)G.nx * G.ny;
  const int blocks = (int)std::min<long long>(npts, (long long)P.ctas * sms);
  k_search_mma<T><<<blocks, kMmaBlock, smem, st>>>(f, g, G, P, tab, list, x, y, u, v, cc, err, tries);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}
template int search_mma<uint8_t>(const uint8_t *, const uint8_t *, const SearchGeom &, const uint4 *, const int *,
                                 double *, double *, double *, double *, double *, int *, unsigned, cudaStream_t);
template int search_mma<uint16_t>(const uint16_t *, const uint16_t *, const SearchGeom &, const uint4 *, const int *,
                                  double *, double *, double *, double *, double *, int *, unsigned, cudaStream_t);

}  // namespace aldic
