// k_net.cu -- the forward pass of the learned initial guess (cnn.cu) in two
// tensor-core kernels:
//   k_encode  per patch pair: 8x8 patch embedding (ReLU) and 1x1 layer of both
//             patches' 64 cells and the 64 x 64 correlation of their features
//   k_dense   the 4096 -> 256 layer (ReLU) and the FP32 256 -> 8 output
// The activations between the three products of k_encode never leave the SM:
// a pair is 64 + 64 cells, one 128-row tile.  Run apart (a generic GEMM per
// layer) they moved 4 x 512 B per cell through memory and spent their time
// staging operands.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "aldic_internal.cuh"
#include "kernels.cuh"
#include "tc.cuh"

namespace aldic {

namespace {

using bf16 = __nv_bfloat16;

constexpr int kPx = 64 * 64, kCells = 64, kC = 128, kCorr = kCells * kCells, kF = 256, kOut = 8;

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
// the same with negative values and NaN to 0 (cvt's own relu keeps NaN)
__device__ __forceinline__ uint32_t pack2_relu(float a, float b) {
  uint32_t r;
  asm("{\n\t.reg .b32 t;\n\tcvt.rn.bf16x2.f32 t, %1, %2;\n\tmax.bf16x2 %0, t, %3;\n\t}" : "=r"(r) : "f"(b), "f"(a), "r"(0));
  return r;
}

// both sums in one instruction (16384 pairs: 233 us the call with two, 222 so)
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// byte offset of 16-byte chunk c of row r in a tile of 128-byte rows, 128-byte swizzle
__device__ __forceinline__ uint32_t swz(int r, int c) { return r * 128 + ((c ^ (r & 7)) << 4); }

// ------------------------------------------------------------------ k_encode
// A CTA takes pairs from its stride, two CTAs an SM so that one's epilogue
// runs under the other's products.  Per pair:
//   A0 [128 x 64]  . W1^T -> D   embedding: rows 0..63 the reference's cells,
//                                64..127 the deformed patch's
//   E  [128 x 128] = relu(D + b1) in bf16,  E . W2^T -> D
//   E = D + b2 in bf16,  E . G^T -> C [128 x 64] with G = E[64..127]; rows
//   0..63 are the correlation
// The left operand E stays in tensor memory (64 columns), so that the products
// and the epilogues, which share the SM's shared-memory bandwidth, move 80 KB
// a pair through it for the products instead of 144: a 128 x 128 product with
// both operands in shared memory reads 128 B a cycle, all there is.  G, A0 (16
// KB each) and the weights (48 KB) are there.  The pair's 16 KB are loaded a
// pair ahead, and the next embedding is issued with the correlation.  Eight
// warps do the epilogues; a ninth only issues the products.
// Tensor memory: D 128, C 64, E 64 columns.  16384 pairs: 161 us (ncu), against
// 62 us for their 24 KB each at the copy rate and 68 us for the products; a
// pair's chain of three products and three epilogues is what is left (two CTAs
// an SM hide half of it; 512 epilogue threads a CTA measured 6 % slower).  The
// layers as separate products took 2.05 ms.
constexpr int kEncThreads = 256, kEncBlock = kEncThreads + 32;

struct EncArgs {
  const bf16 *x;            // [B][64][64][2] bf16
  const bf16 *W1, *W2;      // [128][64], [128][128]
  const float *b1, *b2;
  bf16 *e1, *e2;            // training: [2B][64][128], else null
  int B;
  float scale;
  int *err;
};

struct EncShared {
  unsigned char A0[128 * 128];
  uint4 x[kPx / 4];                  // a pair as it comes, both channels interleaved
  unsigned char G[2][kCells * 128];  // two K blocks of 64
  unsigned char out[kCells * 128];   // the correlation on its way to memory
  unsigned char W1[128 * 128];
  unsigned char W2[2][128 * 128];
  uint64_t bar[5];                   // embedding, 1x1, correlation; x has landed; all products ended
  uint32_t tmem;
  int failed;
};

__global__ void __launch_bounds__(kEncBlock, 2) k_encode(const __grid_constant__ CUtensorMap mC,
                                                         const EncArgs A) {
  extern __shared__ unsigned char enc_raw[];
  EncShared &S = *(EncShared *)(((uintptr_t)enc_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int q = tid; q < 128 * 8; q += kEncBlock) {
    const int r = q >> 3, c = q & 7;
    *(uint4 *)(S.W1 + swz(r, c)) = *(const uint4 *)(A.W1 + r * 64 + 8 * c);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb)
      *(uint4 *)(S.W2[kb] + swz(r, c)) = *(const uint4 *)(A.W2 + r * 128 + 64 * kb + 8 * c);
  }
  if (warp == 0) tmem_alloc(&S.tmem, 256);
  if (tid == 0) {
    S.failed = 0;
    for (int k = 0; k < 5; ++k) bar_init(&S.bar[k], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // this warp's quarter of the tensor memory's lanes (rows) and half of the
  // columns.  Tensor memory is read 16 rows at a time so that a thread holds
  // few columns of many rows (lane / 4 and 8 below it; 8 j + 2 (lane % 4) and
  // its neighbour): its 2 x 16 biases fit in registers.  A row a thread
  // needs every bias from shared memory, a quarter of the kernel's time.
  const int quarter = warp & 3, half = (warp >> 2) & 1;
  const int col2 = 2 * (lane & 3);
  float2 b1[8], b2[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    b1[j] = *(const float2 *)(A.b1 + 64 * half + 8 * j + col2);
    b2[j] = *(const float2 *)(A.b2 + 64 * half + 8 * j + col2);
  }
  auto load = [&](int p) {  // one thread: a pair in one copy
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&S.bar[3])),
                 "r"((uint32_t)sizeof(S.x))
                 : "memory");
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(S.x)),
                 "l"(A.x + (long long)p * (2 * kPx)), "r"((uint32_t)sizeof(S.x)), "r"(smem_u32(&S.bar[3]))
                 : "memory");
  };
  auto stage = [&]() {  // four pixels of both channels: 8 bytes of an f row and of a g row
#pragma unroll
    for (int i = 0; i < kPx / 4 / kEncThreads; ++i) {
      const int p = 4 * (tid + kEncThreads * i), y = p >> 6, c = p & 63;
      const int cell = (y >> 3) * 8 + (c >> 3);
      const uint32_t o = swz(cell, y & 7) + (c & 7) * 2;
      const uint4 v = S.x[tid + kEncThreads * i];
      *(uint2 *)(S.A0 + o) = make_uint2(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410));
      *(uint2 *)(S.A0 + o + kCells * 128) = make_uint2(__byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x7632));
    }
  };
  int b = blockIdx.x;
  const bool issuer = uniform(warp) == kEncThreads / 32;
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  if (issuer && lane == 0) load(b);
  if (!bar_wait(&S.bar[3], 0)) S.failed = 1;
  if (!issuer) stage();
  smem_to_async();
  __syncthreads();
  const uint32_t tD = uniform(S.tmem), tC = tD + 128, tE = tD + 192;
  const uint32_t sA0 = uniform(smem_u32(S.A0)), sW1 = uniform(smem_u32(S.W1));
  const uint32_t sW2 = uniform(smem_u32(S.W2[0])), sG = uniform(smem_u32(S.G[0]));
  auto embed = [&]() {
    const uint64_t da = sdesc(sA0), db = sdesc(sW1);
#pragma unroll
    for (int k = 0; k < 4; ++k) mma_bf16(tD, da + 2 * k, db + 2 * k, idesc(128), k > 0);
    mma_commit(&S.bar[0]);
  };
  // D (+ bias, ReLU) -> E in bf16, the deformed patch's rows also to G; and to
  // memory when trained on (pair p)
  auto to_E = [&](const float2 *bias, bool relu, bool toG, bf16 *g, int p) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t lanes = (uint32_t)(32 * quarter + 16 * h) << 16;
      const int row = 32 * quarter + 16 * h + (lane >> 2);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float v[16];
        uint32_t w[8];
        tmem_ld_16x32(tD + lanes + 64 * half + 32 * q, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 bb = bias[4 * q + j];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float2 x = add2(make_float2(v[4 * j + 2 * k], v[4 * j + 2 * k + 1]), bb);
            w[2 * j + k] = relu ? pack2_relu(x.x, x.y) : pack2(x.x, x.y);
          }
        }
        tmem_st_16x16(tE + lanes + 32 * half + 16 * q, w);
        if (toG && quarter >= 2) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k)
              *(uint32_t *)(S.G[half] + swz(row - kCells + 8 * k, 4 * q + j) + 2 * col2) = w[2 * j + k];
        }
        if (g) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int r = row + 8 * k;
            const long long cell = (r < kCells ? (long long)p : (long long)A.B + p) * kCells + (r & 63);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              *(uint32_t *)(g + cell * kC + 64 * half + 32 * q + 8 * j + col2) = w[2 * j + k];
          }
        }
      }
    }
    tmem_st_wait();
  };
  // the correlation in `out` to its place; the issuing thread
  auto store = [&](int p) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(&mC),
                 "r"(smem_u32(S.out)), "r"(0), "r"(p * kCells)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  };
  if (S.failed) {
    // the copy never came; nothing else is under way
  } else if (issuer) {
    uint32_t got = 0;  // parity of the last copy waited for
    if (elect_one()) {
      embed();
      if (b + (int)gridDim.x < A.B) load(b + gridDim.x);
    }
    __syncwarp();
    const int b0 = b;
    for (; b < A.B; b += gridDim.x) {
      __syncthreads();
      if (S.failed) break;
      tc_after_sync();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          mma_bf16_ta(tD, tE + 8 * k, sdesc(sW2 + (k >> 2) * (128 * 128)) + 2 * (k & 3), idesc(128), k > 0);
        mma_commit(&S.bar[1]);
        if (b > b0) {  // the previous pair's correlation; `out` is free again at the next barrier
          store(b - gridDim.x);
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
      }
      __syncwarp();
      __syncthreads();
      if (S.failed) break;
      tc_after_sync();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          mma_bf16_ta(tC, tE + 8 * k, sdesc(sG + (k >> 2) * (kCells * 128)) + 2 * (k & 3), idesc(64), k > 0);
        mma_commit(&S.bar[2]);
        if (b + (int)gridDim.x < A.B) embed();
        if (b + 2 * (int)gridDim.x < A.B) load(b + 2 * gridDim.x);
      }
      __syncwarp();
      got ^= 1;
    }
    // after a failed wait: the copy under way must land before the CTA ends
    if (S.failed && b + (int)gridDim.x < A.B) bar_wait(&S.bar[3], got ^ 1);
  } else {
    uint32_t ph = 0;
    for (; b < A.B; b += gridDim.x, ph ^= 1) {
      if (!bar_wait(&S.bar[0], ph)) S.failed = 1;
      tc_after_sync();
      to_E(b1, true, false, A.e1, b);
      smem_to_async();
      tc_before_sync();
      __syncthreads();
      if (S.failed) break;
      if (b + (int)gridDim.x < A.B) {  // A0 is free: its product is done
        if (!bar_wait(&S.bar[3], ph ^ 1)) S.failed = 1;
        stage();
      }
      if (!bar_wait(&S.bar[1], ph)) S.failed = 1;
      tc_after_sync();
      to_E(b2, false, true, A.e2, b);
      smem_to_async();
      tc_before_sync();
      __syncthreads();
      if (S.failed) break;
      if (!bar_wait(&S.bar[2], ph)) S.failed = 1;
      tc_after_sync();
      if (quarter < 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float v[16];
          tmem_ld_16x32(tC + ((uint32_t)(32 * quarter + 16 * h) << 16) + 32 * half, v);
          const int row = 32 * quarter + 16 * h + (lane >> 2);
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k)
              *(uint32_t *)(S.out + swz(row + 8 * k, 4 * half + j) + 2 * col2) =
                  pack2(v[4 * j + 2 * k] * A.scale, v[4 * j + 2 * k + 1] * A.scale);
        }
      }
    }
    smem_to_async();  // the last correlation
  }
  tc_before_sync();
  __syncthreads();
  if (S.failed) {  // the products under way end before the tensor memory goes
    if (issuer) {
      if (elect_one()) mma_commit(&S.bar[4]);
      __syncwarp();
      bar_wait(&S.bar[4], 0);
    }
    __syncthreads();
  }
  if (issuer && lane == 0) {
    if (!S.failed) store(blockIdx.x + (A.B - 1 - (int)blockIdx.x) / (int)gridDim.x * (int)gridDim.x);
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (S.failed) atomicExch(A.err, 3);
  }
  if (warp == 0) tmem_free(S.tmem, 256);
}

// ------------------------------------------------------------------ k_dense
// y[B x 256] = relu(corr[B x 4096] . W3^T + b3), out = y . W4^T + b4.  The K range
// is summed in eight slices of 512, each in the tensor core's accumulator, and the
// slices are added in FP32 in their order: the accumulator does not round every
// addition to nearest, so a chain of 4096 loses more than eight of 512, and with
// the same slices for every batch a pair's output does not depend on the batch it
// comes in.  One CTA per 128 rows, all 256 columns: 64-wide K steps of both
// operands by TMA into a ring of four stages (one thread), products issued by
// another, a slice's 256 tensor memory columns read by eight warps (a row and half
// of the columns a thread, their sums in its registers) under the next slice's
// products.  With too few row tiles for the SMs (PART) each slice has a CTA of its own,
// blockIdx.y, and k_dense_out adds them; otherwise the epilogue goes on to the output
// layer, the second half of a row's sums after the first.
// Bound: 48 KB of operands a step and SM through L2 (corr once, W3 by every
// tile).  16384 rows: 47.6 us (ncu), 0.72 PFLOP/s; 50.2 us with one chain of 4096 read
// by four warps at its end; the generic product with its split-K sum and the output layer
// took 560 us.
constexpr int kDenseStages = 4, kDenseStage = (128 + kF) * 128, kDenseThreads = 64 + 256;
constexpr int kDenseSlices = 8, kSliceSteps = kCorr / 64 / kDenseSlices;

struct DenseArgs {
  const float *b3, *W4, *b4;
  bf16 *y;
  float *out, *part;         // part: [kDenseSlices][B][256] of PART
  int B;
  int *err;
};

struct DenseShared {
  float W4[kF][kOut], b3[kF], b4[kOut];
  float o[kOut][128];        // the output layer's sums over the first half of a row
  uint64_t full[kDenseStages], empty[kDenseStages];
  uint64_t done[2], read[2]; // a slice's sums are there, and have been read
  uint32_t tmem;
  int failed;
};

__device__ __forceinline__ void tma_2d(const CUtensorMap *m, uint32_t dst, uint64_t *bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(m), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

template <bool PART>
__global__ void __launch_bounds__(kDenseThreads, 1) k_dense(const __grid_constant__ CUtensorMap mA,
                                                            const __grid_constant__ CUtensorMap mB,
                                                            const DenseArgs A) {
  extern __shared__ unsigned char dense_raw[];
  unsigned char *ring = (unsigned char *)(((uintptr_t)dense_raw + 1023) & ~(uintptr_t)1023);
  DenseShared &S = *(DenseShared *)(ring + kDenseStages * kDenseStage);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int slices = PART ? 1 : kDenseSlices, steps = slices * kSliceSteps;
  const int m0 = blockIdx.x * 128, z0 = blockIdx.y;
  if (warp == 0) tmem_alloc(&S.tmem, 2 * kF);
  if (tid == 0) {
    S.failed = 0;
    for (int s = 0; s < kDenseStages; ++s) {
      bar_init(&S.full[s], 1);
      bar_init(&S.empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      bar_init(&S.done[s], 1);
      bar_init(&S.read[s], 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int q = tid; q < kF * kOut; q += kDenseThreads) S.W4[q % kF][q / kF] = A.W4[q];
  for (int q = tid; q < kF; q += kDenseThreads) S.b3[q] = A.b3[q];
  if (tid < kOut) S.b4[tid] = A.b4[tid];
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const uint32_t tD = uniform(S.tmem);
  if (warp == 0) {
    if (lane == 0) {
      int k = 0;
      for (; k < steps; ++k) {
        const int s = k % kDenseStages;
        if (k >= kDenseStages && !bar_wait(&S.empty[s], (k / kDenseStages - 1) & 1)) {
          S.failed = 1;
          break;
        }
        const uint32_t a = smem_u32(ring + s * kDenseStage);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&S.full[s])),
                     "r"(kDenseStage)
                     : "memory");
        tma_2d(&mA, a, &S.full[s], 64 * (z0 * kSliceSteps + k), m0);
        tma_2d(&mB, a + 128 * 128, &S.full[s], 64 * (z0 * kSliceSteps + k), 0);
      }
      // every copy has landed before the CTA may end, also after a failed wait
      for (int q = k > kDenseStages ? k - kDenseStages : 0; q < k; ++q)
        if (!bar_wait(&S.full[q % kDenseStages], (q / kDenseStages) & 1)) S.failed = 1;
    }
  } else if (uniform(warp) == 1) {
    const uint32_t base = uniform(smem_u32(ring));
    bool ok = true;
    for (int z = 0, k = 0; z < slices && ok; ++z) {
      const uint32_t d = tD + (z & 1) * kF;
      if (z >= 2) {  // the slice before last has been read
        ok = __all_sync(0xffffffffu, bar_wait(&S.read[z & 1], ((z >> 1) - 1) & 1));
        tc_after_sync();
      }
      for (int q8 = 0; q8 < kSliceSteps && ok; ++q8, ++k) {
        const int s = k % kDenseStages;
        ok = __all_sync(0xffffffffu, bar_wait(&S.full[s], (k / kDenseStages) & 1));
        if (!ok) break;
        tc_after_sync();
        const uint64_t da = sdesc(base + s * kDenseStage), db = sdesc(base + s * kDenseStage + 128 * 128);
        if (elect_one()) {
#pragma unroll
          for (int q = 0; q < 4; ++q) mma_bf16(d, da + 2 * q, db + 2 * q, idesc(kF), q8 > 0 || q > 0);
          mma_commit(&S.empty[s]);
        }
        __syncwarp();
      }
      if (!ok) S.failed = 1;
      if (elect_one()) mma_commit(&S.done[z & 1]);
      __syncwarp();
      // after a failed wait: no product is under way when the CTA ends
      if (!ok) bar_wait(&S.done[z & 1], (z >> 1) & 1);
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2, row = 32 * quarter + lane, m = m0 + row;
    const uint32_t t = tD + ((uint32_t)(32 * quarter) << 16) + half * (kF / 2);
    float sum[PART ? 1 : kF / 2] = {};
    bool ok = true;
    for (int z = 0; z < slices && ok; ++z) {
      ok = __all_sync(0xffffffffu, bar_wait(&S.done[z & 1], (z >> 1) & 1) && !*(volatile int *)&S.failed);
      if (!ok) break;
      tc_after_sync();
#pragma unroll
      for (int c = 0; c < kF / 2; c += 16) {
        float v[16];
        tmem_ld16(t + (z & 1) * kF + c, v);
        if constexpr (PART) {
          if (m < A.B) {
            float4 *p = (float4 *)(A.part + ((long long)z0 * A.B + m) * kF + half * (kF / 2) + c);
#pragma unroll
            for (int k = 0; k < 4; ++k) p[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
          }
          __syncwarp();
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k) sum[c + k] += v[k];
        }
      }
      tc_before_sync();
      __syncwarp();
      if (lane == 0) bar_arrive(&S.read[z & 1]);
    }
    if (!ok) S.failed = 1;
    if constexpr (!PART) {
      float o[kOut];
#pragma unroll
      for (int k = 0; k < kOut; ++k) o[k] = S.b4[k];
      if (half) {
        named_sync(1 + quarter, 64);  // the first half's sums
#pragma unroll
        for (int k = 0; k < kOut; ++k) o[k] = S.o[k][row];
      }
#pragma unroll
      for (int c = 0; c < kF / 2; c += 8) {
        const int n = half * (kF / 2) + c;
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          w[k] = pack2(fmaxf(sum[c + 2 * k] + S.b3[n + 2 * k], 0.f), fmaxf(sum[c + 2 * k + 1] + S.b3[n + 2 * k + 1], 0.f));
        if (ok && m < A.B) *(uint4 *)(A.y + (long long)m * kF + n) = make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float y = __uint_as_float(k & 1 ? w[k >> 1] & 0xffff0000u : w[k >> 1] << 16);
          const float4 wa = *(const float4 *)&S.W4[n + k][0], wb = *(const float4 *)&S.W4[n + k][4];
          o[0] += y * wa.x; o[1] += y * wa.y; o[2] += y * wa.z; o[3] += y * wa.w;
          o[4] += y * wb.x; o[5] += y * wb.y; o[6] += y * wb.z; o[7] += y * wb.w;
        }
      }
      if (!half) {
#pragma unroll
        for (int k = 0; k < kOut; ++k) S.o[k][row] = o[k];
        named_sync(1 + quarter, 64);
      } else if (ok && m < A.B) {
        float4 *p = (float4 *)(A.out + (long long)m * kOut);
        p[0] = make_float4(o[0], o[1], o[2], o[3]);
        p[1] = make_float4(o[4], o[5], o[6], o[7]);
      }
    }
  }
  tc_before_sync();
  __syncthreads();
  if (tid == 0 && S.failed) atomicExch(A.err, 3);
  if (warp == 0) tmem_free(tD, 2 * kF);
}

// the slices of the layer added in their order; a warp a row, 8 columns a lane,
// then a thread an output of the block's four rows
__global__ void __launch_bounds__(128) k_dense_out(const DenseArgs A) {
  __shared__ float W4[kOut][kF + 1], y[4][kF];
  for (int q = threadIdx.x; q < kF * kOut; q += 128) W4[q / kF][q % kF] = A.W4[q];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.x * 4 + warp;
  if (b < A.B) {
    float s[8] = {};
#pragma unroll
    for (int z = 0; z < kDenseSlices; ++z) {
      const float4 *p = (const float4 *)(A.part + ((long long)z * A.B + b) * kF + 8 * lane);
      const float4 u = p[0], v = p[1];
      s[0] += u.x; s[1] += u.y; s[2] += u.z; s[3] += u.w;
      s[4] += v.x; s[5] += v.y; s[6] += v.z; s[7] += v.w;
    }
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      w[k] = pack2(fmaxf(s[2 * k] + A.b3[8 * lane + 2 * k], 0.f), fmaxf(s[2 * k + 1] + A.b3[8 * lane + 2 * k + 1], 0.f));
    *(uint4 *)(A.y + (long long)b * kF + 8 * lane) = make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      y[warp][8 * lane + k] = __uint_as_float(k & 1 ? w[k >> 1] & 0xffff0000u : w[k >> 1] << 16);
  }
  __syncthreads();
  const int r = threadIdx.x / kOut, o = threadIdx.x % kOut, m = blockIdx.x * 4 + r;
  if (r >= 4 || m >= A.B) return;
  float t = A.b4[o];
#pragma unroll 16
  for (int k = 0; k < kF; ++k) t += y[r][k] * W4[o][k];
  A.out[(long long)m * kOut + o] = t;
}

// rows x cols bf16 matrix, boxes of `box` rows x 64 columns in the 128-byte swizzle
int make_map(CUtensorMap *m, const void *p, long long rows, long long cols, int box) {
  using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);
  static const Encode enc = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return (Encode)f;
  }();
  ALDIC_CHECK(enc, E_CUDA, "the driver has no cuTensorMapEncodeTiled");
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t b[2] = {64, (cuuint32_t)box}, es[2] = {1, 1};
  ALDIC_CHECK(enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(p), dims, strides, b, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
              E_CUDA, "tensor map refused");
  return OK;
}

int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace

int net_encode(const void *x, int B, const void *W1, const float *b1, const void *W2, const float *b2,
               float scale, void *corr, void *e1, void *e2, int *err, cudaStream_t st) {
  CUtensorMap mC;
  int rc = make_map(&mC, corr, (long long)B * kCells, kCells, kCells);
  if (rc) return rc;
  EncArgs A;
  A.x = (const bf16 *)x;
  A.W1 = (const bf16 *)W1; A.W2 = (const bf16 *)W2; A.b1 = b1; A.b2 = b2;
  A.e1 = (bf16 *)e1; A.e2 = (bf16 *)e2;
  A.B = B; A.scale = scale; A.err = err;
  const int smem = sizeof(EncShared) + 1024;
  ALDIC_CUDA(cudaFuncSetAttribute(k_encode, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int grid = 2 * sm_count();
  k_encode<<<B < grid ? B : grid, kEncBlock, smem, st>>>(mC, A);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

// A CTA a slice while all of them run at once; beyond, the partials' way through
// memory costs more than idle SMs (whole predictions, a CTA a slice against all: 256
// pairs 56 / 64 us, 2048 74 / 83, 2500 88 / 83, 4096 111 / 108, 9000 197 / 152; two
// or four slices a CTA lie between or above).
bool dense_apart(int B) { return (B + 127) / 128 * kDenseSlices <= 148; }

size_t net_dense_part(int B) { return dense_apart(B) ? sizeof(float) * kDenseSlices * kF * (size_t)B : 0; }

int net_dense(const void *corr, int B, const void *W3, const float *b3, const float *W4, const float *b4,
              void *y, float *out, float *part, int *err, cudaStream_t st) {
  CUtensorMap mA, mB;
  int rc;
  if ((rc = make_map(&mA, corr, B, kCorr, 128)) || (rc = make_map(&mB, W3, kF, kCorr, kF))) return rc;
  const bool apart = dense_apart(B);
  DenseArgs A;
  A.b3 = b3; A.W4 = W4; A.b4 = b4;
  A.y = (bf16 *)y; A.out = out; A.part = part;
  A.B = B; A.err = err;
  const int smem = kDenseStages * kDenseStage + sizeof(DenseShared) + 1024;
  auto *fn = apart ? k_dense<true> : k_dense<false>;
  ALDIC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  fn<<<dim3((B + 127) / 128, apart ? kDenseSlices : 1), kDenseThreads, smem, st>>>(mA, mB, A);
  if (apart) k_dense_out<<<(B + 3) / 4, 128, 0, st>>>(A);
  ALDIC_CUDA(cudaGetLastError());
  return OK;
}

}  // namespace aldic
