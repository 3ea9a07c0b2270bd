// Masked autoregressive proposal network (MADE, Germain et al. 2015): BF16 GEMMs with
// FP32 accumulation on the Blackwell tensor cores (tcgen05.mma, accumulators in TMEM),
// fused epilogues, and the loss / gradient / Adam kernels of its training.
//
// Network: x in {0,1}^n (scan order) -> h1 = relu((W1*M1) x + b1) -> h2 = relu((W2*M2) h1
// + b2) -> z = (W3*M3) h2 + b3, q(x_d = 1 | x_<d) = sigmoid(z_d).  Masks M1..M3 enforce
// the autoregressive order; the masked weights are kept as BF16 copies for the GEMMs and
// as FP32 masters for the optimiser.  Everything stays on the device (no host round
// trips per step).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "common.hpp"
#include "made.hpp"
#include "tcgen05.cuh"
#include "tma_map.hpp"

namespace rgs {

// Set when a bounded wait of this file's GEMM gave up (read by tensor_core_status).
__device__ int g_tc_timeout = 0;

int wht_tensor_core_timeout(int* timed_out);
int fourier_tma_timeout(int* timed_out);

namespace {

// CTA tile of the tensor-core GEMM: 128 x 128 outputs (one TMEM accumulator of 128 lanes
// x 128 fp32 columns), K in slices of 64.  Operands staged by the threads use two
// shared-memory stages; TMA-loaded operands a three-stage pipeline (the loads of slices
// k + 1 and k + 2 in flight while slice k is multiplied), two CTAs per SM.
constexpr int TBM = 128, TBN = 128, TBK = 64, kStages = 2, kTmaStages = 3;
constexpr int kTileBytes = TBM * TBK * 2;  // one 128 x 64 bf16 operand tile (16 KiB)
constexpr int kGemmSmem = kTmaStages * 2 * kTileBytes + 1024 + 64;
// Split K: the blocks of a cluster take consecutive ranges of K slices and add their FP32
// tiles through distributed shared memory (rows of kPartPitch floats: 16-byte stores of
// eight consecutive rows hit distinct banks).
constexpr int kMaxSplit = 8, kPartPitch = TBN + 4;
static_assert(TBM * kPartPitch * 4 <= kTmaStages * 2 * kTileBytes, "the partial tile reuses the operand stages");

// Byte offset of the 16-byte chunk (row r, k-chunk kc) of a 128 x 64 operand tile in the
// K-major no-swizzle layout: core matrices of 8 rows x 16 bytes, the eight k-chunks of a
// row group 128 bytes apart (LBO), row groups 1024 bytes apart (SBO).
__device__ __forceinline__ uint32_t cm_off(int r, int kc) { return (uint32_t)((r >> 3) * 1024 + kc * 128 + (r & 7) * 16); }

__device__ __forceinline__ unsigned bf_bits(const __nv_bfloat16* p) { return (unsigned)__bfloat16_as_ushort(*p); }

__device__ __forceinline__ unsigned word_of(const uint4& v, int w) {
  return w == 0 ? v.x : (w == 1 ? v.y : (w == 2 ? v.z : v.w));
}

// Eight consecutive bf16 values, those at index >= valid replaced by zero.
__device__ __forceinline__ uint4 load8_partial(const __nv_bfloat16* src, int valid) {
  unsigned w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < valid) w[j >> 1] |= bf_bits(src + j) << (16 * (j & 1));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Eight consecutive bf16 values of rows whose chunks are `unit` elements (8, 4, 2 or 1)
// aligned; those at index >= valid replaced by zero.
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* src, int valid, int unit) {
  if (valid < 8) return load8_partial(src, valid);
  if (unit == 1) return load8_partial(src, 8);
  if (unit == 8) return __ldg(reinterpret_cast<const uint4*>(src));
  if (unit == 4) {
    const uint2 a = __ldg(reinterpret_cast<const uint2*>(src)), b = __ldg(reinterpret_cast<const uint2*>(src) + 1);
    return make_uint4(a.x, a.y, b.x, b.y);
  }
  const unsigned* p = reinterpret_cast<const unsigned*>(src);
  return make_uint4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// Elements of the widest load that row starts `ld` apart from `p` allow.
__device__ __forceinline__ int row_unit(const __nv_bfloat16* p, int ld) {
  const unsigned low = (unsigned)(uintptr_t)p | (unsigned)ld * 2u;
  return (low & 15u) == 0 ? 8 : ((low & 7u) == 0 ? 4 : ((low & 3u) == 0 ? 2 : 1));
}

// Rows [r0, r0 + 128) x k [k0, k0 + 64) of a logical R x K operand into the K-major
// layout; zero outside the operand.  kmajor: element (r, k) at G[r * ld + k]; otherwise
// at G[k * ld + r] (MN-major: transposed in registers on the way).  128 threads, one
// 8 x 8 core matrix each; unit: row_unit of the operand.  Loads of
// two bytes bound the kernel (4096 x 500 x 500: 104 us, with the 8-byte loads that its rows
// allow 32; 4096 x 501 x 501, whole chunks loaded without a test per element: 118 -> 71).
__device__ __forceinline__ void stage_tile(unsigned char* tile, const __nv_bfloat16* __restrict__ G, int ld, int R,
                                           int K, int r0, int k0, bool kmajor, int unit) {
  const int t = threadIdx.x;
  if (kmajor) {
    const int kc = t & 7, rg = t >> 3;
    const int k = k0 + kc * 8;
    uint4 rows[8];  // all loaded before the first is stored
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = r0 + rg * 8 + ((i + kc) & 7);  // rotated so that a quarter warp hits distinct banks
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (r < R && k < K) {
        const __nv_bfloat16* src = G + (size_t)r * ld + k;
        v = load8(src, K - k, unit);
      }
      rows[i] = v;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(tile + cm_off(rg * 8 + ((i + kc) & 7), kc)) = rows[i];
  } else {
    const int rg = t & 15, kc = t >> 4;
    const int r = r0 + rg * 8;
    uint4 rows[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = k0 + kc * 8 + j;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (k < K && r < R) {
        const __nv_bfloat16* src = G + (size_t)k * ld + r;
        // Two-byte loads: one path for the whole warp, whose lanes meet the ragged end here.
        v = unit == 1 ? load8_partial(src, R - r) : load8(src, R - r, unit);
      }
      rows[j] = v;
    }
    // Row e of the core matrix = element e of the eight loaded k-rows.
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e = (i + rg) & 7;
      const unsigned sel = (e & 1) ? 0x7632u : 0x5410u;
      unsigned w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned a = word_of(rows[2 * j], e >> 1), b = word_of(rows[2 * j + 1], e >> 1);
        w[j] = __byte_perm(a, b, sel);
      }
      *reinterpret_cast<uint4*>(tile + cm_off(rg * 8 + e, kc)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// TMA descriptors of the operands whose rows are 16-byte aligned (boxes of 64 contiguous
// elements, 128-byte swizzle: 64 K-elements x 128 rows of a K-major operand, 64 M- or
// N-elements x 64 k-rows of an MN-major one, two per tile); the others are staged by the
// threads.
struct GemmMaps {
  CUtensorMap a, b;
  int tma_a, tma_b;
  int mn_a, mn_b;  // TMA-loaded MN-major
};

// The epilogue of one output: alpha, bias, ReLU, mask, gate.
__device__ __forceinline__ float finish(const GemmArgs& g, float v, int m, int n) {
  v *= g.alpha;
  if (g.bias) v += g.bias[n];
  if (g.relu) v = fmaxf(v, 0.f);
  if (g.mask) v *= (float)g.mask[(size_t)m * g.N + n];
  if (g.gate && !(__bfloat162float(g.gate[(size_t)m * g.ldc + n]) > 0.f)) v = 0.f;
  return v;
}

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&p);
}

// C[M x N] = op(A)[M x K] * op(B)[K x N]; A row-major [M][lda] (transA: [K][lda]), B
// row-major [K][ldb] (transB: [N][ldb]).  One CTA of 128 threads per 128 x 128 tile of C
// and K range, K in slices of 64.
// Both operands by TMA: one thread issues the loads, three slices ahead, refilling a stage
// once the MMAs that read it have completed (its `done` mbarrier); another waits for a
// slice's bytes (its `full` mbarrier) and issues its four tcgen05.mma (K = 16 each) into
// the TMEM accumulator, so the next slice's MMAs are queued while the last ones run.
// Otherwise the threads stage the operands that TMA cannot load (MN-major ones transposed
// in registers) over two stages.
// After the last slice every warp reads its 32 TMEM lanes (rows) and applies the epilogue,
// 16 columns of a row with 16-byte loads and stores where the row pitch allows; with split
// K (a cluster per tile) the FP32 tiles are added first, each block finishing its share
// of the rows, in block order: the sum does not depend on timing.
//
// What bounds it: the weight gradients (512 x 512 x 4096 and smaller) have 4 to 16 tiles of
// 64 slices, so one CTA per tile leaves most of the chip idle, and operands transposed by
// the threads keep the tensor core waiting.  Split over eight CTAs and loaded by TMA they
// are launch and pipeline latency: the eight GEMMs of a gradient (4096 rows, n = 56, 2 x
// 512 hidden) took 1656 us before and take 81 us.
__global__ void __launch_bounds__(128) gemm_tc_kernel(GemmArgs g, const __grid_constant__ GemmMaps maps, int split) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + kTmaStages * 2 * kTileBytes);  // done[3], full[3]
  uint64_t* full = bars + kTmaStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kTmaStages);
  __shared__ int s_issued;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * TBM, n0 = (blockIdx.x / split) * TBN;
  const bool tma = maps.tma_a || maps.tma_b;
  const uint32_t tx_bytes = (maps.tma_a ? kTileBytes : 0) + (maps.tma_b ? kTileBytes : 0);
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * kTmaStages; ++s) tc::mbar_init(&bars[s], 1);
    tc::fence_barrier_init();
    s_issued = 0;
  }
  if (warp == 0) tc::tmem_alloc(tmem_slot, TBN);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const int unitA = row_unit(g.A, g.lda), unitB = row_unit(g.B, g.ldb);
  // This block's K slices [k0, k0 + KT).
  const int slices = (g.K + TBK - 1) / TBK;
  const int per = (slices + split - 1) / split, rank = split > 1 ? (int)tc::cluster_rank() : 0;
  const int k0 = rank * per;
  const int KT = max(0, min(per, slices - k0));
  const uint32_t idesc = tc::instr_desc(TBM, TBN, 1, maps.mn_a, maps.mn_b);
  bool ok = true;
  // Loads of K slice kt into stage buffers.
  auto load = [&](int kt, unsigned char* As, unsigned char* Bs, uint64_t* bar) {
    const int k = (k0 + kt) * TBK;
    if (maps.tma_a) {
      if (maps.mn_a) {
        tc::tma_load_2d(As, &maps.a, m0, k, bar);
        tc::tma_load_2d(As + kTileBytes / 2, &maps.a, m0 + 64, k, bar);
      } else {
        tc::tma_load_2d(As, &maps.a, k, m0, bar);
      }
    }
    if (maps.tma_b) {
      if (maps.mn_b) {
        tc::tma_load_2d(Bs, &maps.b, n0, k, bar);
        tc::tma_load_2d(Bs + kTileBytes / 2, &maps.b, n0 + 64, k, bar);
      } else {
        tc::tma_load_2d(Bs, &maps.b, k, n0, bar);
      }
    }
  };
  // Operand descriptor of the kk-th 16-element K step of a stage.  TMA tiles: K-major rows
  // 128 bytes apart, step kk at +32 kk bytes; MN-major k-rows 128 bytes apart, 64 elements
  // of M or N per half tile, step kk at +2048 kk.  Staged tiles: core matrices (LBO 128,
  // SBO 1024), step kk at +256 kk.
  auto desc = [&](uint32_t addr, int by_tma, int mn, int kk) {
    if (!by_tma) return tc::smem_desc(addr + kk * 256, 128, 1024, 0);
    return mn ? tc::smem_desc(addr + kk * 2048, kTileBytes / 2, 1024, 2) : tc::smem_desc(addr + kk * 32, 16, 1024, 2);
  };
  auto multiply = [&](int kt, int s) {
    const uint32_t a0 = tc::smem_u32(base + s * 2 * kTileBytes), b0 = a0 + kTileBytes;
#pragma unroll
    for (int kk = 0; kk < TBK / 16; ++kk)
      tc::mma_f16(tmem, desc(a0, maps.tma_a, maps.mn_a, kk), desc(b0, maps.tma_b, maps.mn_b, kk), idesc,
                  (kt > 0 || kk > 0) ? 1u : 0u);
    tc::mma_commit(&bars[s]);
  };
  if (maps.tma_a && maps.tma_b) {
    // Every wait is bounded; after one gives up, the loads still in flight and the last MMAs
    // are waited for (also bounded) before the block frees its TMEM.
    int consumed = 0;
    if (threadIdx.x == 32) {
      int issued = 0, s = 0;
      uint32_t phase = 1;  // of the stage's last use: kt / kTmaStages - 1
      for (int kt = 0; kt < KT; ++kt) {
        if (kt >= kTmaStages && !tc::mbar_wait(&bars[s], phase)) {
          ok = false;
          break;
        }
        unsigned char* As = base + s * 2 * kTileBytes;
        tc::mbar_expect_tx(&full[s], 2 * kTileBytes);
        load(kt, As, As + kTileBytes, &full[s]);
        ++issued;
        if (++s == kTmaStages) {
          s = 0;
          phase ^= 1u;
        }
      }
      s_issued = issued;
    } else if (threadIdx.x == 0) {
      // Descriptors by additions to the first stage's (built anew for each MMA, they and the
      // divisions by the stage count cost 1.5 us of 15.6 at 8192 x 512 x 512).  The address
      // field holds 16-byte units.
      const uint32_t first = tc::smem_u32(base);
      const uint64_t a_first = desc(first, 1, maps.mn_a, 0), b_first = desc(first + kTileBytes, 1, maps.mn_b, 0);
      const uint32_t a_step = maps.mn_a ? 2048 >> 4 : 32 >> 4, b_step = maps.mn_b ? 2048 >> 4 : 32 >> 4;
      int s = 0;
      uint32_t phase = 0;
      for (int kt = 0; kt < KT; ++kt) {
        if (!tc::mbar_wait(&full[s], phase)) {
          ok = false;
          break;
        }
        ++consumed;
        tc::fence_after_sync();
        const uint32_t stage = (uint32_t)s * (2 * kTileBytes >> 4);
#pragma unroll
        for (int kk = 0; kk < TBK / 16; ++kk)
          tc::mma_f16(tmem, a_first + (stage + kk * a_step), b_first + (stage + kk * b_step), idesc,
                      (kt > 0 || kk > 0) ? 1u : 0u);
        tc::mma_commit(&bars[s]);
        if (++s == kTmaStages) {
          s = 0;
          phase ^= 1u;
        }
      }
      if (consumed > 0 &&
          !tc::mbar_wait(&bars[(consumed - 1) % kTmaStages], (uint32_t)((consumed - 1) / kTmaStages) & 1u))
        ok = false;
    }
    ok = __syncthreads_and(ok);
    if (!ok && threadIdx.x == 0)
      for (int kt = consumed; kt < s_issued; ++kt)
        tc::mbar_wait(&full[kt % kTmaStages], (uint32_t)(kt / kTmaStages) & 1u);
  } else {
    for (int kt = 0; kt < KT; ++kt) {
      const int s = kt & 1;
      if (kt >= kStages && !tc::mbar_wait(&bars[s], (uint32_t)((kt >> 1) - 1) & 1u)) ok = false;
      if (!__syncthreads_and(ok)) {
        ok = false;
        break;
      }
      unsigned char* As = base + s * 2 * kTileBytes;
      unsigned char* Bs = As + kTileBytes;
      if (tma && threadIdx.x == 0) {
        tc::mbar_expect_tx(&full[s], tx_bytes);
        load(kt, As, Bs, &full[s]);
      }
      const int k = (k0 + kt) * TBK;
      if (!maps.tma_a) stage_tile(As, g.A, g.lda, g.M, g.K, m0, k, !g.transA, unitA);
      if (!maps.tma_b) stage_tile(Bs, g.B, g.ldb, g.N, g.K, n0, k, g.transB != 0, unitB);
      tc::fence_async_smem();
      __syncthreads();
      if (threadIdx.x == 0) {
        if (tma && !tc::mbar_wait(&full[s], (uint32_t)(kt >> 1) & 1u)) {
          ok = false;  // no MMA: the next wait on this stage gives up too, and every thread leaves
        } else {
          tc::fence_after_sync();
          multiply(kt, s);
        }
      }
    }
    if (ok && KT > 0 && !tc::mbar_wait(&bars[(KT - 1) & 1], (uint32_t)((KT - 1) >> 1) & 1u)) ok = false;
  }
  ok = __syncthreads_and(ok);
  tc::fence_after_sync();
  if (!ok && threadIdx.x == 0) atomicExch(&g_tc_timeout, 1);
  const uint32_t tmem_row = tmem + ((uint32_t)(warp * 32) << 16);
  // Rows of whole 16-byte chunks: of the FP32 output (four columns), and of the bf16 output
  // and gate (eight) where there are such.  (8192 x 500 x 512, FP32 output: 13.6 us, element
  // by element 44.)
  const bool aligned = (g.ldc & (g.Cb || g.gate ? 7 : 3)) == 0 && ((uintptr_t)g.C & 15) == 0 && ((uintptr_t)g.Cb & 15) == 0 &&
                       ((uintptr_t)g.gate & 15) == 0 && (!g.mask || ((g.N & 15) == 0 && ((uintptr_t)g.mask & 15) == 0));
  if (split == 1) {
    const int m = m0 + warp * 32 + lane;
    if (ok) {
      for (int c0 = 0; c0 < TBN && n0 + c0 < g.N; c0 += 16) {
        __syncwarp();  // tcgen05.ld is warp-converged
        uint32_t r[16];
        tc::tmem_ld16(tmem_row + (uint32_t)c0, r);
        const int n = n0 + c0;
        const bool vec = aligned && n + 16 <= g.N && m < g.M;
        // Gate and mask of the 16 columns, loaded while the accumulator is read.
        uint4 gate[2], mask;
        if (vec && g.gate) {
          const uint4* p = reinterpret_cast<const uint4*>(g.gate + (size_t)m * g.ldc + n);
          gate[0] = __ldg(p);
          gate[1] = __ldg(p + 1);
        }
        if (vec && g.mask) mask = __ldg(reinterpret_cast<const uint4*>(g.mask + (size_t)m * g.N + n));
        tc::tmem_ld_wait();
        if (m >= g.M) continue;
        if (vec) {
          float v[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            v[j] = __uint_as_float(r[j]) * g.alpha;
            if (g.bias) v[j] += g.bias[n + j];
            if (g.relu) v[j] = fmaxf(v[j], 0.f);
            if (g.mask) v[j] *= (float)((word_of(mask, j >> 2) >> (8 * (j & 3))) & 255u);
            if (g.gate) {
              const unsigned w = word_of(gate[j >> 3], (j & 7) >> 1);
              if (!(__uint_as_float((j & 1) ? (w & 0xffff0000u) : (w << 16)) > 0.f)) v[j] = 0.f;
            }
          }
          if (g.C) {
            float4* dst = reinterpret_cast<float4*>(g.C + (size_t)m * g.ldc + n);
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          }
          if (g.Cb) {
            uint4* dst = reinterpret_cast<uint4*>(g.Cb + (size_t)m * g.ldc + n);
#pragma unroll
            for (int q = 0; q < 2; ++q)
              dst[q] = make_uint4(pack_bf16(v[8 * q], v[8 * q + 1]), pack_bf16(v[8 * q + 2], v[8 * q + 3]),
                                  pack_bf16(v[8 * q + 4], v[8 * q + 5]), pack_bf16(v[8 * q + 6], v[8 * q + 7]));
          }
          continue;
        }
        if (aligned && !g.Cb && !g.mask && !g.gate && (g.N & 3) == 0) {  // the last columns, by fours
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (n + 4 * q >= g.N) break;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = finish(g, __uint_as_float(r[4 * q + j]), m, n + 4 * q + j);
            *reinterpret_cast<float4*>(g.C + (size_t)m * g.ldc + n + 4 * q) = make_float4(v[0], v[1], v[2], v[3]);
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (n + j >= g.N) break;
          const float v = finish(g, __uint_as_float(r[j]), m, n + j);
          if (g.C) g.C[(size_t)m * g.ldc + n + j] = v;
          if (g.Cb) g.Cb[(size_t)m * g.ldc + n + j] = __float2bfloat16(v);
        }
      }
    }
  } else {
    // This block's FP32 tile into its (now idle) operand stages; zero without K slices.
    float* part = reinterpret_cast<float*>(base);
    float* row = part + (warp * 32 + lane) * kPartPitch;
    for (int c0 = 0; c0 < TBN; c0 += 16) {
      uint32_t r[16];
      if (ok && KT > 0) {
        tc::tmem_ld16(tmem_row + (uint32_t)c0, r);
        tc::tmem_ld_wait();
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = 0u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4*>(row + c0 + 4 * q) = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
    }
    tc::cluster_sync();
    // A warp per row of this block's share: 32 lanes x 4 columns.
    const int share = TBM / split;
    for (int i = warp; i < share; i += 4) {
      const int rr = rank * share + i, m = m0 + rr, n = n0 + 4 * lane;
      if (m >= g.M || n >= g.N) continue;
      float4 p[kMaxSplit];
#pragma unroll
      for (int k = 0; k < kMaxSplit; ++k)
        if (k < split) p[k] = tc::ld_cluster_f4(part + rr * kPartPitch + 4 * lane, (uint32_t)k);
      float v[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
      for (int k = 1; k < kMaxSplit; ++k)
        if (k < split) {
          v[0] += p[k].x;
          v[1] += p[k].y;
          v[2] += p[k].z;
          v[3] += p[k].w;
        }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n + j < g.N) v[j] = finish(g, v[j], m, n + j);
      if (aligned && n + 4 <= g.N) {
        if (g.C) *reinterpret_cast<float4*>(g.C + (size_t)m * g.ldc + n) = make_float4(v[0], v[1], v[2], v[3]);
        if (g.Cb)
          *reinterpret_cast<uint2*>(g.Cb + (size_t)m * g.ldc + n) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (n + j >= g.N) break;
          if (g.C) g.C[(size_t)m * g.ldc + n + j] = v[j];
          if (g.Cb) g.Cb[(size_t)m * g.ldc + n + j] = __float2bfloat16(v[j]);
        }
      }
    }
    tc::cluster_sync();  // no block leaves while a peer reads its tile
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, TBN);
}

// dz = sigmoid(z) - target; loss partials: softplus(z) - target * z (per block, float64).
__global__ void bce_grad_kernel(const float* __restrict__ z, const float* __restrict__ target, int count,
                                float scale, __nv_bfloat16* __restrict__ dz, double* __restrict__ partial) {
  __shared__ double red[256];
  double loss = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const float x = z[i], t = target[i];
    const float s = 1.f / (1.f + __expf(-x));
    dz[i] = __float2bfloat16((s - t) * scale);
    const float sp = x > 0.f ? x + log1pf(__expf(-x)) : log1pf(__expf(x));
    loss += (double)(sp - t * x);
  }
  red[threadIdx.x] = loss;
  __syncthreads();
  for (int off = blockDim.x / 2; off; off >>= 1) {
    if ((int)threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// Column sums of up to three [rows x cols] bf16 matrices (bias gradients) in one launch:
// a cluster of kSumChunks blocks per 64 columns, a range of rows each, the blocks' sums
// added through distributed shared memory in block order.  (One thread per column over
// all rows is a serial chain of row loads in four blocks: 256 us for the three sums over
// 4096 rows, n = 56, hidden 512, against 7.5 in one launch here.)
constexpr int kSumChunks = 8, kSumCols = 64;
struct ColsumJob {
  const __nv_bfloat16* x;
  float* out;
  int cols;
};
struct ColsumJobs {
  ColsumJob job[3];
};
__global__ void __launch_bounds__(256) colsum_kernel(const __grid_constant__ ColsumJobs jobs, int rows) {
  __shared__ __align__(16) float part[32][kSumCols + 4];
  __shared__ __align__(16) float total[kSumCols];
  const ColsumJob job = jobs.job[blockIdx.z];
  const int cols = job.cols, c0 = (blockIdx.x / kSumChunks) * kSumCols, rank = (int)tc::cluster_rank();
  const int per = (rows + kSumChunks - 1) / kSumChunks;
  const int r0 = rank * per, r1 = min(rows, r0 + per);
  const int cg = threadIdx.x & 7, rl = threadIdx.x >> 3;  // 8 columns per thread, 32 rows at a time
  const int c = c0 + cg * 8;
  const bool vec = (cols % 8 == 0) && (((uintptr_t)job.x & 15) == 0);
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c < cols) {
#pragma unroll 4
    for (int r = r0 + rl; r < r1; r += 32) {
      const __nv_bfloat16* p = job.x + (size_t)r * cols + c;
      const uint4 v = vec ? __ldg(reinterpret_cast<const uint4*>(p)) : load8_partial(p, cols - c);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const unsigned w = word_of(v, j >> 1);
        s[j] += __uint_as_float((j & 1) ? (w & 0xffff0000u) : (w << 16));
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) part[rl][cg * 8 + j] = s[j];
  __syncthreads();
  if (threadIdx.x < kSumCols) {
    float t = 0.f;
    for (int k = 0; k < 32; ++k) t += part[k][threadIdx.x];
    total[threadIdx.x] = t;
  }
  tc::cluster_sync();
  if (rank == 0 && threadIdx.x < kSumCols / 4) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kSumChunks; ++k) {
      const float4 p = tc::ld_cluster_f4(total + 4 * threadIdx.x, (uint32_t)k);
      t.x += p.x;
      t.y += p.y;
      t.z += p.z;
      t.w += p.w;
    }
    const float v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c0 + 4 * (int)threadIdx.x + j < cols) job.out[c0 + 4 * threadIdx.x + j] = v[j];
  }
  tc::cluster_sync();
}

// Adam step on FP32 masters, then the masked BF16 copy used by the GEMMs.
__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ grad, float* __restrict__ m1,
                            float* __restrict__ m2, const unsigned char* __restrict__ mask,
                            __nv_bfloat16* __restrict__ wb, int count, float lr, float b1, float b2, float eps,
                            float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float gr = grad[i];
  const float a = b1 * m1[i] + (1.f - b1) * gr;
  const float v = b2 * m2[i] + (1.f - b2) * gr * gr;
  m1[i] = a;
  m2[i] = v;
  const float nw = w[i] - lr * (a / c1) / (sqrtf(v / c2) + eps);
  w[i] = nw;
  if (wb) wb[i] = __float2bfloat16(mask ? nw * (float)mask[i] : nw);
}

// One autoregressive position for a batch: x[:, d] ~ Bernoulli(sigmoid(z[:, d])) with a
// Philox-free counter hash uniform, and log q accumulation.  Rows of x are bf16 {0, 1}.
__device__ __forceinline__ double hash_uniform(unsigned long long seed, unsigned long long a, unsigned b) {
  unsigned long long h = seed ^ (a * 0x9E3779B97F4A7C15ull) ^ ((unsigned long long)b * 0xC2B2AE3D27D4EB4Full);
  h ^= h >> 31;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 27;
  h *= 0x94D049BB133111EBull;
  h ^= h >> 31;
  return (double)(h >> 11) * 0x1.0p-53;
}

__global__ void sample_position_kernel(const float* __restrict__ z, int n, int d, int count, unsigned long long seed,
                                       unsigned long long first, __nv_bfloat16* __restrict__ x,
                                       double* __restrict__ logq) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float zd = z[(size_t)i * n + d];
  const double q1 = 1.0 / (1.0 + exp(-(double)zd));
  const double u = hash_uniform(seed, first + i, (unsigned)d);
  const int bit = u < q1 ? 1 : 0;
  x[(size_t)i * n + d] = __float2bfloat16((float)bit);
  logq[i] += log(bit ? q1 : 1.0 - q1);
}

// log q(x) = sum_d log sigmoid(+-z_d) for given x.
__global__ void logq_kernel(const float* __restrict__ z, const __nv_bfloat16* __restrict__ x, int n, int count,
                            double* __restrict__ logq) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  double s = 0.0;
  for (int d = 0; d < n; ++d) {
    const double zd = z[(size_t)i * n + d];
    const double sign = __bfloat162float(x[(size_t)i * n + d]) > 0.5f ? 1.0 : -1.0;
    const double t = sign * zd;  // log sigmoid(t) = -softplus(-t)
    s += t > 0 ? -log1p(exp(-t)) : t - log1p(exp(t));
  }
  logq[i] = s;
}

}  // namespace

namespace {
// Tensor map of a bf16 operand [rows][ld] whose contiguous extent is `inner`: boxes of 64
// contiguous elements x `box_rows` with 128-byte swizzle, zero fill outside the operand.
// False when TMA cannot load it (row pitch not a multiple of 16 bytes, unaligned base, or
// no encoder).
bool tma_operand(CUtensorMap* map, const __nv_bfloat16* ptr, int ld, int inner, int rows, int box_rows) {
  if (((uintptr_t)ptr & 15) != 0 || (ld % 8) != 0 || inner <= 0 || rows <= 0) return false;
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)ptr, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// TMA operand loads on (default) or off (every operand staged by the threads).
bool g_gemm_tma = true;
}  // namespace

int gemm_set_tma(int on) {
  g_gemm_tma = on != 0;
  return RGS_OK;
}

int gemm_bf16(const GemmArgs& g, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || !g.A || !g.B || (!g.C && !g.Cb)) return fail(RGS_ERR_ARG, "bad GEMM");
  static bool configured[64] = {false};
  int device = 0;
  RGS_CUDA_TRY(cudaGetDevice(&device));
  if (device >= 0 && device < 64 && !configured[device]) {
    RGS_CUDA_TRY(cudaFuncSetAttribute(gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
    configured[device] = true;
  }
  GemmMaps maps;
  std::memset(&maps, 0, sizeof(maps));
  // A is K-major unless transposed; B is K-major when transposed ([N][ldb]).
  if (g_gemm_tma) {
    maps.tma_a = g.transA ? tma_operand(&maps.a, g.A, g.lda, g.M, g.K, TBK) : tma_operand(&maps.a, g.A, g.lda, g.K, g.M, TBM);
    maps.tma_b = g.transB ? tma_operand(&maps.b, g.B, g.ldb, g.K, g.N, TBN) : tma_operand(&maps.b, g.B, g.ldb, g.N, g.K, TBK);
    // An MN-major operand goes by TMA only together with the other one: a staged partner
    // would leave the block waiting for its threads either way.
    if (!(maps.tma_a && maps.tma_b)) {
      if (g.transA) maps.tma_a = 0;
      if (!g.transB) maps.tma_b = 0;
    }
    maps.mn_a = maps.tma_a && g.transA;
    maps.mn_b = maps.tma_b && !g.transB;
  }
  // Split K where a long K meets few tiles (weight gradients: K is the batch): up to eight
  // blocks per tile, four slices or more each but for the last of a cluster (33 slices over
  // eight blocks: six of 5, one of 3, one of none).  Shorter sums (K < 1024) stay in one
  // accumulator, in slice order.
  const int tiles = ((g.N + TBN - 1) / TBN) * ((g.M + TBM - 1) / TBM), slices = (g.K + TBK - 1) / TBK;
  int split = 1;
  if (g.K >= 1024)
    while (split < kMaxSplit && 2 * split * tiles <= sm_count(device) && slices >= 8 * split) split *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(split * ((g.N + TBN - 1) / TBN)), (unsigned)((g.M + TBM - 1) / TBM));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = kGemmSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)split;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = split > 1 ? 1 : 0;
  RGS_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_tc_kernel, g, maps, split));
  return RGS_OK;
}

int tensor_core_status(int* timed_out) {
  int h = 0, zero = 0;
  RGS_CUDA_TRY(cudaMemcpyFromSymbol(&h, g_tc_timeout, sizeof(int)));
  RGS_CUDA_TRY(cudaMemcpyToSymbol(g_tc_timeout, &zero, sizeof(int)));
  int w = 0, f = 0;
  int rc = wht_tensor_core_timeout(&w);
  if (rc) return rc;
  if ((rc = fourier_tma_timeout(&f))) return rc;
  *timed_out = h | w | f;
  return RGS_OK;
}

int bce_grad(const float* z, const float* target, int count, float scale, __nv_bfloat16* dz, double* partial,
             int blocks, cudaStream_t s) {
  bce_grad_kernel<<<blocks, 256, 0, s>>>(z, target, count, scale, dz, partial);
  RGS_CUDA_TRY(cudaGetLastError());
  return RGS_OK;
}

int colsum3_bf16(const __nv_bfloat16* const x[3], const int cols[3], float* const out[3], int rows, cudaStream_t s) {
  ColsumJobs jobs;
  int most = 1;
  for (int k = 0; k < 3; ++k) {
    jobs.job[k] = ColsumJob{x[k], out[k], cols[k]};
    most = cols[k] > most ? cols[k] : most;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(kSumChunks * ((most + kSumCols - 1) / kSumCols)), 1, 3);
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kSumChunks;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  RGS_CUDA_TRY(cudaLaunchKernelEx(&cfg, colsum_kernel, jobs, rows));
  return RGS_OK;
}

int adam_step(float* w, const float* grad, float* m1, float* m2, const unsigned char* mask, __nv_bfloat16* wb,
              int count, float lr, float b1, float b2, float eps, int t, cudaStream_t s) {
  const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
  adam_kernel<<<(count + 255) / 256, 256, 0, s>>>(w, grad, m1, m2, mask, wb, count, lr, b1, b2, eps, c1, c2);
  RGS_CUDA_TRY(cudaGetLastError());
  return RGS_OK;
}

int sample_position(const float* z, int n, int d, int count, unsigned long long seed, unsigned long long first,
                    __nv_bfloat16* x, double* logq, cudaStream_t s) {
  sample_position_kernel<<<(count + 255) / 256, 256, 0, s>>>(z, n, d, count, seed, first, x, logq);
  RGS_CUDA_TRY(cudaGetLastError());
  return RGS_OK;
}

int log_q(const float* z, const __nv_bfloat16* x, int n, int count, double* logq, cudaStream_t s) {
  logq_kernel<<<(count + 255) / 256, 256, 0, s>>>(z, x, n, count, logq);
  RGS_CUDA_TRY(cudaGetLastError());
  return RGS_OK;
}

}  // namespace rgs
