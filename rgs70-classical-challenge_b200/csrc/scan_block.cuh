// Run kernel: k consecutive scan positions (DevBlock, plan.hpp) in one pass over HBM.
//
// A thread owns one string and, in shared memory, one column of 2^dmax slots.  Per group
// it gathers the group's rows of the input table, carries them through the k positions --
// every interior table lives in the column, in place -- and stores the group's rows of the
// output table; no interior table reaches memory.  Threads never exchange data, so the
// group loop has no barrier; lanes are consecutive strings, so every access of a warp is
// one contiguous piece of a row.
//
// Arithmetic per entry as in the position-by-position sweep: same combos in the same
// order, every interior entry rounded to the storage type, also where a fused stage keeps
// it in registers, so that a string's result has the bits of the position-by-position sweep
// (complex64 with float64 arithmetic: 4096 strings at n = 40 18.7 ms without that rounding,
// 21.0 with it; one order of sums for all schedules cost 1% in float32 arithmetic, 2% at
// rank 11).  Renormalisation as in the
// pair kernel: the first position is scaled from the previous maximum, the others by the
// power of two of their own weights (2^0 for a row of a unitary), recorded as the maximum
// 4^e / 4 of the interior tables so that the finalisation's exponents add up.
//
// What bounds it: the pair kernels moved 2.8M entries per string of the n = 40, rank 20
// instance at 79% of the copy bandwidth; runs move 1.1M and are bound by instruction issue
// and the latency of column accesses (peak run of that instance, float32 arithmetic: issue
// slots 49% busy, DRAM 28%; 14 warps per SM, as many as columns and registers allow).  Hence
//   * a row operation reads one 32-byte record with its ready-made slot offsets, rows and
//     signs (shared memory, the same for every thread), several gathers are in flight per
//     thread, only the last stage tracks maxima;
//   * a growing position and the next one form one stage, so that the level of the peak rank
//     has no slots: 16 slots per column instead of 32, and half the column traffic (4096
//     strings 13.8 -> 11.6 ms, in complex128 25.7 -> 21.0 ms);
//   * float32 arithmetic carries two strings per thread (packed FMAs, one set of index work
//     for both) in launches large enough (launch_block).
// Fetching the next group's maps ahead changed nothing (11.6 ms), prefetching its rows into
// L2 cost 4%.
#pragma once
#include <atomic>

#include "f32x2.cuh"
#include "scan_device.cuh"

namespace rgs {

// Threads per block.  64: two warps share the row operations, and blocks are small enough
// to fill an SM's shared memory (with 32 slots per column, 4096 strings of the n = 40
// instance, float32 arithmetic: 13.8 ms with 64, 15.9 with 128, 18.8 with 32; complex128
// 25.7 / 29.7 / 36.1).
constexpr int kBlockThreads = 64, kBlockLogThreads = 6;

struct __align__(16) BlockOp {
  unsigned ld[4];   // slot byte offset, or (first position) input row of each combo
  unsigned st;      // slot byte offset, or (last position) output row of the first output
  unsigned sign;    // bits 31 - c: local sign of combo c; fused: 27 - c: A's sign, 23 - c: A's y
  unsigned pad[2];
};

// What a thread computes on: NV strings, S storage, M arithmetic.  R holds one real per
// string.  Two complex64 strings with float32 arithmetic run as packed pairs (one FMA for
// both, and one set of index work); rows in HBM are interleaved (re, im) per string,
// columns hold (re, re, im, im).
template <typename S, typename M, int NV>
struct BlockLane {
  static_assert(NV == 1, "one string per thread, except two for float32 arithmetic");
  typedef M R;
  static constexpr int bytes = 2 * (int)sizeof(S);  // of a slot, and of this thread's part of a row
  struct E {
    R re, im;
  };
  struct alignas(2 * sizeof(S)) V {
    S x, y;
  };
  static __device__ __forceinline__ E row(const char* p) {
    if (sizeof(S) == 8) {
      const double2 v = __ldg(reinterpret_cast<const double2*>(p));
      return E{(M)v.x, (M)v.y};
    }
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    return E{(M)v.x, (M)v.y};
  }
  static __device__ __forceinline__ E slot(const char* p) {
    const V v = *reinterpret_cast<const V*>(p);
    return E{(M)v.x, (M)v.y};
  }
  // Rounded to the storage type; `mx` as given is unchanged for columns.
  static __device__ __forceinline__ void to_slot(char* p, const E& e) { *reinterpret_cast<V*>(p) = V{(S)e.re, (S)e.im}; }
  static __device__ __forceinline__ void to_row(char* p, const E& e, S (&mx)[NV]) {
    const V v{(S)e.re, (S)e.im};
    *reinterpret_cast<V*>(p) = v;
    mx[0] = fmax(mx[0], norm2(v.x, v.y));
  }
  // As if the entry had been stored between two positions.
  static __device__ __forceinline__ void store_rounded(E& e) { e.re = (M)(S)e.re, e.im = (M)(S)e.im; }
  static __device__ __forceinline__ R zero() { return (M)0; }
  static __device__ __forceinline__ R mad(R a, R b, R c) { return fma(a, b, c); }
  static __device__ __forceinline__ R neg(R a) { return -a; }
  static __device__ __forceinline__ R flip(R a, unsigned m);
  static __device__ __forceinline__ R pack(const double (&x)[NV]) { return (M)x[0]; }
};
// x with its sign flipped where bit 31 of m is set.
__device__ __forceinline__ float flip_top(float x, unsigned m) {
  return __uint_as_float(__float_as_uint(x) ^ (m & 0x80000000u));
}
__device__ __forceinline__ double flip_top(double x, unsigned m) {
  return __hiloint2double(__double2hiint(x) ^ (int)(m & 0x80000000u), __double2loint(x));
}
template <typename S, typename M, int NV>
__device__ __forceinline__ typename BlockLane<S, M, NV>::R BlockLane<S, M, NV>::flip(R a, unsigned m) {
  return flip_top(a, m);
}
template <>
struct BlockLane<float, float, 2> {
  typedef float2 R;
  static constexpr int bytes = 16;
  struct E {
    R re, im;
  };
  static __device__ __forceinline__ E row(const char* p) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    return E{make_float2(v.x, v.z), make_float2(v.y, v.w)};
  }
  static __device__ __forceinline__ E slot(const char* p) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    return E{make_float2(v.x, v.y), make_float2(v.z, v.w)};
  }
  static __device__ __forceinline__ void to_slot(char* p, const E& e) {
    *reinterpret_cast<float4*>(p) = make_float4(e.re.x, e.re.y, e.im.x, e.im.y);
  }
  static __device__ __forceinline__ void to_row(char* p, const E& e, float (&mx)[2]) {
    *reinterpret_cast<float4*>(p) = make_float4(e.re.x, e.im.x, e.re.y, e.im.y);
    mx[0] = fmaxf(mx[0], norm2(e.re.x, e.im.x));
    mx[1] = fmaxf(mx[1], norm2(e.re.y, e.im.y));
  }
  static __device__ __forceinline__ void store_rounded(E&) {}
  static __device__ __forceinline__ R zero() { return make_float2(0.f, 0.f); }
  static __device__ __forceinline__ R mad(R a, R b, R c) { return f2fma(a, b, c); }
  static __device__ __forceinline__ R neg(R a) { return make_float2(-a.x, -a.y); }
  static __device__ __forceinline__ R flip(R a, unsigned m) { return make_float2(flip_top(a.x, m), flip_top(a.y, m)); }
  static __device__ __forceinline__ R pack(const double (&x)[2]) { return make_float2((float)x[0], (float)x[1]); }
};

// Weights of one position: output = e f(0) and e f(1) terms (merge positions: f(0) + f(1)
// and f(0) - f(1)).
template <typename L>
struct BlockWeights {
  typename L::R ar, ai, br, bi;
};
template <typename R>
struct BlockCoef {
  R re, im, nim;  // nim = -im
};

// acc += e w, in cmad's order.
template <typename L>
__device__ __forceinline__ void block_mad(typename L::E& acc, typename L::R er, typename L::R ei,
                                          const BlockCoef<typename L::R>& w) {
  acc.re = L::mad(er, w.re, acc.re);
  acc.re = L::mad(ei, w.nim, acc.re);
  acc.im = L::mad(er, w.im, acc.im);
  acc.im = L::mad(ei, w.re, acc.im);
}

// Group and thread constants of one position.
struct BlockStep {
  const char* in;      // first position: this thread's part of input row 0
  char* out;           // last position: this thread's part of output row 0
  char* col;           // this thread's column
  unsigned pitch;      // bytes of a table row (first / last position)
  unsigned x0, xk;     // the group's input and output rows
  unsigned swap;       // xor of the first output's place where the group's y is 1
  unsigned pair;       // xor between a pair's two places
  unsigned flip;       // the group's signs (and A's y), xor-ed into BlockOp::sign
  unsigned twin;       // fused: xor between the two gathers' places
  unsigned twin_sign;  // fused: 0x80000000 where the twin gather's signs are flipped
};

// U row operations, their gathers in flight together.  FUSED: a growing position A before
// B: combo c's gathered entry e gives the two rows e f_A(0) and +-e f_A(1) of A's output;
// the one with the gather's y bit goes to the operation itself, the other to its twin
// (same kappa pattern, own signs), so both of A's outputs are used as they are formed.
// TW: DevBlock::twin_order as a constant; swapping the registers at run time is slower where
// the peak runs decide (16384 strings at n = 40: 46.1 ms constant, 46.6 swapped).
template <typename L, typename S, int NV, bool FUSED, bool PAIR, int NC, int NG0, bool FIRST, bool LAST, int TW, int U>
__device__ __forceinline__ void block_ops(const BlockOp* __restrict__ ops, const BlockStep& g,
                                          const BlockCoef<typename L::R>& wa, const BlockCoef<typename L::R>& wb,
                                          const BlockCoef<typename L::R>& pa, const BlockCoef<typename L::R>& pb,
                                          S (&mx)[NV]) {
  typedef typename L::E E;
  constexpr int NT = FUSED ? 2 : 1;
  E e[U][NC];
  unsigned sign[U], st[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint4 ld = *reinterpret_cast<const uint4*>(ops[u].ld);
    const uint2 ss = *reinterpret_cast<const uint2*>(&ops[u].st);
    st[u] = ss.x;
    sign[u] = ss.y ^ g.flip;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const unsigned l = c == 0 ? ld.x : (c == 1 ? ld.y : (c == 2 ? ld.z : ld.w));
      e[u][c] = FIRST ? L::row(g.in + (u64)(g.x0 ^ l) * g.pitch) : L::slot(g.col + l);
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    E a[NT], b[NT], x[NC][NT];
    unsigned m[NC][NT];  // bit 31: the term's sign
#pragma unroll
    for (int t = 0; t < NT; ++t) a[t] = b[t] = E{L::zero(), L::zero()};
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      m[c][0] = sign[u] << c;
      x[c][0] = e[u][c];
      if constexpr (FUSED) {
        m[c][NT - 1] = m[c][0] ^ g.twin_sign;
        E p{L::zero(), L::zero()}, q{L::zero(), L::zero()};
        block_mad<L>(p, e[u][c].re, e[u][c].im, pa);
        block_mad<L>(q, L::flip(e[u][c].re, sign[u] << (4 + c)), L::flip(e[u][c].im, sign[u] << (4 + c)), pb);
        L::store_rounded(p);
        L::store_rounded(q);
        const bool y = (sign[u] << (8 + c)) & 0x80000000u;
        x[c][0].re = y ? q.re : p.re;
        x[c][0].im = y ? q.im : p.im;
        x[c][NT - 1].re = y ? p.re : q.re;
        x[c][NT - 1].im = y ? p.im : q.im;
      }
    }
    // wa terms first in both outputs of a pair (scan_row.cuh): a over the rows in order, b
    // from row NG0 on, then the rows before it; the twin's rows in its own order.
    auto add_b = [&](int c) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int q = t ? c ^ TW : c;
        if (c < NG0)
          block_mad<L>(b[t], L::flip(x[q][t].re, m[q][t]), L::flip(x[q][t].im, m[q][t]), wb);
        else
          block_mad<L>(b[t], x[q][t].re, x[q][t].im, wa);
      }
    };
#pragma unroll
    for (int c = 0; c < NC; ++c) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int q = t ? c ^ TW : c;
        if (!PAIR)
          block_mad<L>(a[t], x[q][t].re, x[q][t].im, (m[q][t] & 0x80000000u) ? wb : wa);
        else if (c < NG0)
          block_mad<L>(a[t], x[q][t].re, x[q][t].im, wa);
        else
          block_mad<L>(a[t], L::flip(x[q][t].re, m[q][t]), L::flip(x[q][t].im, m[q][t]), wb);
      }
      if (PAIR && (NG0 == NC || c >= NG0)) add_b(c);
    }
    if constexpr (PAIR && NG0 < NC) {
#pragma unroll
      for (int c = 0; c < NG0; ++c) add_b(c);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const unsigned place = st[u] ^ g.swap ^ (t ? g.twin : 0u);
      if (LAST) {
        const unsigned row = g.xk ^ place;
        L::to_row(g.out + (u64)row * g.pitch, a[t], mx);
        if (PAIR) L::to_row(g.out + (u64)(row ^ g.pair) * g.pitch, b[t], mx);
      } else {
        L::to_slot(g.col + place, a[t]);
        if (PAIR) L::to_slot(g.col + (place ^ g.pair), b[t]);
      }
    }
  }
}

// A stage's row operations (a power of two), U at a time or, below U, one by one.
template <typename L, typename S, int NV, bool FUSED, bool PAIR, int NC, int NG0, bool FIRST, bool LAST, int TW>
__device__ __forceinline__ void block_rows(const BlockOp* __restrict__ ops, int rows, const BlockStep& g,
                                           const BlockWeights<L>& w, const BlockWeights<L>& wp, S (&mx)[NV]) {
  constexpr int LOADS = FUSED ? 4 : 8;
  constexpr int U = LOADS >= NC ? LOADS / NC : 1;
  const BlockCoef<typename L::R> wa{w.ar, w.ai, L::neg(w.ai)}, wb{w.br, w.bi, L::neg(w.bi)};
  const BlockCoef<typename L::R> pa{wp.ar, wp.ai, L::neg(wp.ai)}, pb{wp.br, wp.bi, L::neg(wp.bi)};
  if (U > 1 && rows < U) {
#pragma unroll 1
    for (int r = 0; r < rows; ++r)
      block_ops<L, S, NV, FUSED, PAIR, NC, NG0, FIRST, LAST, TW, 1>(ops + r, g, wa, wb, pa, pb, mx);
    return;
  }
#pragma unroll 1
  for (int r = 0; r < rows; r += U)
    block_ops<L, S, NV, FUSED, PAIR, NC, NG0, FIRST, LAST, TW, U>(ops + r, g, wa, wb, pa, pb, mx);
}

template <typename L, typename S, int NV, bool FUSED, bool FIRST, bool LAST>
__device__ __forceinline__ void block_stage(int code, int twin_order, const BlockOp* ops, int rows, const BlockStep& g,
                                            const BlockWeights<L>& w, const BlockWeights<L>& wp, S (&mx)[NV]) {
#define RGS_BLOCK_ROWS(PAIR, NC, NG0, TW) \
  block_rows<L, S, NV, FUSED, PAIR, NC, NG0, FIRST, LAST, FUSED ? TW : 0>(ops, rows, g, w, wp, mx)
  switch (FUSED ? code | twin_order << 3 : code) {
    case RC_P1: RGS_BLOCK_ROWS(true, 1, 1, 0); break;
    case RC_P2H: RGS_BLOCK_ROWS(true, 2, 1, 0); break;
    case RC_P2F: RGS_BLOCK_ROWS(true, 2, 2, 0); break;
    case RC_P4H: RGS_BLOCK_ROWS(true, 4, 2, 0); break;
    case RC_M1: RGS_BLOCK_ROWS(false, 1, 1, 0); break;
    case RC_M2: RGS_BLOCK_ROWS(false, 2, 2, 0); break;
    default:
      if constexpr (FUSED) {
        switch (code | twin_order << 3) {
          case RC_P2F | 1 << 3: RGS_BLOCK_ROWS(true, 2, 2, 1); break;
          case RC_P4H | 1 << 3: RGS_BLOCK_ROWS(true, 4, 2, 1); break;
          case RC_M2 | 1 << 3: RGS_BLOCK_ROWS(false, 2, 2, 1); break;
          default: break;  // make_block gives no other
        }
      }
  }
#undef RGS_BLOCK_ROWS
}

// Shared memory: columns, then the weights of every position and thread, then the row
// operations.
template <typename L>
__host__ __device__ constexpr size_t block_smem_bytes(int dmax, int k, int words) {
  return ((size_t)L::bytes << dmax) * kBlockThreads + (size_t)k * sizeof(BlockWeights<L>) * kBlockThreads +
         (size_t)words * sizeof(BlockOp);
}

// W: weights of position j, `stride` strings between positions; maxprev: maxima of the
// input table; maxrow: row of position j of the maxima.  blockIdx.x: column slice (tiles
// wider than the block), then groups; blockIdx.y: tile, tables e_stride entries apart.
template <typename S, typename M, int NV, int MINB>
__global__ void __launch_bounds__(kBlockThreads, MINB)
    scan_block_kernel(const S* __restrict__ Ein, S* __restrict__ Eout, const __grid_constant__ DevBlock P,
                      const u64* __restrict__ tables, const double4* __restrict__ W, const u64* __restrict__ maxprev,
                      u64* __restrict__ maxrow, int stride, int lbt, u64 e_stride) {
  typedef BlockLane<S, M, NV> L;
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int T = kBlockThreads, kLT = kBlockLogThreads, kLV = NV == 2 ? 1 : 0;
  const int tid = threadIdx.x;
  const int lc = lbt - kLV;                            // log2 threads of a row
  const int lcols = lc < kLT ? lc : kLT;               // ... in this block
  const int lslices = lc - lcols, lslots = kLT - lcols;  // log2 column slices; groups side by side
  const int b = (((int)(blockIdx.x & ((1u << lslices) - 1u)) << lcols) | (tid & ((1 << lcols) - 1))) << kLV;
  const int k = P.k;
  BlockWeights<L>* wts = reinterpret_cast<BlockWeights<L>*>(smem + (((size_t)L::bytes << P.dmax) * T));
  BlockOp* ops = reinterpret_cast<BlockOp*>(reinterpret_cast<unsigned char*>(wts) + sizeof(BlockWeights<L>) * T * k);
  const unsigned* lin = reinterpret_cast<const unsigned*>(tables + P.lin_off);
  if (blockIdx.y) {  // tile y of a chunk of tiles
    const u64 y = blockIdx.y;
    Ein += 2 * y * e_stride;
    Eout += 2 * y * e_stride;
    W += y << lbt;
    maxprev += y << lbt;
    maxrow += y << lbt;
  }

  for (int i = 0; i < P.stages; ++i) {
    const bool first = i == 0, last = i + 1 == P.stages;
    for (int r = tid; r < P.rows[i]; r += T) {
      const u64 w = tables[P.prog_off + P.first[i] + r];
      BlockOp op;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const unsigned s = (unsigned)(w >> (8 * c)) & 63u;
        op.ld[c] = first ? __ldg(lin + s) : s * (unsigned)(T * L::bytes);
      }
      const unsigned s = (unsigned)(w >> 32) & 63u;
      op.st = last ? __ldg(lin + (1 << P.din) + s) : s * (unsigned)(T * L::bytes);
      op.sign = __brev((unsigned)(w >> 40) & 0xfffu);
      op.pad[0] = op.pad[1] = 0u;
      ops[P.first[i] + r] = op;
    }
  }
  // Weights of this thread's strings.
  for (int i = 0; i < k; ++i) {
    const bool first = i == 0;
    double ar[NV], ai[NV], br[NV], bi[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const double4 f = W[(size_t)i * stride + b + v];
      int e = 0;
      if (first) {
        e = scale_exponent(max_value<S>(maxprev[b + v]));
      } else {
        // A power of two only where the weights are far from 1 (never for a unitary's row).
        const double m = fmax(fmax(fabs(f.x), fabs(f.y)), fmax(fabs(f.z), fabs(f.w)));
        if (m > 0.0 && isfinite(m) && (m > 4.0 || m < 0.125)) {
          frexp(m, &e);
          e = e > 60 ? 60 : (e < -60 ? -60 : e);
        }
        if (blockIdx.x < (1u << lslices) && (tid >> lcols) == 0)
          maxrow[(size_t)(i - 1) * stride + b + v] = max_bits<S>((S)ldexp(0.25, 2 * e));
      }
      const double s = ldexp(1.0, -e);
      ar[v] = f.x * s, ai[v] = f.y * s, br[v] = f.z * s, bi[v] = f.w * s;
      if ((P.merges >> i) & 1) {
        const double pr = ar[v] + br[v], pi = ai[v] + bi[v], mr = ar[v] - br[v], mi = ai[v] - bi[v];
        ar[v] = pr, ai[v] = pi, br[v] = mr, bi[v] = mi;
      }
    }
    wts[i * T + tid] = BlockWeights<L>{L::pack(ar), L::pack(ai), L::pack(br), L::pack(bi)};
  }
  __syncthreads();

  const u64 groups = 1ull << P.lg;
  const u64 step = (u64)(gridDim.x >> lslices) << lslots;
  const ulonglong2* __restrict__ maps = reinterpret_cast<const ulonglong2*>(tables + P.tab_off);
  BlockStep g;
  g.in = reinterpret_cast<const char*>(Ein) + (size_t)b * (2 * sizeof(S));
  g.out = reinterpret_cast<char*>(Eout) + (size_t)b * (2 * sizeof(S));
  g.col = reinterpret_cast<char*>(smem) + tid * L::bytes;
  g.pitch = (unsigned)(2 * sizeof(S)) << lbt;
  S mx[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) mx[v] = (S)0;
#pragma unroll 1
  for (u64 gi = ((u64)(blockIdx.x >> lslices) << lslots) + (u64)(tid >> lcols); gi < groups; gi += step) {
    u64 rows = 0, flags = 0;
    for (int q = 0; q < P.nbytes; ++q) {
      const ulonglong2 t = __ldg(maps + (q << 8) + (int)((gi >> (8 * q)) & 255ull));
      rows ^= t.x;
      flags ^= t.y;
    }
    g.x0 = (unsigned)rows;
    g.xk = (unsigned)(rows >> 32);
    const unsigned fl = (unsigned)flags;
#pragma unroll 1
    for (int i = 0; i < P.stages; ++i) {
      const bool last = i + 1 == P.stages, fused = P.fused[i] != 0;
      const int pos = P.step[i];
      const unsigned f = fl >> (2 * pos);  // y and sign of the stage's position(s)
      const unsigned fb = fused ? f >> 2 : f;
      const unsigned unit = (unsigned)(T * L::bytes);
      g.pair = last ? __ldg(lin + (1 << P.din) + P.pair[i]) : (unsigned)P.pair[i] * unit;
      g.swap = (fb & 1u) ? g.pair : 0u;
      g.flip = (fb & 2u) ? 0xf0000000u : 0u;
      const BlockOp* op = ops + P.first[i];
      const BlockWeights<L> w = wts[(fused ? pos + 1 : pos) * T + tid];
      if (fused) {
        g.flip |= ((f & 2u) ? 0x0f000000u : 0u) | ((f & 1u) ? 0x00f00000u : 0u);
        g.twin = last ? __ldg(lin + (1 << P.din) + P.twin[i]) : (unsigned)P.twin[i] * unit;
        g.twin_sign = (unsigned)P.twin_sign[i] << 31;
        const BlockWeights<L> wp = wts[pos * T + tid];
        if (i == 0)
          block_stage<L, S, NV, true, true, false>(P.code[i], P.twin_order[i], op, P.rows[i], g, w, wp, mx);
        else if (last)
          block_stage<L, S, NV, true, false, true>(P.code[i], P.twin_order[i], op, P.rows[i], g, w, wp, mx);
        else
          block_stage<L, S, NV, true, false, false>(P.code[i], P.twin_order[i], op, P.rows[i], g, w, wp, mx);
      } else if (i == 0) {
        block_stage<L, S, NV, false, true, false>(P.code[i], 0, op, P.rows[i], g, w, w, mx);
      } else if (last) {
        block_stage<L, S, NV, false, false, true>(P.code[i], 0, op, P.rows[i], g, w, w, mx);
      } else {
        block_stage<L, S, NV, false, false, false>(P.code[i], 0, op, P.rows[i], g, w, w, mx);
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NV; ++v)
    if (mx[v] > (S)0) atomicMax(&maxrow[(size_t)(k - 1) * stride + b + v], max_bits<S>(mx[v]));
}

template <typename S, typename M, int NV, int MINB>
cudaError_t launch_block_as(int device, int sms, cudaStream_t s, const void* Ein, void* Eout, const DevBlock& P,
                            const u64* tables, const double4* W, const u64* mp, u64* mrow, int stride, int lbt,
                            int tiles, u64 es) {
  typedef BlockLane<S, M, NV> L;
  const size_t smem = block_smem_bytes<L>(P.dmax, P.k, P.words);
  static std::atomic<bool> configured[64];  // the attribute is per device; setting it twice is harmless
  if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
  if (!configured[device].load(std::memory_order_acquire)) {
    const cudaError_t e =
        cudaFuncSetAttribute(scan_block_kernel<S, M, NV, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)block_smem_bytes<L>(kBlockDim, kBlockLen, kBlockLen << kBlockEnds));
    if (e != cudaSuccess) return e;
    configured[device].store(true, std::memory_order_release);
  }
  const int lc = lbt - (NV == 2 ? 1 : 0);
  const int lcols = lc < kBlockLogThreads ? lc : kBlockLogThreads, lslices = lc - lcols, lslots = kBlockLogThreads - lcols;
  const u64 units = ((1ull << P.lg) + (1ull << lslots) - 1) >> lslots;  // group sets
  const u64 fit = 227 * 1024 / (smem + 1024);
  u64 per_slice = (((u64)sms * (fit < MINB ? fit : MINB)) >> lslices) / (u64)tiles;
  if (per_slice < 1) per_slice = 1;
  if (per_slice > units) per_slice = units;
  scan_block_kernel<S, M, NV, MINB><<<dim3((unsigned)(per_slice << lslices), (unsigned)tiles), kBlockThreads, smem, s>>>(
      (const S*)Ein, (S*)Eout, P, tables, W, mp, mrow, stride, lbt, es);
  return cudaGetLastError();
}

}  // namespace rgs
