// On-chip sweeps: plans of rank <= 13, tables in shared memory, no launch per position.
//
// The streaming executor (scan.cu) runs one launch per scan position because a
// rank-30 table lives in HBM.  Plans of rank <= 13 (complex64) fit in shared memory, so
// a block runs a whole sweep -- every position of one instance for nb strings -- with no
// HBM traffic besides the inputs and the outputs.  Two callers:
//   * resident_launch: many uneven instances (ResidentBatch), one block per work unit,
//     largest units first;
//   * resident_run_plan: many strings of one plan, for the scan and the chain sampler.
// Kinds of work:
//   0  amplitudes of given bitstrings (the streaming executor's arithmetic, bit for bit:
//      same weights, same fma order, same renormalisation);
//   1  exact chain-rule samples (chain.cu's algorithm: both branch masses from the
//      position's Gram matrix, one read of the table, or in closed form; inverse-CDF
//      choice with the item's uniform; then the chosen branch as one step);
//   2  chain-rule conditionals of given bitstrings: as 1 with the branch given, so that
//      the Gram matrix and the step share one pass over the table.
// Table layout per block: E[c][b] (b fastest) for the unit's nb items.
//
// What bounds it: latency at low ranks (a position is a chain of reductions and weight
// arithmetic over a few rows), instruction issue and shared-memory bandwidth at ranks 9
// and up.  Hence
//   * one warp per block where the tables allow it (T = 32): positions are separated by
//     warp synchronisation, the maximum and the Gram sums by shuffles, and two dozen
//     independent sweeps per SM cover each other's latency; larger blocks only for ranks
//     whose tables leave an SM with few blocks;
//   * index work by GF(2) increments: the gathered row, its sign, and the output row of
//     row r are one linear word q(r) (ResStep), so a Gray-code walk advances all of them
//     with one XOR per row instead of byte-table loads, a popcount and a bit deposit;
//   * every thread derives its item's weights from the reduced maximum, so a position
//     costs one barrier (two in samples) and no serial phase of a few threads.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <numeric>

#include "common.hpp"
#include "philox.cuh"
#include "plan.hpp"
#include "resident.hpp"
#include "scan_device.cuh"

namespace rgs {

ResDevice::~ResDevice() {
  if (device < 0) return;
  int prev = -1;
  cudaGetDevice(&prev);
  cudaSetDevice(device);
  if (insts) cudaFree(insts);
  if (work) cudaFree(work);
  if (status) cudaFree(status);
  if (prev >= 0) cudaSetDevice(prev);
}

namespace {

constexpr unsigned kFull = 0xffffffffu;

template <typename S>
struct Pair2;
template <>
struct Pair2<float> {
  typedef float2 T;
};
template <>
struct Pair2<double> {
  typedef double2 T;
};

// x with its sign flipped where bit 31 of sgn is set (exact).
__device__ __forceinline__ float flip31(float x, unsigned sgn) { return __uint_as_float(__float_as_uint(x) ^ sgn); }
__device__ __forceinline__ double flip31(double x, unsigned sgn) {
  return __hiloint2double(__double2hiint(x) ^ (int)sgn, __double2loint(x));
}

// scale_exponent (scan_device.cuh) in the storage type.  `done` becomes 1 on a zero and 2
// on a non-finite maximum, with e = 0 from there on.
__device__ __forceinline__ int half_exponent(float m2, int& done) {
  const unsigned x = __float_as_uint(m2) >> 23;  // m2 >= 0
  int k = (int)x - 126;
  if (x - 1u >= 254u) {
    if (x == 0u && m2 > 0.f) {
      k = (int)(__float_as_uint(m2 * 0x1.0p64f) >> 23) - 126 - 64;
    } else {
      if (!done) done = x ? 2 : 1;
      return 0;
    }
  }
  return (k + 1) >> 1;
}
__device__ __forceinline__ int half_exponent(double m2, int& done) {
  const unsigned x = (unsigned)__double2hiint(m2) >> 20;
  int k = (int)x - 1022;
  if (x - 1u >= 2046u) {
    if (x == 0u && m2 > 0.0) {
      k = (int)((unsigned)__double2hiint(m2 * 0x1.0p64) >> 20) - 1022 - 64;
    } else {
      if (!done) done = x ? 2 : 1;
      return 0;
    }
  }
  return (k + 1) >> 1;
}
// 2^-e in the arithmetic type.  Scaling by it commutes with the rounding of the weights.
__device__ __forceinline__ void pow2_neg(int e, float& s) { s = __int_as_float((127 - e) << 23); }
__device__ __forceinline__ void pow2_neg(int e, double& s) { s = __hiloint2double((1023 - e) << 20, 0); }

// Weights of one item for one position before the power-of-two scale (scan_row_kernel's).
// A fixed vertex (f(y) with sign (-1)^{y par}) runs as a merge whose two weights differ in
// that sign.
template <typename M>
__device__ __forceinline__ void branch_weights(double2 f0, double2 f1, int mode, int yfix, Cx<M>& a, Cx<M>& b) {
  double ar = f0.x, ai = f0.y, br = f1.x, bi = f1.y;
  if (mode != MODE_PAIR) {
    if (mode == MODE_MERGE) {
      ar = f0.x + f1.x;
      ai = f0.y + f1.y;
      br = f0.x - f1.x;
      bi = f0.y - f1.y;
    } else if (yfix) {
      ar = f1.x;
      ai = f1.y;
      br = -f1.x;
      bi = -f1.y;
    } else {
      br = f0.x;
      bi = f0.y;
    }
  }
  a = Cx<M>{(M)ar, (M)ai};
  b = Cx<M>{(M)br, (M)bi};
}
template <typename M>
__device__ __forceinline__ Cx<M> scaled(const Cx<M>& w, M s) {
  return Cx<M>{w.re * s, w.im * s};
}

// A thread's walk over its rows of one position: rows slot + (Gray(k) << ls), k < iters.
struct Walk {
  unsigned q;      // word of the first row
  unsigned iters;  // rows of this thread (a power of two, or 0)
  int ls, lnb, b;  // log2 slots, log2 items, item
  unsigned mask, t, ovs;  // input row mask, pair offset, affine sign of the item (bit 31)
};

// One row (pair mode: a row pair) given its gathered entries: the Gram terms (GRAM: alpha
// and beta of every output, so that output = alpha f(0) + beta f(1); chain_gram_kernel's
// sums) and the step (STEP: outputs of the branch with weights wA, wB, maximum of |E|^2).
template <typename S, typename M, bool PAIR, int NC, int NG0, bool STEP, bool GRAM>
__device__ __forceinline__ void one_row(unsigned qu, const unsigned (&cm)[NC], const typename Pair2<S>::T (&e)[NC],
                                        typename Pair2<S>::T* __restrict__ Eout, const Walk& w, const Cx<M>& wA,
                                        const Cx<M>& wB, S& mx, double (&g)[4]) {
  typedef typename Pair2<S>::T V;
  if (GRAM) {
    double a0r = 0.0, a0i = 0.0, b0r = 0.0, b0i = 0.0, a1r = 0.0, a1i = 0.0, b1r = 0.0, b1i = 0.0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const unsigned sgn = ((qu ^ cm[c]) << 16) & 0x80000000u;
      const double er = (double)e[c].x, ei = (double)e[c].y;
      const double sr = flip31(er, sgn), si = flip31(ei, sgn);
      if (!PAIR || c < NG0) {
        a0r += er;
        a0i += ei;
        if (PAIR) {
          b1r += sr;
          b1i += si;
        } else {
          b0r += sr;
          b0i += si;
        }
      } else {
        a1r += er;
        a1i += ei;
        b0r += sr;
        b0i += si;
      }
    }
    g[0] = fma(a0r, a0r, fma(a0i, a0i, g[0]));
    if (!PAIR || NG0 < NC) {
      g[1] = fma(b0r, b0r, fma(b0i, b0i, g[1]));
      g[2] = fma(a0r, b0r, fma(a0i, b0i, g[2]));
      g[3] = fma(a0i, b0r, fma(-a0r, b0i, g[3]));
    }
    if (PAIR) {
      g[1] = fma(b1r, b1r, fma(b1i, b1i, g[1]));
      if (NG0 < NC) {
        g[0] = fma(a1r, a1r, fma(a1i, a1i, g[0]));
        g[2] = fma(a1r, b1r, fma(a1i, b1i, g[2]));
        g[3] = fma(a1i, b1r, fma(-a1r, b1i, g[3]));
      }
    }
  }
  if (STEP) {
    Cx<M> oa{(M)0, (M)0}, ob{(M)0, (M)0};
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const unsigned sgn = (((qu ^ cm[c]) << 16) & 0x80000000u) ^ w.ovs;
      const M er = (M)e[c].x, ei = (M)e[c].y;
      if (PAIR) {
        // wA terms first in both outputs (scan_row.cuh).
        if (c < NG0)
          cmad(oa, er, ei, wA);
        else
          cmad(oa, flip31(er, sgn), flip31(ei, sgn), wB);
        const int d = (c + NG0) % NC;
        const unsigned sgd = (((qu ^ cm[d]) << 16) & 0x80000000u) ^ w.ovs;
        const M dr = (M)e[d].x, di = (M)e[d].y;
        if (d < NG0)
          cmad(ob, flip31(dr, sgd), flip31(di, sgd), wB);
        else
          cmad(ob, dr, di, wA);
      } else {
        cmad(oa, er, ei, sgn ? wB : wA);
      }
    }
    const unsigned d0 = qu >> 16;
    const S ar = (S)oa.re, ai = (S)oa.im;
    Eout[(d0 << w.lnb) + w.b] = V{ar, ai};
    mx = fmax(mx, norm2(ar, ai));
    if (PAIR) {
      const S br = (S)ob.re, bi = (S)ob.im;
      Eout[((d0 ^ w.t) << w.lnb) + w.b] = V{br, bi};
      mx = fmax(mx, norm2(br, bi));
    }
  }
}

// Rows of one position for one thread.  U rows are gathered before any is used; fewer
// than U rows go one by one.
template <typename S, typename M, bool PAIR, int NC, int NG0, bool STEP, bool GRAM>
__device__ __forceinline__ void rows(const typename Pair2<S>::T* __restrict__ Ein,
                                     typename Pair2<S>::T* __restrict__ Eout, const unsigned* __restrict__ st,
                                     const Walk& w, const Cx<M>& wA, const Cx<M>& wB, S& mx, double (&g)[4]) {
  typedef typename Pair2<S>::T V;
  constexpr int U = NC == 1 ? 4 : (NC == 2 ? 2 : 1);
  constexpr int LU = NC == 1 ? 2 : (NC == 2 ? 1 : 0);
  unsigned cm[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) cm[k] = __ldg(st + 13 + k);
  unsigned q = w.q, left = w.iters;
  if (U > 1 && left < (unsigned)U) {
    for (unsigned k = 1; left > 0; --left, ++k) {
      V e[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) e[c] = Ein[(((q ^ cm[c]) & w.mask) << w.lnb) + w.b];
      one_row<S, M, PAIR, NC, NG0, STEP, GRAM>(q, cm, e, Eout, w, wA, wB, mx, g);
      if (left > 1) q ^= __ldg(st + w.ls + __ffs((int)k) - 1);
    }
    return;
  }
  unsigned off[U];
  off[0] = 0;
  if (U >= 2) off[1 % U] = __ldg(st + w.ls);
  if (U == 4) {
    off[3 % U] = __ldg(st + w.ls + 1);
    off[2 % U] = off[1 % U] ^ off[3 % U];
  }
#pragma unroll 1
  for (unsigned k = 1; left > 0; left -= U, ++k) {
    const unsigned delta = left > (unsigned)U ? __ldg(st + w.ls + LU + __ffs((int)k) - 1) : 0u;
    V e[U][NC];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int c = 0; c < NC; ++c) e[u][c] = Ein[(((q ^ off[u] ^ cm[c]) & w.mask) << w.lnb) + w.b];
#pragma unroll
    for (int u = 0; u < U; ++u)
      one_row<S, M, PAIR, NC, NG0, STEP, GRAM>(q ^ off[u], cm, e[u], Eout, w, wA, wB, mx, g);
    q ^= delta;
  }
}

template <typename S, typename M, bool STEP, bool GRAM>
__device__ __forceinline__ void rows_of(int code, const typename Pair2<S>::T* Ein, typename Pair2<S>::T* Eout,
                                        const unsigned* st, const Walk& w, const Cx<M>& wA, const Cx<M>& wB, S& mx,
                                        double (&g)[4]) {
  switch (code) {
    case RC_P1:
      // A Gram pass alone never meets this code (analytic branch masses).
      if (STEP) rows<S, M, true, 1, 1, STEP, false>(Ein, Eout, st, w, wA, wB, mx, g);
      break;
    case RC_P2H: rows<S, M, true, 2, 1, STEP, GRAM>(Ein, Eout, st, w, wA, wB, mx, g); break;
    case RC_P2F: rows<S, M, true, 2, 2, STEP, GRAM>(Ein, Eout, st, w, wA, wB, mx, g); break;
    case RC_P4H: rows<S, M, true, 4, 2, STEP, GRAM>(Ein, Eout, st, w, wA, wB, mx, g); break;
    case RC_P4F: rows<S, M, true, 4, 4, STEP, GRAM>(Ein, Eout, st, w, wA, wB, mx, g); break;
    case RC_M1: rows<S, M, false, 1, 1, STEP, GRAM>(Ein, Eout, st, w, wA, wB, mx, g); break;
    default: rows<S, M, false, 2, 2, STEP, GRAM>(Ein, Eout, st, w, wA, wB, mx, g); break;
  }
}

// max over the threads of an item; nonnegative IEEE values order as their bits.
__device__ __forceinline__ float lane_max(float x, int lnb) {
  unsigned v = __float_as_uint(x);
  if (lnb == 0) return __uint_as_float(__reduce_max_sync(kFull, v));
  for (int o = 16; o >> lnb; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o));
  return __uint_as_float(v);
}
__device__ __forceinline__ double lane_max(double x, int lnb) {
  for (int o = 16; o >> lnb; o >>= 1) x = fmax(x, __shfl_xor_sync(kFull, x, o));
  return x;
}

// Sum over the threads of an item in a warp of two doubles at once: the first exchange
// leaves each half of the threads with one of the two, the last hands both to everyone
// (12 shuffles instead of 20 at one item per warp).
__device__ __forceinline__ void lane_sum2(double& x, double& y, int lnb, int lane) {
  if (lnb == 5) return;
  const bool up = lane & 16;
  double mine = up ? y : x;
  const double other = up ? x : y;
  mine += __shfl_xor_sync(kFull, other, 16);
  for (int o = 8; o >> lnb; o >>= 1) mine += __shfl_xor_sync(kFull, mine, o);
  const double swapped = __shfl_xor_sync(kFull, mine, 16);
  x = up ? swapped : mine;
  y = up ? mine : swapped;
}

// One unit: `num` items (nb lanes' worth) of one instance through every position, by one
// warp (narrow) or by the whole block (wide).  The step records are read through L1,
// where every unit of the plan on the SM finds them.
// Shared memory: two tables of nb << rmax entries (dynamic; a narrow unit uses its warp's
// share); for wide units the warps' maxima (three positions deep, so that one barrier per
// position suffices) and branch masses.
template <int T>
struct UnitShared {
  static constexpr int kWarps = T / 32;
  static constexpr int kNb = T == 32 ? 1 : kMaxBlockItems;
  u64 max[3][kNb];
  double mass[kWarps][kNb][2];
};

template <typename S, typename M, int T, bool BATCH, int KIND>
__device__ __forceinline__ void run_unit(const ResInstance& in, long long first, int num, bool wide, unsigned char* smem,
                                         int table_bytes, UnitShared<T>& sh, int* __restrict__ status) {
  typedef typename Pair2<S>::T V;
  constexpr int kWarps = T / 32;
  constexpr int kNb = UnitShared<T>::kNb;
  constexpr int kLs = T == 32 ? 5 : (T == 128 ? 7 : 9);
  constexpr bool sample = KIND == 1, given = KIND == 2;
  if (T == 32) wide = false;
  auto& smax = sh.max;
  auto& smass = sh.mass;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto unit_sync = [&]() {
    if (wide)
      __syncthreads();
    else
      __syncwarp();
  };
  const int tid = wide ? threadIdx.x : lane;       // thread of the unit
  const int n = in.n, nb = in.nb, lnb = 31 - __clz(nb);
  const int b = tid & (nb - 1), slot = tid >> lnb, ls = (wide ? kLs : 5) - lnb;
  const int wslots = 32 >> lnb, wslot = lane >> lnb;  // threads per item in a warp, and which one this is
  const bool active = b < num;
  const long long item = first + b;
  const double2* __restrict__ U2 = (const double2*)in.U;
  const unsigned* __restrict__ st = (const unsigned*)in.steps;
  unsigned char* tab = smem;
  int half = table_bytes;
  if (BATCH && !wide) {
    half = table_bytes / kWarps;
    tab += 2 * warp * half;
  }
  const V* Ein = (const V*)tab;
  V* Eout = (V*)(tab + half);

  unsigned bits[4] = {0, 0, 0, 0};  // the item's bits (given, or drawn so far)
  u64 olo = 0, ohi = 0;             // affine syndrome offsets owed to later positions (fixed vertices)
  if (!sample && active && in.bits) {
    const u64 lo = in.bits[2 * item], hi = in.bits[2 * item + 1];
    bits[0] = (unsigned)lo;
    bits[1] = (unsigned)(lo >> 32);
    bits[2] = (unsigned)hi;
    bits[3] = (unsigned)(hi >> 32);
  }
  auto bit_at = [&](int v) {
    const unsigned w = (v & 64) ? ((v & 32) ? bits[3] : bits[2]) : ((v & 32) ? bits[1] : bits[0]);
    return (int)((w >> (v & 31)) & 1u);
  };
  // Contraction vectors of the next position, fetched one position ahead: f(0), f(1) of
  // the given bit (or of the caller's vectors), or both rows of U for branch masses.
  double2 f00, f01, f10, f11;
  f00 = f01 = f10 = f11 = make_double2(0.0, 0.0);
  auto fetch = [&](int v) {
    if (KIND == 0) {
      const double2* f = in.fvec ? (const double2*)in.fvec + ((size_t)(active ? item : first) * n + v) * 2
                                 : U2 + (v * 2 + bit_at(v)) * 2;
      f00 = f[0];
      f01 = f[1];
    } else {
      const double2* f = U2 + v * 4;
      f00 = f[0];
      f01 = f[1];
      f10 = f[2];
      f11 = f[3];
    }
  };
  if (wide)
    for (int i = tid; i < 3 * kNb; i += T) smax[i / kNb][i % kNb] = 0;
  if (slot == 0) ((V*)tab)[b] = V{(S)1, (S)0};
  unsigned first_col[kLs];  // all ones where this thread's slot has the bit
#pragma unroll
  for (int i = 0; i < kLs; ++i) first_col[i] = 0u - ((unsigned)(slot >> i) & 1u);
  uint4 w4 = __ldg((const uint4*)st + 4), w5 = __ldg((const uint4*)st + 5);
  fetch((int)w5.y);
  unit_sync();

  S m2 = (S)1;
  double logp = 0.0, uni = 0.0;
  double kept_x = 0.0, kept_1 = 0.0, kept_t = 1.0;  // masses of the position this thread records
  int esum = 0;
  int done = 0;  // 1: the table became zero, 2: non-finite
  bool bad = false;
  int r3 = 0;
#pragma unroll 1
  for (int j = 0; j < n; ++j, st += 32) {
    // Words 17..22: t, code, r_in, lrows, vertex, mode.
    const int code = (int)w4.z, lrows = (int)w5.x, v = (int)w5.y, mode = (int)w5.z;
    const double2 f0c = f00, f1c = f01, h0c = f10, h1c = f11;

    Walk w;
    w.ls = ls;
    w.lnb = lnb;
    w.b = b;
    w.mask = (1u << w4.w) - 1u;
    w.t = w4.y;
    w.ovs = 0;
    {
      // Word of this thread's first row: columns past the rank are zero.
      const uint4 c0 = __ldg((const uint4*)st), c1 = __ldg((const uint4*)st + 1);
      const unsigned col[9] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w, kLs > 8 ? __ldg(st + 8) : 0u};
      w.q = 0;
#pragma unroll
      for (int i = 0; i < kLs; ++i) w.q ^= col[i] & first_col[i];
    }
    w.iters = lrows >= ls ? (1u << (lrows - ls)) : (slot < (1 << lrows) ? 1u : 0u);
    if (j + 1 < n) {
      w4 = __ldg((const uint4*)st + 12);
      w5 = __ldg((const uint4*)st + 13);
      // The record after the next: a first sweep on this SM finds it in L1.
      if (j + 2 < n) asm volatile("prefetch.global.L1 [%0];" ::"l"(st + 64));
    }

    const int e = half_exponent(m2, done);
    esum += e;
    M sc;
    pow2_neg(e, sc);
    if (!active) sc = (M)0;
    Cx<M> wA, wB;
    S mx = (S)0;
    double g[4] = {0.0, 0.0, 0.0, 0.0};

    if (KIND == 0) {
      int y = 0;
      if (in.has_fixed) {
        const int ov = (int)((j < 64 ? (olo >> j) : (ohi >> (j - 64))) & 1ull);
        w.ovs = (unsigned)ov << 31;
        if (mode == MODE_FIXED) {
          y = hypot(f0c.x, f0c.y) > 1e-12 ? 0 : 1;
          if (y) {
            // Offsets of earlier positions are never read again.
            olo ^= (u64)__ldg(st + 23) | ((u64)__ldg(st + 24) << 32);
            ohi ^= (u64)__ldg(st + 25) | ((u64)__ldg(st + 26) << 32);
          }
        }
      }
      branch_weights<M>(f0c, f1c, mode, y, wA, wB);
      wA = scaled(wA, sc);
      wB = scaled(wB, sc);
      if (j + 1 < n) fetch((int)w5.y);
      rows_of<S, M, true, false>(code, Ein, Eout, st, w, wA, wB, mx, g);
    } else {
      const bool analytic = code == RC_P1;
      if (j + 1 < n) fetch((int)w5.y);
      // Uniforms of the next wslots positions, one per thread of the item.
      if (sample && (j & (wslots - 1)) == 0) {
        const int jj = j + wslot;
        uni = in.uniforms ? ((active && jj < n) ? in.uniforms[(size_t)item * n + jj] : 0.0)
                          : philox_uniform(in.seed, (u64)item, jj);
      }
      int x = 0;
      if (given) {
        x = bit_at(v);
        branch_weights<M>(x ? h0c : f0c, x ? h1c : f1c, mode, 0, wA, wB);
        wA = scaled(wA, sc);
        wB = scaled(wB, sc);
        rows_of<S, M, true, true>(code, Ein, Eout, st, w, wA, wB, mx, g);
      } else if (!analytic) {
        rows_of<S, M, false, true>(code, Ein, Eout, st, w, wA, wB, mx, g);
      }
      // Both branch masses (branch_mass of the Gram matrix): linear in the Gram sums, so
      // every thread applies it to its own sums and only the two masses are reduced.
      if (analytic) g[0] = g[1] = 1.0;
      double m0, m1;
      {
        const double zr0 = f0c.x * f1c.x + f0c.y * f1c.y, zi0 = f0c.y * f1c.x - f0c.x * f1c.y;
        const double zr1 = h0c.x * h1c.x + h0c.y * h1c.y, zi1 = h0c.y * h1c.x - h0c.x * h1c.y;
        m0 = g[0] * (f0c.x * f0c.x + f0c.y * f0c.y) + g[1] * (f1c.x * f1c.x + f1c.y * f1c.y) +
             2.0 * (g[2] * zr0 - g[3] * zi0);
        m1 = g[0] * (h0c.x * h0c.x + h0c.y * h0c.y) + g[1] * (h1c.x * h1c.x + h1c.y * h1c.y) +
             2.0 * (g[2] * zr1 - g[3] * zi1);
      }
      if (!analytic) {
        lane_sum2(m0, m1, lnb, lane);
        if (wide) {
          if (wslot == 0) {
            smass[warp][b % kNb][0] = m0;
            smass[warp][b % kNb][1] = m1;
          }
          __syncthreads();
          m0 = m1 = 0.0;
          for (int k = 0; k < kWarps; ++k) {
            m0 += smass[k][b % kNb][0];
            m1 += smass[k][b % kNb][1];
          }
        }
        m0 = m0 > 0.0 ? m0 : 0.0;
        m1 = m1 > 0.0 ? m1 : 0.0;
      }
      const double tot = m0 + m1;
      const bool wrong = !(tot > 0.0) || !isfinite(tot);
      bad |= wrong && active;
      if (sample) {
        // Inverse-CDF choice of x_v, and the chosen branch.
        const double un = __shfl_sync(kFull, uni, ((j & (wslots - 1)) << lnb) | (lane & (nb - 1)));
        x = (!wrong && !(un * tot < m0)) ? 1 : 0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if ((v >> 5) == i) bits[i] |= (unsigned)x << (v & 31);
        branch_weights<M>(x ? h0c : f0c, x ? h1c : f1c, mode, 0, wA, wB);
        wA = scaled(wA, sc);
        wB = scaled(wB, sc);
        rows_of<S, M, true, false>(code, Ein, Eout, st, w, wA, wB, mx, g);
      }
      // log p(x_v | prefix) and p(x_v = 1 | prefix): kept by one thread of the item per
      // position and evaluated for wslots positions at once.
      if (wslot == (j & (wslots - 1))) {
        kept_x = x ? m1 : m0;
        kept_1 = m1;
        kept_t = tot;
      }
      if (((j + 1) & (wslots - 1)) == 0 || j + 1 == n) {
        const int jj = (j & ~(wslots - 1)) + wslot;
        if (jj <= j) {
          logp += log(kept_x / kept_t);
          if (in.out_cond && (!wide || warp == 0) && active)
            in.out_cond[(size_t)item * n + jj] = (float)(kept_1 / kept_t);
        }
      }
    }

    // Maximum |E|^2 of the new table, per item.
    mx = lane_max(mx, lnb);
    if (wide) {
      const int r3n = r3 == 2 ? 0 : r3 + 1;
      if (wslot == 0) atomicMax(&smax[r3][b % kNb], max_bits<S>(mx));
      if (tid < kNb) smax[r3n][tid] = 0;
      __syncthreads();
      m2 = (S)max_value<S>(smax[r3][b % kNb]);
      r3 = r3n;
    } else {
      __syncwarp();
      m2 = mx;
    }
    const V* const in_table = Ein;
    Ein = Eout;
    Eout = const_cast<V*>(in_table);
  }
  half_exponent(m2, done);  // the last table's zero / non-finite bookkeeping
  if (bad) atomicExch(status, 1);
  if (KIND != 0)
    for (int o = 16; o >> lnb; o >>= 1) logp += __shfl_xor_sync(kFull, logp, o);
  if (slot == 0 && active) {
    const V fin = Ein[b];  // row 0 of the final table
    S re = fin.x, im = fin.y;
    if (done == 1) re = im = (S)0;
    if (done == 2) re = im = (S)NAN;
    const double lsc = (double)esum * 0.69314718055994530942;
    if (sample) {
      in.sample_bits[2 * item] = (u64)bits[0] | ((u64)bits[1] << 32);
      in.sample_bits[2 * item + 1] = (u64)bits[2] | ((u64)bits[3] << 32);
      reinterpret_cast<V*>(in.sample_value)[item] = V{re, im};
      in.sample_logscale[item] = lsc;
    } else {
      reinterpret_cast<V*>(in.out_value)[item] = V{re, im};
      in.out_logscale[item] = lsc;
    }
    if (KIND != 0 && in.sample_logp) in.sample_logp[item] = logp;
  }
}

// T: block size.  BATCH: units, kinds and instances from the work list (T / 32 entries
// per block, one per warp; a wide unit repeats its entry).  Else every unit is wide
// (T = 32: one warp) and KIND gives the work.
template <typename S, typename M, int T, int MINB, bool BATCH, int KIND>
__global__ void __launch_bounds__(T, MINB)
    resident_kernel(const __grid_constant__ ResInstance single, const ResInstance* __restrict__ insts,
                    const ResWork* __restrict__ work, int table_bytes, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ UnitShared<T> sh;
  if (BATCH) {
    const ResWork wk = work[(size_t)blockIdx.x * (T / 32) + (threadIdx.x >> 5)];
    if (wk.num == 0) return;  // padding of a block of narrow units
    if (wk.kind == 0)
      run_unit<S, M, T, BATCH, 0>(insts[wk.inst], wk.first, wk.num, wk.wide != 0, smem, table_bytes, sh, status);
    else
      run_unit<S, M, T, BATCH, 1>(insts[wk.inst], wk.first, wk.num, wk.wide != 0, smem, table_bytes, sh, status);
  } else {
    const long long first = (long long)blockIdx.x * single.nb;
    run_unit<S, M, T, BATCH, KIND < 0 ? 0 : KIND>(single, first, (int)min((long long)single.nb, single.count - first),
                                                  T > 32, smem, table_bytes, sh, status);
  }
}

// Dynamic shared memory above 48 KiB is an attribute of each kernel and device.
template <typename K>
int allow_smem(K kernel, int device, int bytes, bool (&done)[64]) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (device < 0 || device >= 64) return fail(RGS_ERR_ARG, "device ordinal above 63");
  if (!done[device]) {
    RGS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    RGS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      cudaSharedmemCarveoutMaxShared));
    done[device] = true;
  }
  return RGS_OK;
}

template <typename S, typename M, int T, int MINB, bool BATCH, int KIND>
int launch_units(int device, long long blocks, size_t smem, const ResInstance& single, const ResInstance* insts,
                 const ResWork* work, int* status, cudaStream_t stream) {
  static bool attr[64] = {false};
  int rc = allow_smem(resident_kernel<S, M, T, MINB, BATCH, KIND>, device, kResSmemMax, attr);
  if (rc) return rc;
  resident_kernel<S, M, T, MINB, BATCH, KIND>
      <<<(unsigned)blocks, T, smem, stream>>>(single, insts, work, (int)(smem / 2), status);
  RGS_CUDA_TRY(cudaGetLastError());
  return RGS_OK;
}

template <typename S, typename M>
int launch_batch(const ResDevice& dev, cudaStream_t stream) {
  const ResInstance none{};
#define RGS_BATCH(V_, MINB_) \
  launch_units<S, M, kResThreadsOf[V_], MINB_, true, -1>(dev.device, dev.nblocks, (size_t)kResSmemOf[V_], none, \
                                                         dev.insts, dev.work, dev.status, stream)
  if (dev.variant == 2) return RGS_BATCH(2, 6);
  if (dev.variant == 1) return RGS_BATCH(1, 4);
  return RGS_BATCH(0, 1);
#undef RGS_BATCH
}

template <typename S, typename M, int KIND>
int launch_plan(int threads, int device, long long units, size_t smem, const ResInstance& in, int* status,
                cudaStream_t stream) {
  if (threads == 32)
    return launch_units<S, M, 32, 16, false, KIND>(device, units, smem, in, nullptr, nullptr, status, stream);
  return launch_units<S, M, 128, 4, false, KIND>(device, units, smem, in, nullptr, nullptr, status, stream);
}

template <typename S, typename M>
int launch_kind(int kind, int threads, int device, long long units, size_t smem, const ResInstance& in, int* status,
                cudaStream_t stream) {
  if (kind == 0) return launch_plan<S, M, 0>(threads, device, units, smem, in, status, stream);
  if (kind == 1) return launch_plan<S, M, 1>(threads, device, units, smem, in, status, stream);
  return launch_plan<S, M, 2>(threads, device, units, smem, in, status, stream);
}

size_t esize_of(int precision) { return precision == RGS_PREC_C128 ? 16 : 8; }

size_t table_entries(int precision, int variant) { return (size_t)kResSmemOf[variant] / (2 * esize_of(precision)); }

}  // namespace

int resident_max_rank(int precision, int variant) {
  const size_t cap = table_entries(precision, variant);
  int r = 0;
  while (((size_t)2 << r) <= cap) ++r;
  return std::min(r, kResMaxRank);
}

// A unit is narrow (one warp, its share of the block's tables) where an item fits there.
int resident_items(int rmax, int precision, int variant, bool* wide) {
  if (wide) *wide = false;
  if (rmax < 0 || rmax > resident_max_rank(precision, variant)) return 0;
  const size_t cap = table_entries(precision, variant);
  const size_t share = cap / (kResThreadsOf[variant] / 32);
  const bool narrow = ((size_t)1 << rmax) <= share;
  int nb = narrow ? kMaxWarpItems : kMaxBlockItems;
  while (nb > 1 && ((size_t)nb << rmax) > (narrow ? share : cap)) nb >>= 1;
  if (wide) *wide = !narrow;
  return nb;
}

int resident_prepare(const std::vector<ResInstance>& insts_in, int precision, int variant, ResDevice& dev) {
  if (dev.device < 0) return fail(RGS_ERR_ARG, "batch has no device");
  if (variant < 0 || variant >= kResVariants) return fail(RGS_ERR_ARG, "unknown launch variant");
  std::vector<ResInstance> insts(insts_in);
  std::vector<char> wide(insts.size());
  for (size_t i = 0; i < insts.size(); ++i) {
    bool w = false;
    insts[i].nb = resident_items(insts[i].rmax, precision, variant, &w);
    wide[i] = w ? 1 : 0;
    if (insts[i].nb < 1) return fail(RGS_ERR_UNSUPPORTED, "an instance's tables do not fit this launch variant");
  }
  std::vector<ResWork> work;
  std::vector<double> cost;
  for (size_t i = 0; i < insts.size(); ++i) {
    const ResInstance& in = insts[i];
    const double c = (double)in.n * (double)(1ull << in.rmax);
    for (int kind = 0; kind < 2; ++kind) {
      const long long total = kind ? in.nsamples : in.count;
      for (long long f = 0; f < total; f += in.nb) {
        ResWork w;
        w.inst = (int)i;
        w.kind = kind;
        w.first = f;
        w.num = (int)std::min<long long>(in.nb, total - f);
        w.wide = wide[i];
        work.push_back(w);
        cost.push_back(kind ? 2.0 * c : c);
      }
    }
  }
  // Largest units first: blocks start in index order, so the short units fill the end.
  // Wide units take a block each; narrow units share a block, kWarps neighbours of the
  // order (similar length) at a time, the last block padded with empty entries.
  std::vector<size_t> idx(work.size());
  std::iota(idx.begin(), idx.end(), 0);
  std::stable_sort(idx.begin(), idx.end(), [&](size_t a, size_t b) { return cost[a] > cost[b]; });
  const size_t warps = (size_t)kResThreadsOf[variant] / 32;
  std::vector<ResWork> sorted;
  for (size_t k : idx)
    if (work[k].wide) sorted.insert(sorted.end(), warps, work[k]);
  for (size_t k : idx)
    if (!work[k].wide) sorted.push_back(work[k]);
  while (sorted.size() % warps) sorted.push_back(ResWork{});
  if (sorted.size() / warps > 0x7fffffffull) return fail(RGS_ERR_ARG, "more than 2^31 - 1 blocks in one batch");

  RGS_CUDA_TRY(cudaSetDevice(dev.device));
  if (!dev.status) RGS_CUDA_TRY(cudaMalloc(&dev.status, sizeof(int)));
  if (insts.size() > dev.insts_cap) {
    if (dev.insts) RGS_CUDA_TRY(cudaFree(dev.insts));
    dev.insts = nullptr;
    RGS_CUDA_TRY(cudaMalloc(&dev.insts, insts.size() * sizeof(ResInstance)));
    dev.insts_cap = insts.size();
  }
  if (sorted.size() > dev.work_cap) {
    if (dev.work) RGS_CUDA_TRY(cudaFree(dev.work));
    dev.work = nullptr;
    RGS_CUDA_TRY(cudaMalloc(&dev.work, sorted.size() * sizeof(ResWork)));
    dev.work_cap = sorted.size();
  }
  if (!insts.empty())
    RGS_CUDA_TRY(cudaMemcpy(dev.insts, insts.data(), insts.size() * sizeof(ResInstance), cudaMemcpyHostToDevice));
  if (!sorted.empty())
    RGS_CUDA_TRY(cudaMemcpy(dev.work, sorted.data(), sorted.size() * sizeof(ResWork), cudaMemcpyHostToDevice));
  dev.nwork = (long long)work.size();
  dev.nblocks = (long long)(sorted.size() / warps);
  dev.variant = variant;
  return RGS_OK;
}

int resident_launch(const ResDevice& dev, int precision, cudaStream_t stream, int* blocks_out) {
  if (dev.device < 0 || !dev.status) return fail(RGS_ERR_ARG, "batch is not prepared");
  RGS_CUDA_TRY(cudaSetDevice(dev.device));
  RGS_CUDA_TRY(cudaMemsetAsync(dev.status, 0, sizeof(int), stream));
  if (blocks_out) *blocks_out = (int)dev.nblocks;
  if (!dev.nwork) return RGS_OK;
  if (precision == RGS_PREC_C128) return launch_batch<double, double>(dev, stream);
  if (precision == RGS_PREC_C64_F32) return launch_batch<float, float>(dev, stream);
  return launch_batch<float, double>(dev, stream);
}

bool resident_plan_fits(const Plan& plan) { return !plan.res.empty() && plan.rmax <= kResPlanRank; }

int resident_run_plan(const Plan& plan, const Plan::DeviceCopy& dc, int kind, int precision, ResInstance in, int device,
                      int* status, cudaStream_t stream) {
  if (!resident_plan_fits(plan) || !dc.res) return fail(RGS_ERR_UNSUPPORTED, "plan rank above the on-chip maximum");
  if (in.count <= 0) return RGS_OK;
  in.steps = (const ResStep*)dc.res;
  in.n = plan.n;
  in.rmax = plan.rmax;
  in.has_fixed = 0;
  for (const PlanStep& p : plan.steps)
    if (!p.free) in.has_fixed = 1;
  const size_t item = 2 * esize_of(precision) << plan.rmax;  // both tables of one item
  // Threads per unit.  One warp while an SM holds seven units or more (32 KiB of tables
  // each), else four warps: every warp of a unit repeats the per-position work, which one
  // warp per unit pays once, but 64 KiB items leave three units per SM (8192 strings of
  // rank 10, complex64, float32 arithmetic: 183 us with one warp, 425 with four; rank 11:
  // 443 and 561; one string of rank 11 in samples: 105 and 94).
  const int threads = item <= 32 * 1024 ? 32 : 128;
  // Strings per unit: they share the per-position work, but larger units are fewer.
  // Amplitudes (and complex128) up to 1024 table entries per unit, complex64 samples up
  // to 2048, while the GPU keeps kResMinUnits of them (8192 strings of rank 7: 56 us with
  // one string per unit, 28 with eight; samples of rank 9: 235 and 198 with two; 1000
  // strings of rank 7: 22 with one, 27 with eight).
  const long long entries = (kind == 0 || precision == RGS_PREC_C128) ? 1024 : 2048;
  int nb = 1;
  if (threads == 32)
    while (nb < kMaxWarpItems && ((4ll * nb) << plan.rmax) <= entries && in.count >= 2ll * nb * kResMinUnits) nb *= 2;
  in.nb = nb;
  const long long units = (in.count + nb - 1) / nb;
  const size_t smem = (size_t)nb * item;
  if (units > 0x7fffffffll) return fail(RGS_ERR_ARG, "more than 2^31 - 1 work units in one call");
  if (precision == RGS_PREC_C128)
    return launch_kind<double, double>(kind, threads, device, units, smem, in, status, stream);
  if (precision == RGS_PREC_C64_F32)
    return launch_kind<float, float>(kind, threads, device, units, smem, in, status, stream);
  return launch_kind<float, double>(kind, threads, device, units, smem, in, status, stream);
}

}  // namespace rgs
