// Scan-program compiler (host).  Algorithm of W/upstream_scan/scan_plan.py:35-152
// (whyihaveyou/rgs70-classical-challenge), restated on 128-bit masks.
#include "plan.hpp"

#include <algorithm>
#include <cmath>
#include <map>

namespace rgs {

std::vector<u128> future_masks(int n, const std::vector<std::pair<int, int>>& edges,
                               const std::vector<int>& order) {
  // scan_plan.py:45-55 -- later neighbours of each position, as a mask over positions.
  std::vector<int> where(n, 0);
  for (int p = 0; p < n; ++p) where[order[p]] = p;
  std::vector<u128> later(n, 0);
  for (auto& e : edges) {
    int a = where[e.first], b = where[e.second];
    if (a > b) std::swap(a, b);
    later[a] |= one_at(b);
  }
  return later;
}

namespace {

// Reduce `vec` against `rows` in insertion order (scan_plan.py:35-42).  `used`
// collects the rows added, as a mask over row indices.
inline u128 eliminate(u128 vec, const std::vector<u128>& rows, const std::vector<int>& pivots, u128& used) {
  used = 0;
  for (size_t k = 0; k < rows.size(); ++k) {
    if (bit_of(vec, pivots[k])) {
      vec ^= rows[k];
      used |= one_at((int)k);
    }
  }
  return vec;
}

std::string validate(int n, const std::vector<std::pair<int, int>>& edges, const std::vector<int>& order,
                     const std::vector<uint8_t>& fixed) {
  if (n < 1 || n > 128) return "n must be in [1, 128]";
  if ((int)order.size() != n) return "order must have n entries";
  std::vector<char> seen(n, 0);
  for (int v : order) {
    if (v < 0 || v >= n || seen[v]) return "order must be a permutation of 0..n-1";
    seen[v] = 1;
  }
  for (auto& e : edges) {
    if (e.first < 0 || e.first >= n || e.second < 0 || e.second >= n) return "edge endpoint out of range";
    if (e.first == e.second) return "self-loop in edge list";
  }
  if (!fixed.empty() && (int)fixed.size() != n) return "fixed must have n entries";
  return "";
}

// Compiles the steps; when `keep` is false only ranks are recorded.
void run_compiler(int n, const std::vector<u128>& later, const std::vector<int>& order,
                  const std::vector<uint8_t>& fixed, bool keep, std::vector<PlanStep>& steps,
                  std::vector<int>& ranks) {
  std::vector<u128> basis;
  std::vector<u128> images, rows, columns;
  std::vector<int> pivots;
  ranks.assign(n, 0);
  if (keep) steps.assign(n, PlanStep());
  for (int j = 0; j < n; ++j) {
    const int v = order[j];
    const bool is_free = fixed.empty() || !fixed[v];
    const int r_in = (int)basis.size();
    u128 beta = 0;
    for (int i = 0; i < r_in; ++i)
      if (bit_of(basis[i], j)) beta |= one_at(i);
    images.clear();
    for (auto& b : basis) images.push_back(b & ~one_at(j));
    if (is_free) images.push_back(later[j]);
    rows.clear();
    pivots.clear();
    columns.clear();
    for (auto img : images) {
      u128 used;
      u128 res = eliminate(img, rows, pivots, used);
      if (res) {
        pivots.push_back(lowest_bit(res));
        rows.push_back(res);
        used |= one_at((int)rows.size() - 1);
      }
      columns.push_back(used);
    }
    const int r_out = (int)rows.size();
    ranks[j] = r_out;
    if (keep) {
      PlanStep& st = steps[j];
      st.v = v;
      st.free = is_free;
      st.r_in = r_in;
      st.r_out = r_out;
      st.beta = beta;
      // creator[k]: first column whose highest coefficient bit is k (scan_plan.py:79-83).
      std::vector<int> creator(r_out, -1);
      for (size_t i = 0; i < columns.size(); ++i) {
        if (!columns[i]) continue;
        int top = highest_bit(columns[i]);
        if (creator[top] < 0) creator[top] = (int)i;
      }
      // Right inverse (scan_plan.py:84-91).
      st.lcols.assign(r_out, 0);
      for (int k = 0; k < r_out; ++k) {
        const int i = creator[k];
        u128 pre = one_at(i);
        for (int l = 0; l < k; ++l)
          if (bit_of(columns[i], l)) pre ^= st.lcols[l];
        st.lcols[k] = pre;
      }
      // Kernel (scan_plan.py:92-102).
      st.kernel.clear();
      for (size_t i = 0; i < columns.size(); ++i) {
        if (std::find(creator.begin(), creator.end(), (int)i) != creator.end()) continue;
        u128 vec = one_at((int)i);
        for (int k = 0; k < r_out; ++k)
          if (bit_of(columns[i], k)) vec ^= st.lcols[k];
        st.kernel.push_back(vec);
      }
      st.ycol = is_free ? columns[r_in] : 0;
      st.mcols = columns;
    }
    basis.swap(rows);
  }
}

}  // namespace

void byte_tables(const std::vector<u128>& cols, int nbits, std::vector<u128>& out, int& nbytes) {
  // scan_plan.py:133-145
  nbytes = std::max(1, (nbits + 7) / 8);
  out.assign((size_t)nbytes * 256, 0);
  for (int b = 0; b < nbytes; ++b)
    for (int v = 1; v < 256; ++v) {  // entry of v: that of v without its lowest bit, and the bit's column
      const int i = 8 * b + __builtin_ctz((unsigned)v);
      out[(size_t)b * 256 + v] = out[(size_t)b * 256 + (v & (v - 1))] ^ (i < nbits ? cols[i] : (u128)0);
    }
}

std::vector<u128> kernel_combos(const std::vector<u128>& kernel) {
  // scan_plan.py:148-152 -- span in doubling order.
  std::vector<u128> out{0};
  for (auto k : kernel) {
    size_t m = out.size();
    for (size_t i = 0; i < m; ++i) out.push_back(out[i] ^ k);
  }
  return out;
}

std::string rank_profile(int n, const std::vector<std::pair<int, int>>& edges, const std::vector<int>& order,
                         const std::vector<uint8_t>& fixed, std::vector<int>& ranks) {
  std::string err = validate(n, edges, order, fixed);
  if (!err.empty()) return err;
  std::vector<PlanStep> unused;
  run_compiler(n, future_masks(n, edges, order), order, fixed, false, unused, ranks);
  return "";
}

void small_runs(const Plan& p, int& h, int& t) {
  auto small = [&](int j) { return std::max(p.steps[j].r_in, p.steps[j].r_out) <= kSmallRank; };
  h = 0;
  while (h < p.n && small(h)) ++h;
  t = p.n;
  while (t > h && small(t - 1)) --t;
}

namespace {

u128 apply_cols(const std::vector<u128>& cols, u128 x) {
  u128 r = 0;
  for (size_t i = 0; i < cols.size(); ++i)
    if (bit_of(x, (int)i)) r ^= cols[i];
  return r;
}

// Pair code of a step as it runs in a fused pair, or -1 if the pair kernel does not
// cover it.  `basis` receives the listing basis of the step's projected combos (kappa-0
// vectors first), used when the step is B.
int pair_code(const PlanStep& st, const DevStep& d, std::vector<u128>& basis) {
  basis.clear();
  if (!st.free) return -1;
  const u128 mask = one_at(st.r_in) - 1;
  if (d.mode == MODE_MERGE) {
    if (d.ncombos != 2) return -1;
    basis.push_back((u128)d.combos[1] & mask);
    return PC_M2;
  }
  if (d.mode != MODE_PAIR) return -1;
  if (d.ncombos == 1) return PC_P1;
  if (d.ncombos == 2) {
    basis.push_back(st.kernel[0] & mask);
    return bit_of(st.kernel[0], st.r_in) ? PC_P2H : PC_P2F;
  }
  // Four combos: one kappa-0 and one kappa-1 basis vector (kappa nonzero), else unsupported.
  const u128 k1 = st.kernel[0], k2 = st.kernel[1];
  const u128 cand[3] = {k1, k2, k1 ^ k2};
  u128 zero = 0, one = 0;
  bool has0 = false, has1 = false;
  for (u128 c : cand) {
    if (!bit_of(c, st.r_in) && !has0) {
      zero = c;
      has0 = true;
    } else if (bit_of(c, st.r_in) && !has1) {
      one = c;
      has1 = true;
    }
  }
  if (!has0 || !has1) return -1;
  basis.push_back(zero & mask);
  basis.push_back(one & mask);
  return PC_P4H;
}

// Echelon pivots (highest bits, ascending) of the span of `vecs`; false if dependent.
bool pivots_of(std::vector<u128> vecs, std::vector<int>& piv) {
  piv.clear();
  for (size_t i = 0; i < vecs.size(); ++i) {
    u128 v = vecs[i];
    for (size_t k = 0; k < i; ++k)
      if (bit_of(v, highest_bit(vecs[k]))) v ^= vecs[k];
    if (!v) return false;
    vecs[i] = v;
    // keep earlier vectors free of the new pivot so later reductions stay consistent
    for (size_t k = 0; k < i; ++k)
      if (bit_of(vecs[k], highest_bit(v))) vecs[k] ^= v;
    piv.push_back(highest_bit(v));
  }
  std::sort(piv.begin(), piv.end());
  return true;
}

// The pair record of positions j, j + 1, or false when they cannot be fused.
bool make_pair(Plan& p, int j, DevPair& out, std::vector<unsigned long long>& mb_tables) {
  const PlanStep& A = p.steps[j];
  const PlanStep& B = p.steps[j + 1];
  const DevStep& dA = p.dev[j];
  const DevStep& dB = p.dev[j + 1];
  std::vector<u128> basisA, basisB;
  const int cA = pair_code(A, dA, basisA);
  const int cB = pair_code(B, dB, basisB);
  if (cA < 0 || cB < 0) return false;
  const int m = A.r_out;
  if (B.r_in != m || m < 1) return false;
  const bool pairA = cA != PC_M2;
  const u128 tA = pairA ? A.ycol : 0;
  // t_A must lie outside span(basisB) (else W is smaller than the kernel assumes).
  std::vector<u128> listing;
  if (pairA) listing.push_back(tA);
  for (u128 b : basisB) listing.push_back(b);
  std::vector<int> piv;
  if (!pivots_of(listing, piv)) return false;
  const int dw = (int)listing.size();
  if (dw > 3 || dw > m) return false;
  const int nw = 1 << dw;
  auto w_of = [&](int i) {
    u128 w = 0;
    for (int k = 0; k < dw; ++k)
      if ((i >> k) & 1) w ^= listing[k];
    return w;
  };
  DevPair d{};
  d.j = j;
  d.codeA = cA;
  d.codeB = cB;
  d.a = A.r_in;
  d.m = m;
  d.o = B.r_out;
  d.maskA = (unsigned long long)(one_at(A.r_in) - 1);
  d.betaA = (unsigned long long)A.beta;
  for (int k = 0; k < 4; ++k) d.combA[k] = dA.combos[k];
  d.betaB = (unsigned long long)B.beta;
  d.tB = (unsigned long long)(cB == PC_M2 ? 0 : B.ycol);
  const int ncb = 1 << (int)basisB.size();
  const int na = ncb;  // A-units: pairs of registers (PAIR A) or single registers (MERGE A)
  for (int u = 0; u < na; ++u) {
    const u128 w = pairA ? w_of(2 * u) : w_of(u);
    d.LAw[u] = (unsigned long long)apply_cols(A.lcols, w);
  }
  const std::vector<u128> mB(B.mcols.begin(), B.mcols.begin() + m);
  d.MB0[0] = 0;
  d.MB0[1] = pairA ? (unsigned long long)apply_cols(mB, tA) : 0;
  d.pwB = 0;
  for (int i = 0; i < nw; ++i) {
    const u128 x = w_of(i) & B.beta;
    const int par = (__builtin_popcountll((uint64_t)x) + __builtin_popcountll((uint64_t)(x >> 64))) & 1;
    d.pwB |= (unsigned)par << i;
  }
  d.dw = dw;
  for (int k = 0; k < 3; ++k) d.piv[k] = k < dw ? piv[k] : 0;
  if (cB == PC_P2F || cB == PC_P4H || cB == PC_M2) {
    const int own = highest_bit(basisB[0]);
    if (std::find(piv.begin(), piv.end(), own) == piv.end()) return false;  // cannot happen: W contains basisB[0]
    d.swapB = pairA && bit_of(tA, own) ? 1 : 0;
  }
  d.tabA_off = dA.table_off;
  d.nbA = dA.nbytes;
  std::vector<u128> tab;
  int nb = 0;
  byte_tables(mB, m, tab, nb);
  if (nb != dA.nbytes) return false;
  // One 16-byte entry per (byte, value): A's table entry and M_B's, so the kernel reads
  // both maps of a group with one load per byte.
  if ((p.tables.size() + mb_tables.size()) & 1) mb_tables.push_back(0ull);
  d.tab2_off = p.tables.size() + mb_tables.size();
  d.nbMB = nb;
  for (size_t i = 0; i < tab.size(); ++i) {
    mb_tables.push_back(p.tables[dA.table_off + i]);
    mb_tables.push_back((unsigned long long)tab[i]);
  }
  out = d;
  return true;
}

// Chooses the fused pairs: non-overlapping (j, j + 1) with j >= 1 and j + 1 < n - 1 (the last
// position runs alone, scaled from the true maximum of the table before it: the exponents
// then sum to that maximum's own, whatever the passes before), inside one of the
// leading / middle / trailing runs, maximising the intermediate entries kept out of
// HBM (2^m each); rebuilds p.pairs and p.pair_at.
void build_pairs(Plan& p) {
  p.pairs.clear();
  p.pair_at.assign(p.n, -1);
  // Drop the byte tables of an earlier pair build (they follow the step tables).
  size_t step_tables = 0;
  for (auto& d : p.dev) step_tables = std::max(step_tables, (size_t)d.table_off + ((size_t)d.nbytes << 8));
  p.tables.resize(step_tables);
  if (!p.fuse || !p.exec_ok) return;
  for (auto& st : p.steps)
    if (!st.free) return;
  int h = 0, t = 0;
  small_runs(p, h, t);
  auto region = [&](int j) { return j < h ? 0 : (j < t ? 1 : 2); };
  std::vector<DevPair> cand(p.n);
  std::vector<char> ok(p.n, 0);
  std::vector<unsigned long long> scratch;
  for (int j = 1; j + 2 < p.n; ++j) {
    if (region(j) != region(j + 1)) continue;
    scratch.clear();
    ok[j] = make_pair(p, j, cand[j], scratch) ? 1 : 0;
  }
  std::vector<double> best(p.n + 2, 0.0);
  std::vector<char> take(p.n + 1, 0);
  for (int j = p.n - 1; j >= 0; --j) {
    best[j] = best[j + 1];
    if (ok[j]) {
      const double g = std::ldexp(1.0, p.steps[j].r_out) + best[j + 2];
      if (g > best[j]) {
        best[j] = g;
        take[j] = 1;
      }
    }
  }
  std::vector<unsigned long long> mb;
  for (int j = 0; j < p.n; ++j) {
    if (!take[j]) continue;
    DevPair d;
    make_pair(p, j, d, mb);
    p.pair_at[j] = (int)p.pairs.size();
    p.pairs.push_back(d);
    ++j;
  }
  p.tables.insert(p.tables.end(), mb.begin(), mb.end());
}

// A small subspace as a reduced echelon basis (highest-bit pivots, each pivot in one vector).
struct Subspace {
  static constexpr int kMax = 8;
  u128 basis[kMax];
  int piv[kMax];
  int n = 0;
  bool full = false;  // a vector beyond kMax was added
  int dim() const { return n; }
  bool add(u128 v) {
    for (int i = 0; i < n; ++i)
      if (bit_of(v, piv[i])) v ^= basis[i];
    if (!v) return false;
    if (n == kMax) {
      full = true;
      return false;
    }
    const int h = highest_bit(v);
    for (int i = 0; i < n; ++i)
      if (bit_of(basis[i], h)) basis[i] ^= v;
    basis[n] = v;
    piv[n++] = h;
    return true;
  }
  // Coordinates of v; false when v lies outside.
  bool coords(u128 v, unsigned& c) const {
    c = 0;
    for (int i = 0; i < n; ++i)
      if (bit_of(v, piv[i])) {
        c |= 1u << i;
        v ^= basis[i];
      }
    return !v;
  }
  u128 at(unsigned c) const {
    u128 v = 0;
    for (int i = 0; i < n; ++i)
      if ((c >> i) & 1) v ^= basis[i];
    return v;
  }
};

// apply_cols over the set bits of a row of at most 64 bits.
u128 apply_row(const std::vector<u128>& cols, u128 x) {
  u128 r = 0;
  for (uint64_t w = (uint64_t)x; w; w &= w - 1) r ^= cols[__builtin_ctzll(w)];
  return r;
}

// Closes D[level] over `v` and its images: M of the positions after a level, the c part of L
// of the positions before it, for levels 0 .. D.size() - 1 of the run from position j.
// False when a level outgrows kBlockEnds.
bool close_over(const Plan& p, int j, std::vector<Subspace>& D, int level, u128 v) {
  // Every added vector leaves at most two more to add: never more than the vectors that the
  // levels hold, plus one.
  struct {
    u128 x;
    int l;
  } todo[(kBlockLen + 1) * Subspace::kMax + 2];
  int top = 0;
  todo[top++] = {v, level};
  while (top) {
    --top;
    const u128 x = todo[top].x;
    const int l = todo[top].l;
    if (!D[l].add(x)) {
      if (D[l].full) return false;
      continue;
    }
    if (D[l].dim() > kBlockEnds) return false;
    if (l + 1 < (int)D.size()) todo[top++] = {apply_row(p.steps[j + l].mcols, x), l + 1};
    if (l > 0) {
      const PlanStep& st = p.steps[j + l - 1];
      todo[top++] = {apply_row(st.lcols, x) & (one_at(st.r_in) - 1), l - 1};
    }
  }
  return true;
}

// Appends position j + i to the closed levels D[0 .. i] of a run: the images of level i, the
// pair offset, the kernel.
bool extend_run(const Plan& p, int j, int i, std::vector<Subspace>& D) {
  const PlanStep& st = p.steps[j + i];
  if (!st.free || st.r_in > 31 || st.r_out > 31) return false;
  D.push_back(Subspace());
  const Subspace before = D[i];
  for (int b = 0; b < before.dim(); ++b)
    if (!close_over(p, j, D, i + 1, apply_row(st.mcols, before.basis[b]))) return false;
  if (st.ycol && !close_over(p, j, D, i + 1, st.ycol)) return false;
  for (u128 v : st.kernel)
    if (!close_over(p, j, D, i, v & (one_at(st.r_in) - 1))) return false;
  return true;
}

// The record of the run [j, j + k) with closed levels D, or false when they are too large.
// words_out: appends the run's tables (u64 words, offsets from the start of p.tables); null:
// feasibility only.
bool make_block(const Plan& p, int j, int k, const std::vector<Subspace>& D, DevBlock& out,
                std::vector<unsigned long long>* words_out) {
  if (k < 2 || k > kBlockLen || j < 1 || j + k > p.n) return false;
  auto cmask = [&](int i) { return one_at(p.steps[j + i].r_in) - 1; };
  // Stages, from the right: a growing position joins the next one unless its pair offset
  // lies in the next one's kernel (or the two are the whole run: the pair kernel's case).
  auto growing = [&](int i) { return p.dev[j + i].mode == MODE_PAIR && p.dev[j + i].ncombos == 1; };
  int stage_of[kBlockLen + 1] = {-1, -1, -1, -1, -1, -1, -1};  // 1: a fused stage starts here, 0: a single one
  for (int i = k - 1; i >= 0; --i) {
    bool join = k > 2 && i > 0 && growing(i - 1);
    if (join) {
      Subspace ker;
      for (u128 v : p.steps[j + i].kernel) ker.add(v & cmask(i));
      join = ker.add(p.steps[j + i - 1].ycol);
    }
    if (join) --i;
    stage_of[i] = join ? 1 : 0;
  }
  int dmax = 0;
  for (int i = 0; i <= k; ++i) {
    if (D[i].dim() > kBlockEnds) return false;
    if (i > 0 && i < k && stage_of[i] >= 0) dmax = std::max(dmax, D[i].dim());
  }
  if (dmax > kBlockDim) return false;
  if (!words_out) return true;  // feasible; the tables are built for chosen runs only
  DevBlock d{};
  d.j = j;
  d.k = k;
  d.r_in = p.steps[j].r_in;
  d.r_out = p.steps[j + k - 1].r_out;
  d.din = D[0].dim();
  d.dout = D[k].dim();
  d.dmax = dmax;
  d.lg = d.r_out - d.dout;
  std::vector<unsigned long long>& words = *words_out;
  auto parity = [](u128 x) {
    return (__builtin_popcountll((uint64_t)x) + __builtin_popcountll((uint64_t)(x >> 64))) & 1;
  };
  // Slots of the levels that have them: linear images of the local basis vectors.
  std::vector<std::vector<unsigned>> slot(k + 1);
  auto slot_of = [&](int i, unsigned c) {
    unsigned s = 0;
    for (size_t b = 0; b < slot[i].size(); ++b)
      if ((c >> b) & 1) s ^= slot[i][b];
    return s;
  };
  for (int i = 0; i < k; ++i)
    if (p.dev[j + i].mode == MODE_MERGE) d.merges |= 1u << i;
  std::vector<unsigned long long> prog;
  for (int i = 0; i < k;) {
    const bool fused = stage_of[i] == 1;
    const int ib = fused ? i + 1 : i, o = ib + 1;  // B's position, output level
    const PlanStep &sa = p.steps[j + i], &sb = p.steps[j + ib];
    const DevStep& db = p.dev[j + ib];
    const bool pair = db.mode == MODE_PAIR, last = o == k;
    // One position consumes one bit of the basis, so its kernel has one dimension without the
    // y column: four combos always include y bits (RC_P4H), and the run kernel has no RC_P4F.
    if (pair && db.ncombos == 4 && db.ng0 == 4) return false;
    // Input row (level i) of a row of level ib, and A's y bit there.
    auto input_of = [&](u128 row) { return fused ? apply_cols(sa.lcols, row) & cmask(i) : row; };
    unsigned tloc = 0, vloc = 0;
    if (pair && !D[o].coords(sb.ycol, tloc)) return false;
    if (fused && !D[o].coords(apply_cols(sb.mcols, sa.ycol), vloc)) return false;
    // Row operations: local output rows without the pivot coordinates of t and v.
    auto top = [](unsigned x) { return 31 - __builtin_clz(x); };
    const int pt = pair ? top(tloc) : -1;
    unsigned vred = vloc, tred = tloc;
    bool v_has_t = false, t_has_v = false;
    if (fused && pair && ((vloc >> pt) & 1)) {
      vred ^= tloc;
      v_has_t = true;
    }
    if (fused && !vred) return false;
    const int pv = fused ? top(vred) : -1;
    if (fused && pair && ((tloc >> pv) & 1)) {
      tred ^= vred;
      t_has_v = true;
    }
    // Slots of the output level.
    if (!last) {
      if (i == 0) {
        for (int b = 0; b < D[o].dim(); ++b) slot[o].push_back(1u << b);
      } else {
        Subspace span;
        for (unsigned s : slot[i]) span.add(s);
        auto fresh = [&]() -> unsigned {  // a slot bit outside the level's span
          for (int b = 0; b < kBlockDim; ++b) {
            Subspace t = span;
            if (t.add(one_at(b))) {
              span = t;
              return 1u << b;
            }
          }
          return 0u;
        };
        // Offsets between the inputs of one operation: images of B's kernel.
        std::vector<unsigned> offs;
        Subspace seen;
        for (u128 v : sb.kernel) {
          unsigned c = 0;
          const u128 in = input_of(v & cmask(ib));
          if (!in || !D[i].coords(in, c)) continue;
          if (seen.add(slot_of(i, c))) offs.push_back(slot_of(i, c));
        }
        size_t next = 0;
        auto take = [&]() { return next < offs.size() ? offs[next++] : fresh(); };
        const unsigned st = pair ? take() : 0u, sv = fused ? take() : 0u;
        if ((pair && !st) || (fused && !sv)) return false;
        const unsigned s_vred = sv ^ (v_has_t ? st : 0u), s_tred = st ^ (t_has_v ? s_vred : 0u);
        std::vector<unsigned> base(D[o].dim(), 0);
        for (int b = 0; b < D[o].dim(); ++b) {
          if (b == pt || b == pv) continue;
          unsigned c = 0;
          if (!D[i].coords(input_of(apply_cols(sb.lcols, D[o].at(1u << b)) & cmask(ib)), c)) return false;
          base[b] = slot_of(i, c);
        }
        slot[o].assign(D[o].dim(), 0);
        for (int b = 0; b < D[o].dim(); ++b) {
          unsigned c = 1u << b, s = 0;
          if (pair && ((c >> pt) & 1)) {
            c ^= tred;
            s ^= s_tred;
          }
          if (fused && ((c >> pv) & 1)) {
            c ^= vred;
            s ^= s_vred;
          }
          for (int q = 0; q < D[o].dim(); ++q)
            if ((c >> q) & 1) s ^= base[q];
          slot[o][b] = s;
        }
      }
    }
    auto place = [&](unsigned c) { return last ? c : slot_of(o, c); };
    const int sg = d.stages++;
    d.step[sg] = i;
    d.fused[sg] = fused ? 1 : 0;
    d.code[sg] = pair ? (db.ncombos == 1 ? RC_P1
                                         : (db.ncombos == 2 ? (db.ng0 == 2 ? RC_P2F : RC_P2H)
                                                            : (db.ng0 == 4 ? RC_P4F : RC_P4H)))
                      : (db.ncombos == 1 ? RC_M1 : RC_M2);
    d.first[sg] = (int)prog.size();
    d.pair[sg] = pair ? (int)place(tloc) : 0;
    d.twin[sg] = fused ? (int)place(vloc) : 0;
    d.twin_sign[sg] = fused ? parity(sa.ycol & sb.beta) : 0;
    if (fused) {
      const u128 off = (sa.ycol ^ apply_cols(sb.lcols, apply_cols(sb.mcols, sa.ycol))) & cmask(ib);
      while (d.twin_order[sg] < db.ncombos && (((u128)db.combos[d.twin_order[sg]] ^ off) & cmask(ib))) ++d.twin_order[sg];
      // Cannot happen: off lies in the kernel, and has y bit 0 like L_B M_B t_A and t_A.
      if (d.twin_order[sg] >= (pair ? db.ng0 : db.ncombos)) return false;
    }
    for (unsigned c = 0; c < (1u << D[o].dim()); ++c) {
      if ((pair && ((c >> pt) & 1)) || (fused && ((c >> pv) & 1))) continue;
      const u128 l0 = apply_cols(sb.lcols, D[o].at(c));
      const unsigned y0 = pair ? (unsigned)bit_of(l0, sb.r_in) : 0u;
      unsigned long long w = (unsigned long long)place(y0 ? c ^ tloc : c) << 32;
      for (int q = 0; q < db.ncombos; ++q) {
        const u128 row = (l0 ^ (u128)db.combos[q]) & cmask(ib);
        w |= (unsigned long long)parity(row & sb.beta) << (40 + q);
        u128 in = row;
        if (fused) {
          const u128 la = apply_cols(sa.lcols, row);
          in = la & cmask(i);
          w |= (unsigned long long)parity(in & sa.beta) << (44 + q);
          w |= (unsigned long long)bit_of(la, sa.r_in) << (48 + q);
        }
        unsigned loc = 0;
        if (!D[i].coords(in, loc)) return false;
        w |= (unsigned long long)(i == 0 ? loc : slot_of(i, loc)) << (8 * q);
      }
      prog.push_back(w);
      ++d.rows[sg];
    }
    i = o;
  }
  d.words = (int)prog.size();
  // Group maps of every group-index bit, then byte tables.
  std::vector<unsigned long long> rows_of(d.lg), flags_of(d.lg);
  int bit = 0;
  for (int pos = 0; pos < d.r_out; ++pos) {
    if (std::find(D[k].piv, D[k].piv + D[k].dim(), pos) != D[k].piv + D[k].dim()) continue;
    u128 x = one_at(pos);
    unsigned long long flags = 0;
    const unsigned long long outrow = (unsigned long long)x;
    for (int i = k - 1; i >= 0; --i) {
      const PlanStep& st = p.steps[j + i];
      const u128 q = apply_cols(st.lcols, x);
      x = q & cmask(i);
      flags |= (unsigned long long)bit_of(q, st.r_in) << (2 * i);
      flags |= (unsigned long long)parity(x & st.beta) << (2 * i + 1);
    }
    rows_of[bit] = (unsigned long long)x | (outrow << 32);
    flags_of[bit] = flags;
    ++bit;
  }
  d.nbytes = (d.lg + 7) / 8;
  if ((p.tables.size() + words.size()) & 1) words.push_back(0ull);
  d.tab_off = p.tables.size() + words.size();
  const size_t tab = words.size();
  words.resize(tab + (size_t)d.nbytes * 512, 0ull);
  for (int b = 0; b < d.nbytes; ++b)
    for (int v = 1; v < 256; ++v) {
      const int i = 8 * b + __builtin_ctz((unsigned)v);
      unsigned long long* e = &words[tab + 2 * ((size_t)b * 256 + v)];
      const unsigned long long* less = &words[tab + 2 * ((size_t)b * 256 + (v & (v - 1)))];
      e[0] = less[0] ^ (i < d.lg ? rows_of[i] : 0ull);
      e[1] = less[1] ^ (i < d.lg ? flags_of[i] : 0ull);
    }
  d.prog_off = p.tables.size() + words.size();
  words.insert(words.end(), prog.begin(), prog.end());
  d.lin_off = p.tables.size() + words.size();
  std::vector<unsigned> lin;
  for (unsigned c = 0; c < (1u << d.din); ++c) lin.push_back((unsigned)D[0].at(c));
  for (unsigned c = 0; c < (1u << d.dout); ++c) lin.push_back((unsigned)D[k].at(c));
  if (lin.size() & 1) lin.push_back(0u);
  for (size_t i = 0; i < lin.size(); i += 2) words.push_back((unsigned long long)lin[i] | ((unsigned long long)lin[i + 1] << 32));
  out = d;
  return true;
}

// Chooses the segments of positions [lo, hi) -- one position, a fused pair or a run --
// minimising the table entries read and written plus `launch` entries per segment.
void choose_runs(Plan& p, int lo, int hi, double launch, std::vector<DevBlock>& blocks, std::vector<int>& block_at,
                 std::vector<int>& run_len) {
  std::vector<double> best(p.n + 1, 0.0);
  std::vector<int> take(p.n + 1, 1);
  DevBlock d;
  for (int j = hi - 1; j >= lo; --j) {
    best[j] = HUGE_VAL;
    std::vector<Subspace> D;
    D.reserve(kBlockLen + 1);
    D.emplace_back();
    bool open = true;  // a longer run needs larger subspaces at every level
    for (int k = 1; k <= kBlockLen && j + k <= hi; ++k) {
      open = open && extend_run(p, j, k - 1, D);
      if (k > 1 && (!open || !make_block(p, j, k, D, d, nullptr))) {
        if (!open) break;
        continue;
      }
      const double c = std::ldexp(1.0, p.steps[j].r_in) + std::ldexp(1.0, p.steps[j + k - 1].r_out) + launch + best[j + k];
      if (c < best[j]) {
        best[j] = c;
        take[j] = k;
      }
    }
  }
  std::vector<unsigned long long> words;
  for (int j = lo; j < hi; j += take[j]) {
    run_len[j] = take[j];
    // Two positions that the pair kernel covers run there (its rows stay in registers).
    if (take[j] < 2 || (take[j] == 2 && p.pair_at[j] >= 0)) continue;
    std::vector<Subspace> D(1);
    bool ok = true;
    for (int i = 0; i < take[j]; ++i) ok = ok && extend_run(p, j, i, D);
    if (!ok || !make_block(p, j, take[j], D, d, &words)) {  // not reached: the run was found feasible
      blocks.clear();
      block_at.assign(p.n, -1);
      run_len.assign(p.n, 0);
      return;
    }
    block_at[j] = (int)blocks.size();
    blocks.push_back(d);
  }
  p.tables.insert(p.tables.end(), words.begin(), words.end());
}

// Runs of the middle positions of large plans (rank >= kBlockRank), and of every position
// but the last (see build_pairs) of plans whose tables are just small enough for chunks of
// tiles (kFlatRank and above).
void build_blocks(Plan& p) {
  p.blocks.clear();
  p.block_at.assign(p.n, -1);
  p.run_len.assign(p.n, 0);
  p.flat_blocks.clear();
  p.flat_at.assign(p.n, -1);
  p.flat_len.assign(p.n, 0);
  if (!p.fuse || !p.exec_ok || p.rmax > 31) return;
  for (auto& st : p.steps)
    if (!st.free) return;
  int h = 0, t = 0;
  small_runs(p, h, t);
  if (p.rmax >= kBlockRank && std::max(h, 1) < t)
    choose_runs(p, std::max(h, 1), t, 4096.0, p.blocks, p.block_at, p.run_len);
  if (p.rmax >= kFlatRank && p.rmax <= kSmallRank && p.n > 2)
    choose_runs(p, 1, p.n - 1, 256.0, p.flat_blocks, p.flat_at, p.flat_len);
}

// On-chip step records (plans of rank <= kResMaxRank): see ResStep.
void build_resident(Plan& p) {
  p.res.clear();
  if (p.rmax > kResMaxRank) return;
  for (int j = 0; j < p.n; ++j) {
    const DevStep& d = p.dev[j];
    const PlanStep& st = p.steps[j];
    ResStep r{};
    r.r_in = d.r_in;
    r.v = d.v;
    r.mode = d.mode;
    r.t = (unsigned)d.t;
    r.lrows = d.mode == MODE_PAIR ? d.r_out - 1 : d.r_out;
    auto parity = [&](unsigned long long c) {
      return (unsigned)(__builtin_popcountll(c & ((1ull << d.r_in) - 1ull) & d.beta) & 1);
    };
    for (int i = 0; i < r.lrows; ++i) {
      // Pair mode: the row index skips the pivot bit of t (deposit_zero).
      const int pos = (d.mode == MODE_PAIR && i >= d.pi) ? i + 1 : i;
      const unsigned long long l = (unsigned long long)st.lcols[pos];
      const unsigned y = (unsigned)((l >> d.r_in) & 1ull);
      const unsigned out = (1u << pos) ^ ((d.mode == MODE_PAIR && y) ? (unsigned)d.t : 0u);
      r.col[i] = (unsigned)l | (parity(l) << 15) | (out << 16);
    }
    for (int k = 0; k < d.ncombos; ++k) r.combo[k] = (unsigned)d.combos[k] | (parity(d.combos[k]) << 15);
    if (d.mode == MODE_PAIR)
      r.code = d.ncombos == 1 ? RC_P1
                              : (d.ncombos == 2 ? (d.ng0 == 2 ? RC_P2F : RC_P2H) : (d.ng0 == 4 ? RC_P4F : RC_P4H));
    else
      r.code = d.ncombos == 1 ? RC_M1 : RC_M2;
    const u128 f = p.future[j];
    for (int w = 0; w < 4; ++w) r.fut[w] = (unsigned)(f >> (32 * w));
    p.res.push_back(r);
  }
}

// Builds the device records; fails (without error) when a step is too wide to execute.
void build_device(Plan& p) {
  p.dev.clear();
  p.tables.clear();
  p.exec_ok = true;
  for (int j = 0; j < p.n; ++j) {
    const PlanStep& st = p.steps[j];
    if (st.r_in + 1 > 62 || st.r_out > 62) {
      p.exec_ok = false;
      p.exec_reason = "rank above 61 cannot be executed";
      p.dev.clear();
      p.tables.clear();
      return;
    }
    DevStep d{};
    d.beta = (unsigned long long)st.beta;
    d.r_in = st.r_in;
    d.r_out = st.r_out;
    d.v = st.v;
    d.fixed = st.free ? 0 : 1;
    std::vector<u128> tab;
    int nbytes = 0;
    byte_tables(st.lcols, st.r_out, tab, nbytes);
    d.nbytes = nbytes;
    d.table_off = p.tables.size();
    for (auto x : tab) p.tables.push_back((unsigned long long)x);
    std::vector<u128> combos = kernel_combos(st.kernel);
    if (!st.free) {
      d.mode = MODE_FIXED;
      d.t = 0;
      d.pi = 0;
    } else if (st.ycol != 0) {
      d.mode = MODE_PAIR;
      d.t = (unsigned long long)st.ycol;
      d.pi = highest_bit(st.ycol);
      // Combos with y bit 0 first (stable): the step kernel assigns the two output rows
      // of a pair by the y bit of the row's own image alone.
      std::stable_partition(combos.begin(), combos.end(), [&](u128 c) { return !bit_of(c, st.r_in); });
    } else {
      // e_y lies in the kernel: keep one representative per y pair (the one with y bit 0).
      d.mode = MODE_MERGE;
      d.t = 0;
      d.pi = 0;
      std::vector<u128> reps;
      for (auto c : combos)
        if (!bit_of(c, st.r_in)) reps.push_back(c);
      combos.swap(reps);
    }
    d.ncombos = (int)combos.size();
    d.ng0 = 0;
    for (auto c : combos)
      if (!bit_of(c, st.r_in)) ++d.ng0;
    for (int k = 0; k < 4; ++k) d.combos[k] = k < d.ncombos ? (unsigned long long)combos[k] : 0ull;
    p.dev.push_back(d);
  }
  build_resident(p);
  build_pairs(p);
  build_blocks(p);
}

}  // namespace

void plan_set_fusion(Plan& p, bool on) {
  p.fuse = on;
  build_pairs(p);
  build_blocks(p);
}

std::string compile_plan(int n, const std::vector<std::pair<int, int>>& edges, const std::vector<int>& order,
                         const std::vector<uint8_t>& fixed, Plan& out) {
  std::string err = validate(n, edges, order, fixed);
  if (!err.empty()) return err;
  out.n = n;
  out.order = order;
  out.fixed = fixed.empty() ? std::vector<uint8_t>(n, 0) : fixed;
  out.future = future_masks(n, edges, order);
  run_compiler(n, out.future, order, out.fixed, true, out.steps, out.ranks);
  out.rmax = 0;
  for (int r : out.ranks) out.rmax = std::max(out.rmax, r);
  for (auto& st : out.steps)
    if ((int)st.kernel.size() > 2) return "internal error: kernel dimension above 2";
  build_device(out);
  return "";
}

}  // namespace rgs
