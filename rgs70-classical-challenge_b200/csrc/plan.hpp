// Scan-program compiler: host side, exact GF(2) arithmetic on 128-bit masks.
//
// Compiles a vertex order of a graph with up to 128 vertices into the per-position
// scan program of whyihaveyou/rgs70-classical-challenge
// (W/upstream_scan/scan_plan.py:31-152, W/ = work/rgs_attack/): basis
// reduction in insertion order, lowest-set-bit pivots, the "first column with
// top coefficient k" right inverse and the kernel in column order.  The output is
// bit-identical to that compiler for every field it defines (v, free, r_in, r_out,
// beta, Lcols, kernel, future masks, byte tables, kernel combos); the device
// execution layout adds derived fields (see DevStep).
#pragma once
#include <cstdint>
#include <string>
#include <vector>

namespace rgs {

using u128 = unsigned __int128;

inline int lowest_bit(u128 x) {
  uint64_t lo = (uint64_t)x;
  if (lo) return __builtin_ctzll(lo);
  return 64 + __builtin_ctzll((uint64_t)(x >> 64));
}
inline int highest_bit(u128 x) {  // x != 0
  uint64_t hi = (uint64_t)(x >> 64);
  if (hi) return 127 - __builtin_clzll(hi);
  return 63 - __builtin_clzll((uint64_t)x);
}
inline bool bit_of(u128 x, int i) { return (x >> i) & 1; }
inline u128 one_at(int i) { return (u128)1 << i; }

struct PlanStep {
  int v = 0;
  bool free = true;
  int r_in = 0, r_out = 0;
  u128 beta = 0;               // bit i: basis vector i contains this position
  std::vector<u128> lcols;     // right inverse, r_out columns of r_in+free bits
  std::vector<u128> kernel;    // null space of (c, y) -> c', at most two vectors
  u128 ycol = 0;               // image of the y unit vector in new coordinates (free steps)
  std::vector<u128> mcols;     // the map (c, y) -> c' itself: image of input bit i (i < r_in + free)
};

// Execution modes of one step on the device (derived, not part of the reference plan).
enum StepMode : int {
  MODE_PAIR = 0,   // free, y image t != 0: outputs c' and c'^t read the same inputs
  MODE_MERGE = 1,  // free, y image t == 0: both y values of one input land on one output
  MODE_FIXED = 2,  // fixed vertex: y is known per bitstring
};

// Per-step record passed to the kernels by value.  Requires r_in + 1 <= 62.
struct DevStep {
  unsigned long long beta;
  unsigned long long t;          // pair partner offset (MODE_PAIR)
  unsigned long long combos[4];  // MODE_PAIR/FIXED: span(kernel); MODE_MERGE: y-bit-0 representatives
  unsigned long long table_off;  // offset (in u64) of this step's byte tables in the table blob
  int r_in, r_out, nbytes, ncombos, mode, pi, v, fixed;
  int ng0;                       // MODE_PAIR: the first ng0 combos have y bit 0 (the rest y bit 1)
};

// Step record of the on-chip sweep (resident.cu): 32 words, so that one warp fetches a
// record with one coalesced 128-byte load.  Everything a row needs follows from one
// GF(2)-linear word of the row index r, q(r) = XOR of col[i] over the set bits of r:
//   bits 0..14  L c' of the row's first output (c, and the y bit at r_in)
//   bit 15      parity(c & beta)
//   bits 16..   the output row that takes the kappa-0 combos' f(0) terms: c' itself or,
//               where the row's y bit is 1, its pair partner c' ^ t
// and combo k shifts bits 0..15 by the constant combo[k].  Ranks up to kResMaxRank.
constexpr int kResMaxRank = 13;
enum ResCode : int { RC_P1 = 0, RC_P2H = 1, RC_P2F = 2, RC_P4H = 3, RC_P4F = 4, RC_M1 = 5, RC_M2 = 6 };
struct ResStep {
  unsigned col[13];              // word of row-index bit i
  unsigned combo[4];             // the step's combos (order of DevStep), parity bit at 15
  unsigned t;                    // pair partner offset (0 in merge / fixed mode)
  int code;                      // ResCode: mode, number of combos, kappa pattern
  int r_in, lrows;               // input rank; log2 of the rows (pair mode: of row pairs)
  int v, mode;                   // vertex; StepMode
  unsigned fut[4];               // later-neighbour mask (fixed vertices)
  unsigned pad[5];
};
static_assert(sizeof(ResStep) == 128, "one 128-byte record per position");

// Two consecutive free positions A = j and B = j + 1 run as one pass (scan_pair_kernel):
// the intermediate table (A's output, B's input) stays in registers.  Rows of that
// table fall into groups, cosets q0 + W of a subspace W (dim <= 3) closed under A's
// output pairing and B's gathers; a group's inputs, its |W| intermediate rows and its
// outputs involve no row of another group.  Intermediate row i of a group is
// q0 ^ w_i, w_i = sum of listing-basis vectors by the bits of i: for PAIR A bit 0 is
// A's pair offset t_A and the higher bits (B-term index) span B's projected combos
// (kappa-0 vectors first); for MERGE A the bits span B's projected combos alone.
enum PairCode : int {
  PC_P1 = 0,   // PAIR, one combo
  PC_P2H = 1,  // PAIR, two combos, the second with y bit 1
  PC_P2F = 2,  // PAIR, two combos, both with y bit 0
  PC_P4H = 3,  // PAIR, four combos, the last two with y bit 1
  PC_M2 = 4,   // MERGE, two combos
};
constexpr int kPairCodes = 5;
struct DevPair {
  unsigned long long maskA, betaA;
  unsigned long long combA[4];   // A's combos (step order: kappa-0 first)
  unsigned long long LAw[4];     // L_A w of A-unit u's first row (with A's y bit)
  unsigned long long betaB;
  unsigned long long MB0[2];     // M_B (w | 0) of B-unit b's first row
  unsigned long long tB;         // B's output pair offset (PAIR B)
  unsigned long long tabA_off;   // A's byte tables (q -> L_A q over m bits)
  unsigned long long tab2_off;   // interleaved tables over m bits: entry (b, v) is the pair
                                 // (L_A part, M_B (. | 0) part), 16-byte aligned
  unsigned pwB;                  // bit i: parity(w_i & beta_B)
  int a;                         // r_in(A): A's y bit
  int m, o;                      // intermediate and output ranks
  int nbA, nbMB;                 // byte counts of the two tables
  int dw;                        // dim W: 2^(m - dw) groups
  int piv[3];                    // pivot bits of W (ascending): a group's q0 has zeros there
  int codeA, codeB;              // PairCode of A and B
  int j;                         // position A
  // Order of B's terms.  The unfused step sums over L_B c' ^ combos, where L_B c' has no bit
  // of B's kappa-0 kernel vector's own column (its highest bit).  q0 has none either (that
  // bit is a pivot of W); q0 ^ t_A has it where t_A does, and then the rows i ^ 2 of odd i
  // change places.
  int swapB;
};

// A run of k consecutive free positions j .. j + k - 1 as one pass (scan_block_kernel): the
// rows of every table of the run fall into groups, cosets of subspaces D_0 (input) .. D_k
// (output) closed under the run's gathers, so that the rows of one group at one level
// need only the group's rows of the level before.  A thread carries its strings' rows of a
// group through all k positions in its own shared-memory column.
// Level i of group g is x_i(g) + D_i, with x_k(g) = g with zeros deposited at the pivots of
// D_k and x_i the c part of L x_{i+1}; y_i is its y bit and s_i = parity(x_i & beta).  Local
// rows are coordinates in D_i; the local gathers, signs and destinations do not depend on
// g except through y_i (swaps a pair's outputs) and s_i (flips every sign).
// A stage is one position, or a growing position A (one combo, two outputs) with the next
// position B: B's gathers form A's outputs on the way, so the level between them needs no
// slots.  The other interior levels live in place: an output row takes the slot of one of
// its inputs (a stage that grows adds slot bits), so a column has 2^dmax slots.
constexpr int kBlockLen = 6;      // positions per run
// Dimension of interior levels with slots (16 per column).  32 slots halve the warps per
// SM for a few longer runs: 12.2 against 11.6 ms (float32 arithmetic, 4096 strings of the n =
// 40, rank 20 instance), 22.5 against 21.0 (complex128), 4.85 against 5.04 (rank 26).
constexpr int kBlockDim = 4;
constexpr int kBlockEnds = 6;     // dimension of D_0, D_k and of levels without slots
constexpr int kBlockRank = 18;    // runs are formed in plans of at least this rank,
constexpr int kFlatRank = 9;      // ... and over all positions from here to kSmallRank
struct DevBlock {
  int j, k;
  int r_in, r_out;
  int lg, nbytes;                 // log2 groups; byte tables of the group index
  int din, dout, dmax;
  int stages;
  int step[kBlockLen];            // first position of each stage (relative to j)
  int fused[kBlockLen];           // the stage is (A, B)
  int code[kBlockLen];            // ResCode of the stage's (last) position
  int rows[kBlockLen];            // row operations per group
  int first[kBlockLen];           // first program word
  int pair[kBlockLen];            // offset of a pair's second output (slot or local row)
  int twin[kBlockLen];            // fused: offset of the outputs of the partner gathers
  int twin_sign[kBlockLen];       // fused: parity(t_A & beta_B)
  // Fused: the twin of combo c's row is row c ^ twin_order of the twin operation's own sum
  // (L_B M_B t_A = t_A ^ combo[twin_order]; see DevPair::swapB).
  int twin_order[kBlockLen];
  unsigned merges;                // bit i: position j + i is a merge (weights f(0) +- f(1))
  int words;                      // program words
  unsigned long long tab_off;     // u64 index: per (byte, value) the pair (x_0 | x_k << 32,
                                  // y_i at bit 2 i and s_i at bit 2 i + 1), 16-byte aligned
  // Program word of a row operation: bits 8 c .. 8 c + 5 the slot (first stage: local
  // input row) of combo c, bits 32..37 the slot (last stage: local output row) of the
  // first output for y = 0, bit 40 + c the local sign of combo c; fused: bits 44 + c and
  // 48 + c the local sign and y bit of A at combo c's row.
  unsigned long long prog_off;
  unsigned long long lin_off;     // u32 tables: 2^din input rows, then 2^dout output rows
};

// Positions whose input and output ranks are both at most kSmallRank run once per chunk
// of tiles (scan.cu); a fused pair never straddles the leading / middle / trailing split.
constexpr int kSmallRank = 12;

struct Plan {
  int n = 0;
  std::vector<int> order;
  std::vector<uint8_t> fixed;        // per vertex
  std::vector<u128> future;          // per position
  std::vector<PlanStep> steps;
  std::vector<int> ranks;
  int rmax = 0;
  // Derived execution data (valid when executable()).
  std::vector<DevStep> dev;
  std::vector<ResStep> res;                // on-chip step records (rmax <= kResMaxRank, else empty)
  std::vector<unsigned long long> tables;  // concatenated byte tables
  // Fused pairs: pair_at[j] >= 0 when positions j and j + 1 run as pairs[pair_at[j]].
  std::vector<DevPair> pairs;
  std::vector<int> pair_at;
  bool fuse = true;                        // build fused pairs (plan_set_fusion)
  // Runs of positions as one pass: block_at[j] >= 0 when blocks[block_at[j]] starts at j.
  // run_len[j]: positions of the segment that starts at j (1: alone, 2 without a block: a
  // fused pair), 0 where no segment starts or outside the middle positions.
  std::vector<DevBlock> blocks;
  std::vector<int> block_at, run_len;
  // The same over every position but the first and the last (kFlatRank <= rank <= kSmallRank).
  std::vector<DevBlock> flat_blocks;
  std::vector<int> flat_at, flat_len;
  bool exec_ok = false;
  std::string exec_reason;
  // Device copies, per device ordinal (created lazily by the executor).
  struct DeviceCopy {
    int device = -1;
    void* res = nullptr;      // ResStep[n] (plans of rank <= kResMaxRank)
    void* tables = nullptr;   // u64[tables.size()]
    void* verts = nullptr;    // DevVert[n]
  };
  std::vector<DeviceCopy> device_copies;
  ~Plan();
};

// Vertex record for the per-bitstring weight kernel.
struct DevVert {
  unsigned long long fut_lo, fut_hi;  // future-neighbour mask of this position
  int v;
  int fixed;
};

// Returns an empty string on success, else an error message.
std::string compile_plan(int n, const std::vector<std::pair<int, int>>& edges,
                         const std::vector<int>& order, const std::vector<uint8_t>& fixed, Plan& out);

std::vector<u128> future_masks(int n, const std::vector<std::pair<int, int>>& edges,
                               const std::vector<int>& order);

// Rank profile only (no step data kept); used by the order search.
std::string rank_profile(int n, const std::vector<std::pair<int, int>>& edges, const std::vector<int>& order,
                         const std::vector<uint8_t>& fixed, std::vector<int>& ranks);

// Scan-order search (order_search.cpp): annealing over orders for sum_j 2^{r_j} under
// max r_j <= max_rank (< 0: the starting order's), `threads` independent chains of
// `iterations` proposals each; deterministic for (seed, threads, iterations).  Plans
// without fixed vertices.  Returns an empty string on success, else an error message.
std::string order_search(int n, const std::vector<std::pair<int, int>>& edges, const std::vector<int>& start,
                         int max_rank, long long iterations, uint64_t seed, int threads, std::vector<int>& best_order,
                         std::vector<int>& best_ranks, double& best_cost);

// Byte tables of one step: out[b * 256 + value] = XOR of lcols[8 b + t] over set bits t of value.
void byte_tables(const std::vector<u128>& cols, int nbits, std::vector<u128>& out, int& nbytes);

std::vector<u128> kernel_combos(const std::vector<u128>& kernel);

// Leading / trailing runs of low-rank positions (input and output rank <= kSmallRank):
// positions [0, h) and [t, n) (h <= t).
void small_runs(const Plan& p, int& h, int& t);

// Turns pair fusion on or off (rebuilds the pair records; the device copies are
// refreshed by the executor).
void plan_set_fusion(Plan& p, bool on);

}  // namespace rgs

// Opaque handle of the C ABI (include/rgs_b200.h).
struct rgs_plan {
  rgs::Plan plan;
};
