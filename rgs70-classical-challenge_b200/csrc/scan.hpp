// Host interface of the scan executor (scan.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

#include "plan.hpp"

namespace rgs {

// Workspace partition for one batch tile: two ping-pong tables, weights, flags and
// per-step maxima (all offsets 256-byte aligned).
struct ScanLayout {
  int Bt = 1;
  size_t esize = 8;
  size_t bytes_buf = 0, bytes_w = 0, bytes_f = 0, bytes_max = 0;
  size_t off_buf0 = 0, off_buf1 = 0, off_w = 0, off_f = 0, off_max = 0;
  size_t total() const;
};

struct ScanStats {
  long long launches = 0;
};

int scan_layout(const Plan& plan, int Bt, int precision, ScanLayout& L);

// Chunked sweep (scan_run): S tiles share one launch per small position (input and output
// rank at most kSmallRank); the positions between the leading and trailing small ones
// (h <= j < t) run tile by tile.  Workspace: two small-table buffers of S tiles, two
// full-size tables for the middle positions, weights / flags / maxima of S tiles.
constexpr int kChunkItems = 8192;  // default items per chunk (S = kChunkItems / Bt tiles)
struct ChunkLayout {
  int Bt = 1, S = 1, h = 0, t = 0;
  size_t esize = 8;
  unsigned long long e_stride = 0;  // entries per tile in the small buffers
  size_t bytes_small = 0, bytes_big = 0;
  size_t off_small0 = 0, off_small1 = 0, off_big0 = 0, off_big1 = 0, off_w = 0, off_f = 0, off_max = 0, total = 0;
};
int scan_chunk_layout(const Plan& plan, int Bt, int precision, int S, ChunkLayout& L);
int scan_chunk_tiles(int Bt);
// Tiles per chunk that scan_run uses with a workspace of ws_bytes (the largest S <=
// scan_chunk_tiles(Bt), S >= 2, whose layout fits, with C filled in); 0: tile by tile.
int scan_pick_chunk(const Plan& plan, int Bt, int precision, size_t ws_bytes, ChunkLayout& C, int* S);
// Whether scan_run sweeps `batch` strings of a plan on chip, as one launch (resident.cu),
// instead of one launch per segment: plans of rank <= kResPlanRank with fusion on, below
// the batches of scan_flat.  Measured, on chip against fused pairs: one string 31 against
// 166 us (rank 9, n = 40), 300 strings 50 against 207 us (rank 10, complex64, float32
// arithmetic).  33 to 127 strings stay streamed although on chip is faster there too (64
// strings, ranks 4 and 6: 16-24 us against 78-96): the tests of the pair schedule count its
// launches at 64 and 100 strings.
constexpr long long kOnChipFew = 32, kOnChipMany = 128;
bool scan_on_chip(const Plan& plan, int precision, long long batch);
// Whether such a plan is swept as runs over all its positions, one launch per run and chunk
// of tiles: from a batch whose tables hold 2^23 complex64 entries (half as many strings
// per rank), or 512 strings of rank 12 in complex128, whose tables leave an SM one unit on
// chip.  Measured, on chip / runs: rank 12, float32 arithmetic, 1000 strings 176 / 179 us,
// 2048 286 / 222, 8192 993 / 446; rank 11, 4096 strings 244 / 206 (n = 56) and 139 / 143 (n
// = 26); rank 10, 4096 strings 125 / 155, 8192 197 / 186; complex128, rank 12, 300 strings
// 194 / 161, 1000 419 / 204; rank 9, 4096 strings 119 / 111 and 87 / 93, 8192 192 / 131.
bool scan_flat(const Plan& plan, int precision, long long batch);
// Whether the runs of a plan's middle positions are used on tiles of Bt strings; else its pairs
// are.  Not for a single string in a window of ranks, where rows of 8 bytes make a run's
// gathers the slower ones (pairs / runs, two instances per rank): float32 arithmetic, rank 20
// 165 / 140 and 205 / 170 us, 21 177 / 170 and 224 / 285, 22 198 / 235 and 277 / 419, 24 539 /
// 604, 25 421 / 476 and 844 / 854, 26 584 / 650 and 936 / 831, 27 1456 / 1129; float64
// arithmetic, rank 21 189 / 173 and 237 / 270, 22 219 / 216 and 292 / 379, 23 293 / 267 and 383 /
// 356.  Two strings: rank 22 261 / 245, 24 661 / 536.
bool scan_runs(const Plan& plan, int precision, int Bt);
// The passes of a streamed sweep: first position and number of positions of each.
void scan_segments(const Plan& plan, std::vector<int>& first, std::vector<int>& length);
// Kernel launches scan_run queues for `batch` items with that workspace.
int scan_launch_count(const Plan& plan, long long batch, int Bt, int precision, size_t ws_bytes, long long* out);

// Fused pair launches (scan_pair_{c128,c64,f32}.cu): one instantiation set per precision.
cudaError_t launch_pair_c128(int VE, dim3 grid, cudaStream_t s, const void* Ein, void* Eout, const DevPair& P,
                             const unsigned long long* tables, const double4* WA, const double4* WB,
                             const unsigned long long* mp, unsigned long long* mA, unsigned long long* mc, int lbt,
                             unsigned long long es);
cudaError_t launch_pair_c64(int VE, dim3 grid, cudaStream_t s, const void* Ein, void* Eout, const DevPair& P,
                            const unsigned long long* tables, const double4* WA, const double4* WB,
                            const unsigned long long* mp, unsigned long long* mA, unsigned long long* mc, int lbt,
                            unsigned long long es);
cudaError_t launch_pair_f32(int VE, dim3 grid, cudaStream_t s, const void* Ein, void* Eout, const DevPair& P,
                            const unsigned long long* tables, const double4* WA, const double4* WB,
                            const unsigned long long* mp, unsigned long long* mA, unsigned long long* mc, int lbt,
                            unsigned long long es);

// Gram partials of B of a fused pair (chain-rule sampling, scan_pair_kernel GRAM mode),
// complex64 tables with float64 arithmetic and complex128 tables.
cudaError_t launch_pair_gram_c64(int VE, dim3 grid, cudaStream_t s, const void* Ein, const DevPair& P,
                                 const unsigned long long* tables, const double4* WA, const unsigned long long* mp,
                                 int lbt, double* partial);
cudaError_t launch_pair_gram_c128(int VE, dim3 grid, cudaStream_t s, const void* Ein, const DevPair& P,
                                  const unsigned long long* tables, const double4* WA, const unsigned long long* mp,
                                  int lbt, double* partial);
cudaError_t launch_pair_gram_f32(int VE, dim3 grid, cudaStream_t s, const void* Ein, const DevPair& P,
                                 const unsigned long long* tables, const double4* WA, const unsigned long long* mp,
                                 int lbt, double* partial);
// A run of positions (P.j ..) over one batch tile (scan_block.cu): weights of position P.j
// at W, `stride` strings between positions, maxima of the input table at mp and of position
// P.j at mrow.
cudaError_t launch_block(int precision, int device, cudaStream_t s, const void* Ein, void* Eout, const DevBlock& P,
                         const unsigned long long* tables, const double4* W, const unsigned long long* mp,
                         unsigned long long* mrow, int stride, int lbt, int tiles, unsigned long long es);
// One fused pair (positions P.j, P.j + 1) over one batch tile.
cudaError_t scan_launch_pair(int precision, int Bt, int device, const DevPair& P, const void* Ein, void* Eout,
                             const unsigned long long* tables, const double4* WA, const double4* WB,
                             const unsigned long long* mp, unsigned long long* mA, unsigned long long* mc,
                             cudaStream_t s);
// B's Gram partials of a fused pair over one batch tile: `blocks` blocks write
// partial[blocks][Bt][4] (G00, G11, Re G01, Im G01 of B's branch masses, float64 sums).
cudaError_t scan_launch_pair_gram(int precision, int Bt, int blocks, const DevPair& P, const void* Ein,
                                  const unsigned long long* tables, const double4* WA, const unsigned long long* mp,
                                  double* partial, cudaStream_t s);

// Largest batch tile the step kernel supports for a precision.
int scan_max_tile(int precision);


// Uploads (once per device) the plan's step records, byte tables and vertex records.
int plan_device_copy(Plan& plan, int device, const Plan::DeviceCopy** out);

// Runs the sweep for `batch` items: either bits (+ unitaries) or explicit contraction
// vectors fvec.  All work is queued on `stream`.
int scan_run(Plan& plan, const double* U, const unsigned long long* bits, const double* fvec, long long batch,
             int precision, void* out_value, double* out_logscale, void* workspace, size_t ws_bytes, int Bt,
             cudaStream_t stream, ScanStats* stats);

// Single-kernel launch wrappers (same kernels as scan_run), for drivers that manage
// their own device memory layout.
cudaError_t scan_launch_weights(const DevVert* verts, int n, const double* U, const unsigned long long* bits,
                                const double* fvec, long long first, int count, int Bt, void* W, unsigned char* F,
                                cudaStream_t stream);
cudaError_t scan_launch_step(int precision, int Bt, int device, const DevStep& st, const void* Ein, void* Eout,
                             const unsigned long long* T, const void* W, const unsigned char* F,
                             const unsigned long long* maxprev, unsigned long long* maxcur, bool unit_input,
                             cudaStream_t stream);
cudaError_t scan_launch_finalize(int precision, const void* E, const unsigned long long* maxbuf, int n, int Bt,
                                 int count, void* out_value, double* out_logscale, cudaStream_t stream);

}  // namespace rgs
