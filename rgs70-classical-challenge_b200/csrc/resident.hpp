// Host interface of the on-chip sweeps (resident.cu): plans whose whole environment table
// is held in shared memory -- many small instances (amplitudes of given bitstrings and
// exact chain-rule samples) in one launch, or many strings of one plan.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

#include "plan.hpp"

namespace rgs {

// Launch variants of a batch: (threads per block, dynamic shared memory per block for the
// tables).  512 threads and 192 KiB hold the largest ranks; 128 threads and 56 KiB leave
// room for four blocks per SM, 36 KiB for six (fewer items per unit, more units at once).
// rgs_batch_tune picks.
constexpr int kResVariants = 3;
constexpr int kResThreadsOf[kResVariants] = {512, 128, 128};
constexpr int kResSmemOf[kResVariants] = {192 * 1024, 56 * 1024, 36 * 1024};
constexpr int kResSmemMax = 192 * 1024;
constexpr int kMaxWarpItems = 32;   // items of a one-warp unit (a power of two)
constexpr int kMaxBlockItems = 8;   // items of a larger unit
constexpr int kResPlanRank = 12;    // largest plan rank of resident_run_plan (every precision)
constexpr int kResMinUnits = 592;   // resident_run_plan: units below which strings do not share one (4 per SM)

// One instance of a batch.  Device pointers; outputs of an unused kind may be null.
struct ResInstance {
  const ResStep* steps;                  // n step records (the plan's device copy)
  const double* U;                       // complex128[n][2][2]
  const double* fvec;                    // contraction vectors complex128[count][n][2] instead of U and bits
  const unsigned long long* bits;        // given bitstrings uint64[count][2]
  const double* uniforms;                // samples: uniforms [count][n] instead of the Philox ones (may be null)
  void* out_value;                       // complex64/complex128[count]
  double* out_logscale;                  // float64[count]
  unsigned long long* sample_bits;       // uint64[nsamples][2]
  void* sample_value;                    // complex[nsamples]: amplitude of each sample
  double* sample_logscale;               // float64[nsamples]
  double* sample_logp;                   // float64 log p of samples / given strings (may be null)
  float* out_cond;                       // float32 [count][n] conditionals p(x_v = 1 | prefix) (may be null)
  long long count, nsamples;
  unsigned long long seed;               // Philox key of the samples
  int n;                                 // positions
  int nb;                                // items per work unit (power of two)
  int rmax;                              // largest table rank
  int has_fixed;                         // plan has fixed vertices (amplitudes only)
};

// One work unit: `num` consecutive items (amplitudes: kind 0, samples: kind 1) of one instance.
struct ResWork {
  int inst;
  int kind;
  long long first;
  int num;                               // 0: padding
  int wide;                              // the whole block runs the unit (else one warp)
};

// Device buffers of a prepared batch (owned; freed with the batch).
struct ResDevice {
  int device = -1;
  ResInstance* insts = nullptr;
  size_t insts_cap = 0;
  ResWork* work = nullptr;
  size_t work_cap = 0;
  int* status = nullptr;   // 1: a branch pair had zero mass
  long long nwork = 0, nblocks = 0;
  int variant = 0;         // launch variant the work list was prepared for
  ~ResDevice();
};

// Largest table rank a launch variant holds in shared memory for a precision.
int resident_max_rank(int precision, int variant = 0);
// Items per work unit for an instance of rank `rmax` (0 if it does not fit).
int resident_items(int rmax, int precision, int variant = 0, bool* wide = nullptr);
// Sets every instance's items per unit for `variant`, uploads the instance records and
// the cost-ordered work list (synchronous).
int resident_prepare(const std::vector<ResInstance>& insts, int precision, int variant, ResDevice& dev);
// Queues the launch on `stream`: resets the status, then runs every unit.  Capturable
// once prepared.
int resident_launch(const ResDevice& dev, int precision, cudaStream_t stream, int* blocks_out);

// One plan, many strings, one launch: kind 0 amplitudes of in.bits (or in.fvec), kind 1
// samples (sample_* outputs), kind 2 conditionals of in.bits.  `in` names the inputs and
// outputs; steps, n, rmax and nb are filled in.  *status is set to 1 on a zero-mass branch pair.
bool resident_plan_fits(const Plan& plan);
int resident_run_plan(const Plan& plan, const Plan::DeviceCopy& dc, int kind, int precision, ResInstance in, int device,
                      int* status, cudaStream_t stream);

}  // namespace rgs
