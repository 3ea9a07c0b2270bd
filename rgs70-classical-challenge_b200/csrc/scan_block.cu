// scan_block_kernel instantiations: complex64 tables with float32 or float64 arithmetic,
// complex128 tables.
#include "common.hpp"
#include "scan.hpp"
#include "scan_block.cuh"

namespace rgs {

cudaError_t launch_block(int precision, int device, cudaStream_t s, const void* Ein, void* Eout, const DevBlock& P,
                         const u64* tables, const double4* W, const u64* mp, u64* mrow, int stride, int lbt, int tiles, u64 es) {
  const int sms = sm_count(device);
  if (precision == RGS_PREC_C128)
    return launch_block_as<double, double, 1, 8>(device, sms, s, Ein, Eout, P, tables, W, mp, mrow, stride, lbt, tiles,
                                                es);
  if (precision == RGS_PREC_C64)
    return launch_block_as<float, double, 1, 10>(device, sms, s, Ein, Eout, P, tables, W, mp, mrow, stride, lbt, tiles,
                                                es);
  if (lbt >= 1)
    return launch_block_as<float, float, 2, 8>(device, sms, s, Ein, Eout, P, tables, W, mp, mrow, stride, lbt, tiles,
                                                es);
  return launch_block_as<float, float, 1, 14>(device, sms, s, Ein, Eout, P, tables, W, mp, mrow, stride, lbt, tiles,
                                                es);
}

}  // namespace rgs
