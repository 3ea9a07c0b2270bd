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
  // Two strings per thread halve the index work but also the threads: from 2^20 of them in a
  // launch on one tile (always at the largest, 256: 16384 strings at rank 20 46.16 ms, with
  // that threshold 46.38), 2^18 on a chunk of tiles.  Whole sweeps, one string per thread / this
  // rule / two wherever the tile is not 1: n = 40, rank 18, tile 32 195 / 195 / 296 us, tile
  // 128 301 / 300 / 335; rank 20, tile 32 288 / 289 / 419, tile 128 562 / 507 / 543; rank 24,
  // tile 8 1088 / 903 / 984; rank 11, 16384 strings in chunks 425 / 402 / 407.
  const int least = tiles > 1 ? 18 : (lbt >= 8 ? 0 : 20);
  if (lbt >= 1 && ((unsigned long long)tiles << (P.lg + lbt - 1)) >= (1ull << least))
    return launch_block_as<float, float, 2, 8>(device, sms, s, Ein, Eout, P, tables, W, mp, mrow, stride, lbt, tiles,
                                                es);
  return launch_block_as<float, float, 1, 14>(device, sms, s, Ein, Eout, P, tables, W, mp, mrow, stride, lbt, tiles,
                                                es);
}

}  // namespace rgs
