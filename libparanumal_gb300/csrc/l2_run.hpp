// Extent of an L2 request for the geometric factors of a run of elements. No CUDA in it, so
// that it can be checked on the host.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define LPG_HD __host__ __device__ __forceinline__
#else
#define LPG_HD inline
#endif

namespace lpg {

struct L2Run {
  uint64_t lo, bytes;   // address and length, whole 16-byte units; bytes = 0: nothing to ask for
};

// the whole 16-byte units inside `bytes` bytes at p
LPG_HD L2Run l2_units(uint64_t p, uint64_t bytes) {
  const uint64_t lo = (p + 15) & ~(uint64_t)15, hi = (p + bytes) & ~(uint64_t)15;
  return {lo, hi > lo ? hi - lo : 0};
}

// the factors of n >= 1 elements, `stride` entries of `size` bytes apart, from the first entry
// of the first element to the last one that is read of the last element: its six rows of Np
// factors, and the row of wJ where that is read (mass) and lies behind them (wJ and wJStride
// say so). The caller's array may end there, so a full stride of the last element is not asked for.
LPG_HD L2Run l2_factor_run(uint64_t ggeo, int64_t stride, uint64_t wJ, int64_t wJStride, int Np, int size, int64_t n,
                           bool mass) {
  const bool packed = mass && wJ == ggeo + (uint64_t)6 * Np * size && (wJStride == stride || n == 1);
  return l2_units(ggeo, (uint64_t)((n - 1) * stride + (packed ? 7 : 6) * Np) * size);
}

}  // namespace lpg
