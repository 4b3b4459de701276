// rast_pairs.cuh -- (rectangle, tile) pairs of a warp, numbered in lane order
// and taken 32 a round.  Plain C++ as well: its arithmetic is tested on the
// host.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define RAST_PAIRS_FN __host__ __device__ __forceinline__
#else
#define RAST_PAIRS_FN inline
#endif

namespace rast {

// The bit of the round [base, base + 32) at which a lane's pairs begin: the
// lane has n pairs, `before` pairs lie in the lanes below it.  Zero where they
// begin in another round or the lane has none.  All unsigned: 32 rectangles of
// 2^26 tiles (a canvas of 2^31 pixels) are 2^31 pairs.
RAST_PAIRS_FN uint32_t pair_begin_bit(uint32_t before, uint32_t n, uint32_t base) {
  const uint32_t at = before - base;
  return n > 0u && at < 32u ? 1u << at : 0u;
}

}  // namespace rast
