// Arrival count of a grid barrier.
#pragma once

#ifdef __CUDACC__
#define SPOC_BOTH __host__ __device__
#else
#define SPOC_BOTH
#endif

namespace spoc {

// Whether every block has arrived: `count` and `target` are counted modulo 2^32
// and never further apart than a grid's blocks, so the sign of their difference
// tells, also where the count wraps (148 blocks and eight barriers a step: every
// 3.6 million steps of one call).
SPOC_BOTH inline bool barrier_reached(unsigned count, unsigned target) {
  return (int)(count - target) >= 0;
}

}  // namespace spoc
