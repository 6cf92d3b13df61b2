// barrier_word.h -- the counting of the one-launch kernels' grid barriers.
//
// One word counts the arrivals of a whole run, another says that a wait gave
// up.  A run has no bound of its own on its supersteps (592 CTAs pass 2^31
// arrivals after 3.6 million of them, which a BFS along a chain of vertices
// reaches), so the count wraps around, and a wait looks at its distance to the
// target: arrivals are never further than a grid's CTAs from it.  (64-bit
// arrivals cost 0.15 us more per barrier.)
// No CUDA in here, so that a host program can run the same decisions.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define MB_BAR_FN __host__ __device__ __forceinline__
#else
#define MB_BAR_FN inline
#endif

namespace mb {

// Arrivals at which barrier k of a run is passed; the first is 1.
MB_BAR_FN uint32_t bar_target(uint32_t k, uint32_t grid) { return k * grid; }
MB_BAR_FN bool bar_passed(uint32_t arrivals, uint32_t target) { return (int32_t)(arrivals - target) >= 0; }

}  // namespace mb
