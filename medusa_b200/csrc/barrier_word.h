// barrier_word.h -- the word of the one-launch kernels' grid barriers.
//
// The word counts arrivals over a whole run, and its top bit says that a wait
// gave up.  It has 64 bits because a run has no bound of its own on its
// supersteps: 592 CTAs pass 2^31 arrivals after 3.6 million of them, which a
// BFS along a chain of vertices reaches, and a count that ran into the top bit
// would end every wait without anyone having given up.
// No CUDA in here, so that a host program can run the same decisions.
#pragma once

#ifdef __CUDACC__
#define MB_BAR_FN __host__ __device__ __forceinline__
#else
#define MB_BAR_FN inline
#endif

namespace mb {

typedef unsigned long long BarWord;
constexpr BarWord kBarGivenUp = 1ull << 63;
enum BarWait { BAR_WAIT, BAR_PASSED, BAR_GIVEN_UP };

// What a wait for `target` arrivals does after reading v.
MB_BAR_FN BarWait bar_poll(BarWord v, BarWord target) {
    return v >= kBarGivenUp ? BAR_GIVEN_UP : v >= target ? BAR_PASSED : BAR_WAIT;
}

}  // namespace mb
