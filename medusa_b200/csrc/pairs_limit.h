// pairs_limit.h -- how many sources one run of the one-launch SSSP takes.
// No CUDA in here, so that a host program can check the bounds.
#pragma once
#include <algorithm>
#include <cstdint>

namespace mb {

constexpr int32_t kSsspCoopSources = 32;  // at most, in one run
// Several sources: (source, vertex) pairs of a run, 128 MB of distances.
// 32 sources at 2^23 / 2^24 / 2^25 pairs: mild R-MAT 2^20 / 2^24 15.7 / 14.1 / 13.2 ms,
// 2^22 / 2^26 59.0 / 55.6 / 54.0.
constexpr int64_t kPairs = 1 << 25;

// Sources of a run on a graph of V vertices and E edges: at most kPairs pairs,
// and at most 2^31 - 1 out-edges of all pairs together.  A superstep's queue
// can hold every pair, and its edges are numbered in 32 bits: numbers past
// 2^31 leave the signed sums that address them, and numbers within a tile of
// 2^32 the rounding up to whole tiles.
inline int32_t pairs_sources(int32_t V, int64_t E) {
    int64_t n = std::min<int64_t>(kSsspCoopSources, kPairs / std::max<int32_t>(V, 1));
    n = std::min<int64_t>(n, INT32_MAX / std::max<int64_t>(E, 1));
    return (int32_t)std::max<int64_t>(n, 1);
}

}  // namespace mb
