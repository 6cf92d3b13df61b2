// coop.cuh -- the grid barrier and the bounded waits of the one-launch kernels
// (bfs_coop.cu, sssp_coop.cu, multigraph.cu, pagerank.cu).
#pragma once
#include "barrier_word.h"
#include "engine.cuh"

namespace mb {

// Grid barrier of a cooperative launch: bar[0] counts arrivals over the run
// (both words zero before it); barrier k, the first is 1, is passed when they
// reach k times the grid (barrier_word.h).  The wait is bounded: past `polls`
// polls the CTA says in bar[1] that it gave up, which the others see while they
// wait.  Whatever way a wait ends other than by passing, the CTA records
// ERR_BARRIER in *err (host memory) and returns
// false; the caller leaves.  The acquire drops this SM's
// stale L1 lines.  *bar wants a 128-byte line of its own: the waiting CTAs
// poll it, and atomics on counters beside it queue up behind them (SSSP on
// R-MAT 2^20 / 2^24: 1.27 -> 0.97 ms).
__device__ __forceinline__ bool coop_barrier(uint32_t *bar, uint32_t k, long polls, int32_t *err) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t target = bar_target(k, gridDim.x);
        __threadfence();
        atomicAdd(bar, 1u);
        int ok = 0;
        for (long it = 0;; it++) {
            if (bar_passed(ld_acquire_gpu(bar), target)) {
                ok = 1;
                break;
            }
            if (it >= polls) {
                atomicOr(bar + 1, 1u);
                break;
            }
            if ((it & 63) == 63 && ld_acquire_gpu(bar + 1)) break;
        }
        if (!ok) *(volatile int32_t *)err = ERR_BARRIER;
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok;
}

// Room for what a CTA appends in a round: every thread gives the number of its
// vertices and of their out-edges, and gets the packed position (count << 32
// | edges) of its first; one atomic on *ctr per round.  At most 32 warps.
struct CoopRound {
    unsigned long long tot[32];
};
__device__ __forceinline__ unsigned long long coop_round_append(CoopRound &r, uint32_t cnt, uint32_t sum,
                                                                unsigned long long *ctr) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t isum = warp_incl_scan_u32(sum), icnt = warp_incl_scan_u32(cnt);
    if (lane == 31) r.tot[wid] = ((unsigned long long)icnt << 32) | isum;
    __syncthreads();
    if (wid == 0) {
        const unsigned long long t = lane < nw ? r.tot[lane] : 0ull;
        const uint32_t tc = (uint32_t)(t >> 32), ts = (uint32_t)t;
        const uint32_t ic = warp_incl_scan_u32(tc), is = warp_incl_scan_u32(ts);
        unsigned long long base = 0;
        if (lane == 31 && ic) base = atomicAdd(ctr, ((unsigned long long)ic << 32) | is);
        base = __shfl_sync(0xffffffffu, base, 31);
        if (lane < nw) r.tot[lane] = base + (((unsigned long long)(ic - tc) << 32) | (is - ts));
    }
    __syncthreads();
    return r.tot[wid] + (((unsigned long long)(icnt - cnt) << 32) | (isum - sum));
}

}  // namespace mb
