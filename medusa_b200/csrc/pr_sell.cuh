// pr_sell.cuh -- PageRank's sliced ELL, shared by pagerank.cu and the
// many-graph kernel (multigraph.cu).
#pragma once
#include "pr_order.cuh"

namespace mb {

// New rank and contribution of a vertex at position p (-1: no out-edges) with
// out-degree d; MPG/CPUFunctorHoster.cpp:80-82.
template <class Args>
__device__ __forceinline__ void pr_write(const Args &a, int32_t v, float sum, int32_t p, int32_t d) {
    const float r = pr_update(sum);
    if (a.rank_out) a.rank_out[v] = r;
    if (p >= 0) a.contrib_out[p] = r / (float)d;
}

template <class Args>
__device__ __forceinline__ void pr_write(const Args &a, int32_t v, float sum) {
    pr_write(a, v, sum, a.pos[v], a.outdeg[v]);
}

// Streamed index arrays (read once per superstep) bypass L1, which is left
// to the contribution gathers: a hot source's contribution then stays in L1
// for the next warps that gather it (4% at 2^28 edges; an evict_last hint on
// the gathers measured 5% slower).
__device__ __forceinline__ int32_t ld_stream(const int32_t *p) {
    int32_t v;
    asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// The contribution at position i; kNc: nobody writes the array during the
// launch (else plain loads, and a barrier's acquire between two supersteps).
template <bool kNc>
__device__ __forceinline__ float ld_contrib(const float *c, int32_t i) {
    return kNc ? __ldg(c + i) : c[i];
}

// ---- sliced ELL ------------------------------------------------------------------
// Vertices sorted by in-degree (largest first), 32 per group: a group's rows
// are its first vertex's in-degree, so a group pads by at most 31 slots per row
// of the difference to its last vertex: over the groups of a sorted list these
// differences add up to the largest in-degree (31 times that many slots in all,
// beside the empty lanes of the last group).
// Light vertices in both orders, and mid vertices (up to hub_min in-edges) in
// the reference's order.
struct SellArgs {
    const int32_t *v;       // 32 per group (-1: padding)
    const int2 *pd;         // their contribution positions and out-degrees
    const int32_t *rows;    // rows of each group
    const uint32_t *base;   // rows before it
    const int32_t *src;     // position of group g, row j, lane l's source at 32 (base[g] + j) + l (-1: padding)
    int32_t ngroups, nlong; // groups [0, nlong) have more than kSellShort rows
    const float *contrib_in;
    float *contrib_out, *rank_out;
    // vertices without in-edges: their sum is 0 in every superstep, so their
    // contributions are written once to each of the two buffers (zfirst), their
    // ranks with the others'
    const int32_t *zv;
    const int2 *zpd;
    int32_t nz;
    int32_t zfirst;
};

__device__ __forceinline__ void zero_vertices(const SellArgs &a) {
    if (!a.zfirst && !a.rank_out) return;
    const float r = pr_update(0.f);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.nz; i += (int64_t)gridDim.x * blockDim.x) {
        const int2 p = a.zpd[i];
        if (a.zfirst && p.x >= 0) a.contrib_out[p.x] = r / (float)p.y;
        if (a.rank_out) a.rank_out[a.zv[i]] = r;
    }
}
constexpr int kSellShort = 8;
// 16 rows in flight and at least 5 CTAs of 256 threads per SM (8 rows and 8 CTAs:
// R-MAT 2^24 / 2^28 0.955 against 1.011 ms a superstep, uniform 9 10^5 / 3.6 10^6 21
// against 27 us).
constexpr int kSellU = 16, kSellCtas = 5;

// One group: kSellU rows (coalesced index loads, then the gathers) in
// flight; each lane folds its own vertex's slots in order.  Padding slots
// (-1) read 0, and s + 0 = s, so they change no bit.
template <int kSellU, bool kNc = true>
__device__ __forceinline__ void sell_long(const SellArgs &a, int64_t g) {
    const int lane = threadIdx.x & 31;
    const int32_t rows = __ldg(&a.rows[g]);
    const int2 pd = __ldg(&a.pd[g * 32 + lane]);
    const int32_t *src = a.src + (int64_t)__ldg(&a.base[g]) * 32 + lane;
    float sum = 0.f;
    // the next rows' indices load while this block's gathers are in flight
    int32_t nxt[kSellU];
#pragma unroll
    for (int u = 0; u < kSellU; u++) nxt[u] = u < rows ? ld_stream(src + (int64_t)u * 32) : -1;
    for (int32_t j0 = 0; j0 < rows; j0 += kSellU) {
        int32_t idx[kSellU];
#pragma unroll
        for (int u = 0; u < kSellU; u++) idx[u] = nxt[u];
#pragma unroll
        for (int u = 0; u < kSellU; u++) {
            const int32_t j = j0 + kSellU + u;
            nxt[u] = j < rows ? ld_stream(src + (int64_t)j * 32) : -1;
        }
        float x[kSellU];
#pragma unroll
        for (int u = 0; u < kSellU; u++) x[u] = idx[u] >= 0 ? ld_contrib<kNc>(a.contrib_in, idx[u]) : 0.f;
#pragma unroll
        for (int u = 0; u < kSellU; u++) sum += x[u];
    }
    const int32_t v = a.rank_out ? a.v[g * 32 + lane] : 0;
    if (v >= 0) pr_write(a, v, sum, pd.x, pd.y);
}

// kG consecutive groups of at most kSellShort rows at once: a group alone
// would leave a lane with a handful of gathers in flight.
template <int kG, bool kNc = true>
__device__ __forceinline__ void sell_short(const SellArgs &a, int64_t g0) {
    constexpr int kR = 16 / kG;
    const int lane = threadIdx.x & 31;
    int32_t rows[kG];
    int2 pd[kG];
    const int32_t *src[kG];
    float sum[kG];
#pragma unroll
    for (int i = 0; i < kG; i++) {
        const bool in = g0 + i < a.ngroups;
        rows[i] = in ? __ldg(&a.rows[g0 + i]) : 0;
        pd[i] = in ? __ldg(&a.pd[(g0 + i) * 32 + lane]) : make_int2(-1, 0);
        src[i] = a.src + (in ? (int64_t)__ldg(&a.base[g0 + i]) * 32 + lane : 0);
        sum[i] = 0.f;
    }
    const int32_t rmax = rows[0];
    for (int32_t j0 = 0; j0 < rmax; j0 += kR) {
        int32_t idx[kG][kR];
        float x[kG][kR];
#pragma unroll
        for (int i = 0; i < kG; i++)
#pragma unroll
            for (int u = 0; u < kR; u++)
                idx[i][u] = j0 + u < rows[i] ? ld_stream(src[i] + (int64_t)(j0 + u) * 32) : -1;
#pragma unroll
        for (int i = 0; i < kG; i++)
#pragma unroll
            for (int u = 0; u < kR; u++) x[i][u] = idx[i][u] >= 0 ? ld_contrib<kNc>(a.contrib_in, idx[i][u]) : 0.f;
#pragma unroll
        for (int i = 0; i < kG; i++)
#pragma unroll
            for (int u = 0; u < kR; u++) sum[i] += x[i][u];
    }
#pragma unroll
    for (int i = 0; i < kG; i++) {
        if (g0 + i >= a.ngroups) break;
        const int32_t v = a.rank_out ? a.v[(g0 + i) * 32 + lane] : 0;
        if (v >= 0) pr_write(a, v, sum[i], pd[i].x, pd[i].y);
    }
}

}  // namespace mb
