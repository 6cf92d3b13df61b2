// pagerank.cu -- the PageRank app's BSP superstep on sm_100a.
//
// Reference (MPG/UserOperators.h:16-43,119-144,175-270; combiner with
// CUDPP_ADD; CPU form MPG/CPUFunctorHoster.cpp:17-31,60-93,143-163):
//   send    msg = rank[u] / outdeg[u] (float) on every out-edge of u
//   combine sum of the messages of each destination
//   update  rank[v] = 0.15 + 0.85 * sum, with the reference's rounding:
//           sum *= 0.85 is a double multiply rounded to float, and
//           0.15 + sum a double add rounded to float.
// No dangling-rank redistribution; a vertex with no in-edges gets 0.15.
//
// The sum runs in the fixed order of pr_order.cuh, the same for every
// schedule, so schedules never change a bit of the result.  Work mapping:
//   light vertices (in-degree <= kPrLight): a sliced ELL (PrSell, k_pr_sell),
//     vertices sorted by in-degree, 32 per group, row j holding slot j of
//     each, so a warp reads a row of in-edge sources with one coalesced load
//     and lane l folds its own vertex (the message-reading schedule uses
//     k_pr_pull over the full reverse CSR);
//   heavier vertices: their kPrBlock-edge blocks form a work list built once
//     per graph, one 16-byte item per block (edge range, vertex, slot); one
//     warp per long item, or 1, 2 or 4 short items per warp
//     (k_heavy_blocks).  A vertex with a single block is
//     finished there (update and next contribution); a hub's blocks write
//     block sums that k_hub_finalize folds in order -- so hubs and the long
//     tail of R-MAT's hundreds-to-thousands in-degrees spread over every SM
//     instead of serialising in one lane.
// Schedules: 0 fused pull (gather rank/outdeg, fold, update, write the next
// contribution); 6 the reference's split: send into the E-slot message
// array at msgDstID, then the same combine+update reading the messages.
#include <algorithm>
#include <vector>
#include "coop.cuh"
#include "pagerank.cuh"
#include "pr_order.cuh"
#include "pr_sell.cuh"

namespace mb {
namespace {

constexpr int kWin = 512;                // edges staged per warp per window
constexpr int kPrWarps = 8;              // warps per CTA
constexpr int kPrThreads = kPrWarps * 32;
struct PrArgs {
    int32_t V;
    int64_t E;
    const int32_t *rrow, *outdeg, *row, *mslot;  // mslot: of the order in use
    // contributions by position (k_pos): rank[u]/outdeg[u] of the previous
    // superstep at pos[u]
    const int32_t *pos;
    const float *contrib_in;
    float *contrib_out;
    float *rank_out;           // null but in the last superstep: no other reads the ranks
    float *msg;                // E-slot message array (schedule 6)
    const int4 *items;           // heavy blocks: {j0, j1, vertex, hub slot or -1}
    int32_t nitems;
    const int32_t *hub_v;        // vertices with more than one block
    const int32_t *hub_first;    // first slot of each hub (nhub+1 entries)
    int32_t nhub;
    float *blk_sum;              // per-slot block sums of the hubs
    int32_t nlong;               // items [0, nlong) are longer than kPrShortItem
    const int32_t *hcol;         // positions of the in-edge sources, reverse-CSR order
};

// The gathers of contributions are what bounds a superstep: a random 4-byte
// load is one L1 lookup, and where it misses one request and 32-byte sector
// from L2 (measured on tables of 4 to 64 MB: 285 G loads/s, one per clock
// and SM; 800 from L1).  Holding the hottest 32K contributions in shared
// memory (1300 G loads/s) instead made these kernels slower: one CTA of 1024
// threads per SM keeps too few gathers in flight (R-MAT 2^24 / 2^28: 1.13
// against 1.09 ms a superstep; 2^20.3 / 17M: 0.081 against 0.074).
__device__ __forceinline__ float ld_gather(const float *c, int32_t i) { return __ldg(c + i); }

template <bool kFromMsg>
__device__ __forceinline__ float edge_val(const PrArgs &a, int64_t j) {
    if (kFromMsg) return a.msg[j];
    return ld_gather(a.contrib_in, ld_stream(&a.hcol[j]));
}

// Heavy-vertex blocks (<= kPrBlock in-edges each), summed exactly as
// pr_warp_block_sum does: lane l folds edges l, l+32, ... from 0, then the
// xor butterfly.  The list is sorted longest first.  Its head (items longer
// than kPrShortItem) takes one item per warp with kLongU loads of each lane
// in flight; the rest take kShortPair items per warp at once (kShortU loads
// of each item in flight), so short items do not leave a warp waiting on a
// handful of loads.  Neither grouping changes a bit.  A single-block vertex
// is finished here; a hub block writes its block sum.
#ifndef MB_PR_LONG_UNROLL
#define MB_PR_LONG_UNROLL 16
#endif
constexpr int kLongU = MB_PR_LONG_UNROLL;
constexpr int kShortU = 4;
constexpr int kPrShortItem = 32 * kShortU * 4;  // 512 edges
constexpr int kShortPairDefault = 2;  // measured best at 2^20-2^28 edges

__host__ __device__ __forceinline__ int64_t heavy_units(int32_t nitems, int32_t nlong, int pair) {
    return (int64_t)nlong + ((int64_t)nitems - nlong + pair - 1) / pair;
}

__device__ __forceinline__ void heavy_finish(const PrArgs &a, const int4 &it, float acc, int32_t d) {
    if (it.w == -2) return;  // past the list
    if (it.w < 0) pr_write(a, it.z, 0.f + acc, __ldg(&a.pos[it.z]), d);  // one block sum folded from 0
    else a.blk_sum[it.w] = acc;
}

template <bool kFromMsg, int kShortPair>
__global__ void __launch_bounds__(256) k_heavy_blocks(PrArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t units = heavy_units(a.nitems, a.nlong, kShortPair);
    for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < units; u += warps) {
        if (u < a.nlong) {
            const int4 it = __ldg(&a.items[u]);
            const int32_t d = (lane == 0 && it.w < 0) ? __ldg(&a.outdeg[it.z]) : 0;
            const int32_t len = it.y - it.x;
            float acc = 0.f;
            for (int32_t k0 = 0; k0 < len; k0 += 32 * kLongU) {
                float val[kLongU];
#pragma unroll
                for (int q = 0; q < kLongU; q++) {
                    const int32_t k = k0 + lane + 32 * q;
                    val[q] = k < len ? edge_val<kFromMsg>(a, (int64_t)it.x + k) : 0.f;
                }
#pragma unroll
                for (int q = 0; q < kLongU; q++)
                    if (k0 + lane + 32 * q < len) acc += val[q];
            }
#pragma unroll
            for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
            if (lane == 0) heavy_finish(a, it, acc, d);
            continue;
        }
        const int64_t b0 = a.nlong + (u - a.nlong) * kShortPair;
        int4 it[kShortPair];
        int32_t len[kShortPair], d[kShortPair], lmax = 0;
        float acc[kShortPair];
#pragma unroll
        for (int p = 0; p < kShortPair; p++) {
            it[p] = b0 + p < a.nitems ? __ldg(&a.items[b0 + p]) : make_int4(0, 0, 0, -2);
            len[p] = it[p].y - it[p].x;
            lmax = max(lmax, len[p]);
            acc[p] = 0.f;
        }
#pragma unroll
        for (int p = 0; p < kShortPair; p++)
            d[p] = (lane == 0 && it[p].w == -1) ? __ldg(&a.outdeg[it[p].z]) : 0;
        for (int32_t k0 = 0; k0 < lmax; k0 += 32 * kShortU) {
            float val[kShortPair][kShortU];
#pragma unroll
            for (int p = 0; p < kShortPair; p++)
#pragma unroll
                for (int q = 0; q < kShortU; q++) {
                    const int32_t k = k0 + lane + 32 * q;
                    val[p][q] = k < len[p] ? edge_val<kFromMsg>(a, (int64_t)it[p].x + k) : 0.f;
                }
#pragma unroll
            for (int p = 0; p < kShortPair; p++)
#pragma unroll
                for (int q = 0; q < kShortU; q++)
                    if (k0 + lane + 32 * q < len[p]) acc[p] += val[p][q];
        }
#pragma unroll
        for (int p = 0; p < kShortPair; p++) {
#pragma unroll
            for (int off = 16; off; off >>= 1) acc[p] += __shfl_xor_sync(0xffffffffu, acc[p], off);
        }
        if (lane == 0) {
#pragma unroll
            for (int p = 0; p < kShortPair; p++) heavy_finish(a, it[p], acc[p], d[p]);
        }
    }
}

// Hubs (more than one block): fold the block sums in order, then update.
__global__ void k_hub_finalize(PrArgs a) {
    for (int32_t h = blockIdx.x * blockDim.x + threadIdx.x; h < a.nhub; h += gridDim.x * blockDim.x) {
        float sum = 0.f;
        for (int32_t k = a.hub_first[h]; k < a.hub_first[h + 1]; k++) sum += a.blk_sum[k];
        pr_write(a, a.hub_v[h], sum);
    }
}

// Combine+update over the full reverse CSR (the message-reading schedule and
// the reference's MEG order): one warp per 32 consecutive vertices.  The warp
// streams the group's in-edges (contiguous in reverse-CSR order) through a
// shared-memory window, coalesced; each lane then folds its own vertex's
// part of the window in order.  kAllLight (the reference's MEG order): every
// vertex, hubs included, is folded sequentially by its lane.
template <bool kFromMsg, bool kAllLight = false>
__global__ void __launch_bounds__(kPrThreads) k_pr_pull(PrArgs a) {
    __shared__ float win[kPrWarps][kWin];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float *wv = win[wid];
    const int64_t ngroups = ((int64_t)a.V + 31) / 32;
    const int64_t warps = (int64_t)gridDim.x * kPrWarps;
    for (int64_t grp = (int64_t)blockIdx.x * kPrWarps + wid; grp < ngroups; grp += warps) {
        const int32_t v = (int32_t)(grp * 32 + lane);
        const bool valid = v < a.V;
        const int32_t vb = (int32_t)(grp * 32);
        const int32_t ve = (int32_t)min(grp * 32 + 32, (int64_t)a.V);
        int64_t b = 0, e = 0;
        if (valid) {
            b = a.rrow[v];
            e = a.rrow[v + 1];
        }
        const bool heavy = !kAllLight && valid && (e - b) > kPrLight;
        const int64_t g0 = a.rrow[vb], g1 = a.rrow[ve];
        float sum = 0.f;
        // heavy vertices are finished by k_heavy_blocks / k_hub_finalize
        for (int64_t w0 = g0; w0 < g1; w0 += kWin) {
            const int64_t w1 = min(w0 + (int64_t)kWin, g1);
            // skip windows that lie entirely inside heavy ranges
            const bool mine = !heavy && b < w1 && e > w0;
            if (!__any_sync(0xffffffffu, mine)) continue;
            // every load of the window in flight at once
            float vals[kWin / 32];
#pragma unroll
            for (int r = 0; r < kWin / 32; r++) {
                const int64_t j = w0 + lane + 32 * r;
                vals[r] = j < w1 ? edge_val<kFromMsg>(a, j) : 0.f;
            }
#pragma unroll
            for (int r = 0; r < kWin / 32; r++) wv[lane + 32 * r] = vals[r];
            __syncwarp();
            if (mine) {
                const int64_t lo = max(b, w0), hi = min(e, w1);
                for (int64_t j = lo; j < hi; j++) sum += wv[j - w0];
            }
            __syncwarp();
        }
        if (valid && !heavy) pr_write(a, v, sum);
    }
}

// One unit per warp, longest groups first, and as many CTAs as that takes: the
// hardware hands them to the SMs as these get free, beside the hub scans too.
// (A resident grid whose warps took their next unit from a counter, one atomic
// a unit on the same address, us per superstep: R-MAT 2^24 / 2^28 957, now
// 943; 4 10^6 / 6 10^7 250 in the fixed order, now 232; uniform 9 10^5 / 1.4 10^7 67,
// now 57; 9 10^5 / 3.6 10^6 28, now 18.)
template <int kG>
__global__ void __launch_bounds__(256, kSellCtas) k_pr_sell(SellArgs a) {
    const uint32_t units = (uint32_t)a.nlong + (uint32_t)(a.ngroups - a.nlong + kG - 1) / kG;
    const uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    zero_vertices(a);
    if (u >= units) return;
    if (u < (uint32_t)a.nlong) sell_long<kSellU>(a, u);
    else sell_short<kG>(a, a.nlong + (int64_t)(u - a.nlong) * kG);
}

// All supersteps in one cooperative launch, for graphs whose groups fit one
// to a resident warp and that have no other vertices: the group's head and
// the first rows' indices are loaded before the barrier between two
// supersteps, and no superstep waits for a launch.  Contributions are read
// with plain loads (other SMs write them during the launch; the barrier's
// acquire drops stale L1 lines).  A barrier that gives up writes *err (host
// memory) and ends the launch.  Uniform 2^18 / 2^22, ten supersteps: 17.9 us
// each, against 22.8 in launches of their own (the gathers alone: 14).
// 8 rows in flight at 32 registers (64 warps per SM), or 16 where half the
// warps are enough: the fewer rounds, the shorter a small graph's superstep.
constexpr int kResThreads = 1024;
struct ResidentArgs {
    float *contrib[2], *rank;
    const int32_t *zv;  // vertices without in-edges
    const int2 *zpd;
    int32_t nz, iters;
    uint32_t *bar;      // the barrier's two words (coop.cuh), and 128 bytes further the CTAs
                        // done; zero before the launch, which leaves them so
    int32_t *err;
    long polls;
};
template <int kResU>
__global__ void __launch_bounds__(kResThreads, kResU == 8 ? 2 : 1) k_pr_resident(SellArgs a, ResidentArgs r) {
    const int lane = threadIdx.x & 31;
    // the longest groups spread over the CTAs
    const int32_t g = (int32_t)((threadIdx.x >> 5) * gridDim.x + blockIdx.x);
    const bool in = g < a.ngroups;
    const int32_t rows = in ? __ldg(&a.rows[g]) : 0;
    const int2 pd = in ? __ldg(&a.pd[(int64_t)g * 32 + lane]) : make_int2(-1, 0);
    const int32_t *src = a.src + (in ? (int64_t)__ldg(&a.base[g]) * 32 + lane : 0);
    for (int it = 0; it < r.iters; it++) {
        int32_t idx[kResU];
#pragma unroll
        for (int u = 0; u < kResU; u++) idx[u] = u < rows ? __ldg(src + u * 32) : -1;
        if (it > 0 && !coop_barrier(r.bar, (uint32_t)it, r.polls, r.err)) return;
        const float *cin = it & 1 ? r.contrib[1] : r.contrib[0];
        float *cout = it & 1 ? r.contrib[0] : r.contrib[1];
        float *rank = it == r.iters - 1 ? r.rank : nullptr;
        float sum = 0.f;
        for (int32_t j0 = 0; j0 < rows; j0 += kResU) {
            float x[kResU];
#pragma unroll
            for (int u = 0; u < kResU; u++) x[u] = idx[u] >= 0 ? cin[idx[u]] : 0.f;
#pragma unroll
            for (int u = 0; u < kResU; u++) {
                const int32_t j = j0 + kResU + u;
                idx[u] = j < rows ? __ldg(src + j * 32) : -1;
            }
#pragma unroll
            for (int u = 0; u < kResU; u++) sum += x[u];
        }
        if (rows) {
            const float nr = pr_update(sum);
            if (pd.x >= 0) cout[pd.x] = nr / (float)pd.y;
            if (rank) {
                const int32_t v = a.v[(int64_t)g * 32 + lane];
                if (v >= 0) rank[v] = nr;
            }
        }
        if (it < 2 || rank) {
            const float zr = pr_update(0.f);
            for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < r.nz; i += gridDim.x * blockDim.x) {
                const int2 p = r.zpd[i];
                if (it < 2 && p.x >= 0) cout[p.x] = zr / (float)p.y;
                if (rank) rank[r.zv[i]] = zr;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&r.bar[32], 1u) == gridDim.x - 1) {  // no CTA waits any more
        r.bar[0] = 0u;
        r.bar[32] = 0u;
    }
}

__global__ void k_pr_zero(SellArgs a) { zero_vertices(a); }  // a graph without any in-edge list

// ---- the reference's order (MB_PR_ORDER_REFERENCE), in parallel -------------
// Every vertex's sum is the reference's sequential float fold over its MEG
// slots, bit for bit (pr_order.cuh).  Two mappings by in-degree n:
//   n <= hub_min: the sliced ELL above, filled in MEG slot order;
//   n > hub_min: the contributions staged by every SM into one contiguous run
//     per vertex (k_pr_hub_stage), then one warp or CTA per vertex runs the
//     parallel integer scan of pr_order.cuh over it (k_pr_hub_warp,
//     k_pr_hub_exact), on side streams beside the sliced ELL.
constexpr int kHubK = 16;                       // consecutive slots per thread
constexpr int kHubBig = 16384;                  // in-degree above which a hub gets the big CTA
// In-degree above which a vertex is a hub by default: E / 2^14 within these.  A
// sliced-ELL group is a chain of gathers as long as its rows (2048 rows: some
// 150 us), which has to stay short against the superstep; a scan costs more
// per slot.  us per superstep at 512 / 1024 / 2048: skewed R-MAT 10^5 / 2^20 61 /
// 61 / 89, 0.6M / 11M 138 / 124 / 177, 2^21 / 2^25 220 / 212 / 186, 2^23 / 2^27 702 /
// 500 / 500.
constexpr int kHubMinLeast = 512, kHubMinMost = 2048;

struct ExactArgs {
    const int32_t *rrow, *outdeg;
    const int32_t *pos;          // contribution positions, as in PrArgs
    const float *contrib_in;
    float *contrib_out, *rank_out;
    const int32_t *hub_v;        // hubs, largest in-degree first
    int32_t nhub;
    float *x_stage;              // every hub's contributions, in MEG slot order
    const int64_t *stage_off;    // where hub h's run starts (16-byte aligned)
    const int32_t *stage_src;    // positions of their sources, at the same offsets
    const int2 *stage_items;     // staging work: {offset, length}
    int32_t nstage_items;
};

// Staging: every hub's contributions gathered, in MEG slot order, into one
// contiguous run per hub (x_stage), by all SMs at once: one warp per item of
// at most kStageItem slots, kStageU loads of each lane in flight.  The
// scans below then read coalesced data instead of each hub's CTA gathering
// at one SM's rate.
#ifndef MB_STAGE_ITEM
#define MB_STAGE_ITEM 1024
#endif
constexpr int kStageItem = MB_STAGE_ITEM;
constexpr int kStageU = 8;
__device__ __forceinline__ void stage_item(const ExactArgs &a, int64_t it) {
    const int lane = threadIdx.x & 31;
    const int2 item = __ldg(&a.stage_items[it]);
    float *dst = a.x_stage + (uint32_t)item.x;
    const int32_t *src = a.stage_src + (uint32_t)item.x;
    // the next indices load while these gathers are in flight
    int32_t nxt[kStageU];
#pragma unroll
    for (int u = 0; u < kStageU; u++) nxt[u] = 32 * u + lane < item.y ? ld_stream(src + 32 * u + lane) : -1;
    for (int32_t k0 = 0; k0 < item.y; k0 += 32 * kStageU) {
        int32_t idx[kStageU];
#pragma unroll
        for (int u = 0; u < kStageU; u++) idx[u] = nxt[u];
#pragma unroll
        for (int u = 0; u < kStageU; u++) {
            const int32_t k = k0 + 32 * (kStageU + u) + lane;
            nxt[u] = k < item.y ? ld_stream(src + k) : -1;
        }
        float x[kStageU];
#pragma unroll
        for (int u = 0; u < kStageU; u++) x[u] = idx[u] >= 0 ? ld_gather(a.contrib_in, idx[u]) : 0.f;
#pragma unroll
        for (int u = 0; u < kStageU; u++) {
            const int32_t k = k0 + 32 * u + lane;
            if (k < item.y) dst[k] = x[u];
        }
    }
}

__global__ void __launch_bounds__(256) k_pr_hub_stage(ExactArgs a) {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t it = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < a.nstage_items; it += warps)
        stage_item(a, it);
}

// Scan thread t's kHubK consecutive staged values of the chunk at `pos`
// (0 past the vertex's end).  run + pos is 16-byte aligned.
__device__ __forceinline__ void hub_load(const float *run, int32_t n, int32_t pos, int t, float (&x)[kHubK]) {
    const int32_t j0 = pos + t * kHubK;
    if (j0 + kHubK <= n) {
        const float4 *p4 = reinterpret_cast<const float4 *>(run + j0);
#pragma unroll
        for (int r = 0; r < kHubK / 4; r++) {
            const float4 t4 = __ldcs(p4 + r);
            x[4 * r] = t4.x;
            x[4 * r + 1] = t4.y;
            x[4 * r + 2] = t4.z;
            x[4 * r + 3] = t4.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kHubK; k++) x[k] = j0 + k < n ? __ldcs(run + j0 + k) : 0.f;
    }
}

// Hubs [h0, h1) of the list: one CTA of kT threads per vertex, over its
// staged run.  The first kHead values are folded by thread 0 (a multiple of
// 4, so the chunks that follow start 16-byte aligned); then chunks of
// kT * kHubK values, thread t owning kHubK consecutive ones, go through the
// integer scan of pr_order.cuh.  Each chunk's loads are issued one chunk
// ahead of its scan.
template <int kT, int kHead>
__global__ void __launch_bounds__(kT) k_pr_hub_exact(ExactArgs a, int32_t h0, int32_t h1) {
    static_assert(kHead % 4 == 0, "chunks start 16-byte aligned");
    constexpr int kW = kT / 32;
    constexpr int kChunk = kT * kHubK;
    __shared__ __align__(16) float head[kHead];
    __shared__ uint32_t wtot[kW];
    __shared__ int32_t wbad[kW];
    __shared__ float s_sh;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int32_t h = h0 + blockIdx.x; h < h1; h += gridDim.x) {
        const int32_t v = __ldg(&a.hub_v[h]);
        const int32_t n = __ldg(&a.rrow[v + 1]) - __ldg(&a.rrow[v]);
        const float *run = a.x_stage + __ldg(&a.stage_off[h]);
        const int32_t H = min(n, kHead);
        for (int i = tid; i < H; i += kT) head[i] = __ldcs(run + i);
        float x[kHubK], xn[kHubK];
        hub_load(run, n, H, tid, xn);  // the first chunk's loads go out before the head is folded
        __syncthreads();
        if (tid == 0) {  // the adds chain; the shared loads run ahead, 4 at a time
            float s0 = 0.f;
            const float4 *h4 = reinterpret_cast<const float4 *>(head);
            int i = 0;
#pragma unroll 8
            for (; i + 4 <= H; i += 4) {
                const float4 t = h4[i >> 2];
                s0 += t.x;
                s0 += t.y;
                s0 += t.z;
                s0 += t.w;
            }
            for (; i < H; i++) s0 += head[i];
            s_sh = s0;
        }
        __syncthreads();
        float s = s_sh;
        for (int32_t pos = H; pos < n; pos += kChunk) {
#pragma unroll
            for (int k = 0; k < kHubK; k++) x[k] = xn[k];
            if (pos + kChunk < n) hub_load(run, n, pos + kChunk, tid, xn);
            int start = 0;  // threads before it have folded their slots
            for (;;) {
                const uint32_t bits = __float_as_uint(s);
                const uint32_t ks = bits >> 23, base = (bits & 0x7fffffu) | 0x800000u;
                uint32_t L = 0;
                bool tie = false;
                if (tid >= start) {
#pragma unroll
                    for (int k = 0; k < kHubK; k++) L += pr_units(x[k], ks, tie);
                    L = min(L, 1u << 23);
                }
                // inclusive prefix over the CTA.  Up to the first bad thread it
                // stays below 2^24 + 2^23; past it a sum may wrap around 2^32,
                // which changes nothing: only the first bad thread is used
                uint32_t I = L;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, I, off);
                    if (lane >= off) I += y;
                }
                if (lane == 31) wtot[wid] = I;
                __syncthreads();
                uint32_t total = 0;
#pragma unroll
                for (int w = 0; w < kW; w++) {
                    const uint32_t t = wtot[w];
                    if (w < wid) I += t;
                    total += t;
                }
                const bool bad = tid >= start && (ks == 0 || ks == 255 || tie || base + I >= (1u << 24));
                const unsigned bm = __ballot_sync(0xffffffffu, bad);
                if (lane == 0) wbad[wid] = bm ? wid * 32 + __ffs(bm) - 1 : kT;
                __syncthreads();
                int c = kT;
#pragma unroll
                for (int w = 0; w < kW; w++) c = min(c, wbad[w]);
                if (c == kT) {  // the whole chunk stayed in the binade
                    s = pr_make(ks, base + total);
                    break;
                }
                if (tid == c) {  // the float path from the exact running sum
                    float s2 = c == start ? s : pr_make(ks, base + I - L);
#pragma unroll
                    for (int k = 0; k < kHubK; k++) s2 += x[k];
                    s_sh = s2;
                }
                __syncthreads();
                s = s_sh;
                start = c + 1;
                if (start >= kT) break;
            }
        }
        if (tid == 0) pr_write(a, v, s);
        __syncthreads();  // head and s_sh are reused by the next hub
    }
}

// Hubs [h0, h1) of the list: one WARP per vertex over its staged run --
// the integer scan of pr_order.cuh with shuffles only (no CTA barrier), so
// a SM keeps dozens of hubs in flight.  Every lane first folds the first
// kWarpHead values itself (each value broadcast by a shuffle, the same adds
// in every lane); then chunks of 32 * kHubK values, lane l owning kHubK
// consecutive ones, loaded one chunk ahead of their scan.
constexpr int kWarpHead = 64;
__global__ void __launch_bounds__(256) k_pr_hub_warp(ExactArgs a, int32_t h0, int32_t h1) {
    constexpr int kChunk = 32 * kHubK;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t h = h0 + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); h < h1; h += warps) {
        const int32_t v = __ldg(&a.hub_v[h]);
        const int32_t n = __ldg(&a.rrow[v + 1]) - __ldg(&a.rrow[v]);
        const float *run = a.x_stage + __ldg(&a.stage_off[h]);
        const int32_t H = min(n, kWarpHead);
        const float h_lo = lane < H ? __ldcs(run + lane) : 0.f;
        const float h_hi = lane + 32 < H ? __ldcs(run + lane + 32) : 0.f;
        float x[kHubK], xn[kHubK];
        hub_load(run, n, H, lane, xn);  // the first chunk's loads go out before the head is folded
        float s = 0.f;
        for (int i = 0; i < H; i++) s += __shfl_sync(0xffffffffu, i < 32 ? h_lo : h_hi, i & 31);
        for (int32_t pos = H; pos < n; pos += kChunk) {
#pragma unroll
            for (int k = 0; k < kHubK; k++) x[k] = xn[k];
            if (pos + kChunk < n) hub_load(run, n, pos + kChunk, lane, xn);
            int start = 0;  // lanes before it have folded their values
            for (;;) {
                const uint32_t bits = __float_as_uint(s);
                const uint32_t ks = bits >> 23, base = (bits & 0x7fffffu) | 0x800000u;
                uint32_t L = 0;
                bool tie = false;
                if (lane >= start) {
#pragma unroll
                    for (int k = 0; k < kHubK; k++) L += pr_units(x[k], ks, tie);
                    L = min(L, 1u << 23);
                }
                uint32_t I = L;  // inclusive prefix (< 2^28: 32 lanes of at most 2^23)
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, I, off);
                    if (lane >= off) I += y;
                }
                const uint32_t total = __shfl_sync(0xffffffffu, I, 31);
                const bool bad = lane >= start && (ks == 0 || ks == 255 || tie || base + I >= (1u << 24));
                const unsigned bm = __ballot_sync(0xffffffffu, bad);
                if (!bm) {  // the whole chunk stayed in the binade
                    s = pr_make(ks, base + total);
                    break;
                }
                const int c = __ffs(bm) - 1;
                float s2 = c == start ? s : pr_make(ks, base + I - L);
                if (lane == c) {  // the float path from the exact running sum
#pragma unroll
                    for (int k = 0; k < kHubK; k++) s2 += x[k];
                }
                s = __shfl_sync(0xffffffffu, s2, c);
                start = c + 1;
                if (start >= 32) break;
            }
        }
        if (lane == 0) pr_write(a, v, s);
    }
}

// ---- building the sliced ELL (once per graph and order) ------------------------
// Sort keys: vertices of more than max_rows in-edges first, then by in-degree
// (largest first), those without in-edges last; counts[0], [1]: the first and
// the last of these.
__global__ void k_sell_keys(const int32_t *rrow, int32_t V, int32_t max_rows, uint32_t *key, uint32_t *val,
                            uint32_t *counts) {
    uint32_t nh = 0, nz = 0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V;
         v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t d = rrow[v + 1] - rrow[v];
        key[v] = d > max_rows ? 0u : (uint32_t)(max_rows - d) + 1u;
        val[v] = (uint32_t)v;
        nh += d > max_rows;
        nz += d == 0;
    }
    nh = __reduce_add_sync(0xffffffffu, nh);
    nz = __reduce_add_sync(0xffffffffu, nz);
    if ((threadIdx.x & 31) == 0) {
        if (nh) atomicAdd(&counts[0], nh);
        if (nz) atomicAdd(&counts[1], nz);
    }
}
// rows of each group of the n vertices in `order`; counts[0]: groups longer than kSellShort
__global__ void k_sell_rows(const uint32_t *order, int32_t n, int32_t ngroups, const int32_t *rrow, int32_t *rows,
                            uint32_t *counts) {
    uint32_t nl = 0;
    for (int32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gridDim.x * blockDim.x) {
        const uint32_t v = order[(int64_t)g * 32];
        const int32_t r = rrow[v + 1] - rrow[v];
        rows[g] = r;
        nl += r > kSellShort;
    }
    nl = __reduce_add_sync(0xffffffffu, nl);
    if ((threadIdx.x & 31) == 0 && nl) atomicAdd(&counts[0], nl);
}
// Group g: row j, lane l <- position of slot j of the group's vertex l
// (src: the slots of each destination, in the order of the sums).
__global__ void k_sell_fill(const uint32_t *order, int32_t n, int32_t ngroups, const int32_t *rows,
                            const uint32_t *base, const int32_t *rrow, const int32_t *src, const int32_t *pos,
                            const int32_t *outdeg, int32_t *sell_v, int2 *sell_pd, int32_t *sell_src) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ngroups; g += warps) {
        const int64_t i = g * 32 + lane;
        const int32_t v = i < n ? (int32_t)order[i] : -1;
        sell_v[i] = v;
        sell_pd[i] = v >= 0 ? make_int2(pos[v], outdeg[v]) : make_int2(-1, 0);
        const int32_t b = v >= 0 ? rrow[v] : 0;
        const int32_t m = v >= 0 ? rrow[v + 1] - b : 0;
        int32_t *dst = sell_src + (int64_t)base[g] * 32 + lane;
        const int32_t r = rows[g];
        for (int32_t j = 0; j < r; j++) dst[(int64_t)j * 32] = j < m ? pos[src[b + j]] : -1;
    }
}
__global__ void k_zero_fill(const uint32_t *order, int32_t n, const int32_t *pos, const int32_t *outdeg, int32_t *zv,
                            int2 *zpd) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = (int32_t)order[i];
        zv[i] = v;
        zpd[i] = make_int2(pos[v], outdeg[v]);
    }
}
// {first slot, in-degree} of the hubs
__global__ void k_hub_info(const uint32_t *order, int32_t n, const int32_t *rrow, int2 *info) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = order[i];
        info[i] = make_int2(rrow[v], rrow[v + 1] - rrow[v]);
    }
}

// Positions of the staged hubs' sources: item {stage offset, length} of the
// slots from meg_off[item] on.
__global__ void k_stage_fill(const int2 *items, const int32_t *meg_off, int32_t nitems, const int32_t *meg_src,
                             const int32_t *pos, int32_t *stage_src) {
    for (int32_t i = blockIdx.x; i < nitems; i += gridDim.x) {
        const int2 it = items[i];
        const int32_t o = meg_off[i];
        for (int32_t k = threadIdx.x; k < it.y; k += blockDim.x)
            stage_src[(int64_t)it.x + k] = pos[meg_src[(int64_t)o + k]];
    }
}

// ---- contribution layout ------------------------------------------------------
// Sort key of a vertex: its out-degree class, four per octave, the largest
// degrees first (flat: one class, for graphs without hubs), and in a class its
// in-degree, the order of the sliced ELL; vertices without out-edges last.
// The classes keep the hot contributions in few lines; the order in a class
// makes a warp's 32 new contributions a few runs of them (in id order instead,
// us per superstep: uniform 6 10^6 / 6 10^7 285, here 268; R-MAT 4 10^6 / 6 10^7
// 284 / 280, 2^24 / 2^28 965 / 957).
constexpr int kDegClasses = 128;
constexpr int kInKeyBits = 16;  // of the in-degree, at most; fewer where the largest needs fewer
__host__ __device__ inline uint32_t degree_key(uint32_t d) {
    if (d == 0) return kDegClasses;
    uint32_t e = 0;
    while (e < 31 && (d >> (e + 1))) e++;
    const uint32_t frac = e >= 2 ? (d >> (e - 2)) & 3u : (d << (2 - e)) & 3u;
    return kDegClasses - 1 - (4 * e + frac);
}
__global__ void k_deg_keys(const int32_t *outdeg, const int32_t *rrow, int32_t V, bool flat, int in_bits,
                           uint32_t *key, uint32_t *val) {
    const uint32_t mask = (1u << in_bits) - 1u;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V;
         v += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t c = flat && outdeg[v] > 0 ? 0u : degree_key((uint32_t)outdeg[v]);
        const uint32_t in = in_bits ? min((uint32_t)(rrow[v + 1] - rrow[v]), mask) : 0u;
        key[v] = (c << in_bits) | (mask - in);
        val[v] = (uint32_t)v;
    }
}
__global__ void k_pos(const uint32_t *key, const uint32_t *val, int32_t V, int in_bits, int32_t *pos) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V;
         i += (int64_t)gridDim.x * blockDim.x)
        pos[val[i]] = (key[i] >> in_bits) < kDegClasses ? (int32_t)i : -1;
}

__global__ void k_map_pos(const int32_t *src, int64_t E, const int32_t *pos, int32_t *out) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E;
         e += (int64_t)gridDim.x * blockDim.x)
        out[e] = pos[src[e]];
}

// Schedule 6, send (SendMsgAA, MPG/UserOperators.h:48-70): every vertex
// writes its contribution into the message slot of each out-edge.
__global__ void k_pr_send(PrArgs a) {
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < a.V;
         u += (int64_t)gridDim.x * blockDim.x) {
        const int32_t b = a.row[u], n = a.row[u + 1] - b;
        if (n == 0) continue;
        const float m = a.contrib_in[a.pos[u]];
        for (int32_t e = b; e < b + n; e++) a.msg[a.mslot[e]] = m;
    }
}

__global__ void k_pr_init(const int32_t *outdeg, const int32_t *pos, int32_t V, float init, float *contrib) {
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < V;
         u += (int64_t)gridDim.x * blockDim.x) {
        const int32_t d = outdeg[u];
        if (d > 0) contrib[pos[u]] = init / (float)d;
    }
}

// The first superstep's contributions from a given rank vector.
__global__ void k_pr_init_vec(const int32_t *outdeg, const int32_t *pos, int32_t V, const float *init,
                              float *contrib) {
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < V;
         u += (int64_t)gridDim.x * blockDim.x) {
        const int32_t d = outdeg[u];
        if (d > 0) contrib[pos[u]] = init[u] / (float)d;
    }
}

__global__ void k_copy(float *dst, const float *src, int32_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

__global__ void k_fill(float *x, int32_t n, float v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        x[i] = v;
}

// MEG order, step 1: edge e (the k-th out-edge of u in reference order) has
// MEG position colstart[k] + rank[u]; order[pos] = e.
__global__ void k_meg_scatter(const int32_t *row, const int32_t *esrc, const int32_t *rank,
                              const int32_t *colstart, int64_t E, uint32_t *order) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = esrc[e];
        const int32_t k = (int32_t)(e - row[u]);
        order[(int64_t)colstart[k] + rank[u]] = (uint32_t)e;
    }
}

// step 2: (destination, edge) pairs in MEG position order, for the stable
// sort by destination
__global__ void k_meg_keys(const uint32_t *order, const int32_t *col, int64_t E, uint32_t *keys) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < E;
         i += (int64_t)gridDim.x * blockDim.x)
        keys[i] = (uint32_t)col[order[i]];
}

// step 3: slot p of the sorted sequence holds edge vals[p]
__global__ void k_meg_finish(const uint32_t *vals, const int32_t *esrc, int64_t E, int32_t *meg_src,
                             int32_t *meg_slot) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < E;
         p += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t e = vals[p];
        meg_src[p] = esrc[e];
        meg_slot[e] = (int32_t)p;
    }
}

}  // namespace

void build_meg_order(Context &ctx, const Graph &g, PrState &st) {
    if (st.meg_built) return;
    const int32_t V = g.V;
    const int64_t E = g.E;
    cudaStream_t s = ctx.stream;
    std::vector<int32_t> row((size_t)V + 1);
    copy_sync(ctx.stream, row.data(), g.row.p, sizeof(int32_t) * ((size_t)V + 1));
    // GraphIR::sortByDegree: std::sort of the vertices in id order by a
    // degree-descending comparator.  The permutation std::sort produces
    // depends only on the comparison results, so sorting (degree, id)
    // records with the same comparison reproduces the reference's.
    struct Node {
        int32_t deg, id;
    };
    std::vector<Node> nodes((size_t)V);
    for (int32_t v = 0; v < V; v++) nodes[v] = Node{row[v + 1] - row[v], v};
    std::sort(nodes.begin(), nodes.end(), [](const Node &l, const Node &r) { return l.deg > r.deg; });
    std::vector<int32_t> rank((size_t)V);
    for (int32_t i = 0; i < V; i++) rank[nodes[i].id] = i;
    // buildMEG: column k holds the k-th edge of every vertex with more than
    // k edges, in sorted order; colstart[k] = edges in columns before k
    const int32_t maxdeg = V ? nodes[0].deg : 0;
    std::vector<int64_t> cnt((size_t)maxdeg + 2, 0);
    for (int32_t v = 0; v < V; v++) cnt[row[v + 1] - row[v]]++;
    std::vector<int32_t> colstart((size_t)maxdeg + 1, 0);
    int64_t above = (int64_t)V - cnt[0], acc = 0;  // vertices with degree > k
    for (int32_t k = 0; k < maxdeg; k++) {
        colstart[k] = (int32_t)acc;
        acc += above;
        above -= cnt[k + 1];
    }
    colstart[maxdeg] = (int32_t)acc;
    DevBuf d_rank, d_col, order, keys;
    d_rank.reserve(sizeof(int32_t) * std::max<size_t>(V, 1));
    d_col.reserve(sizeof(int32_t) * colstart.size());
    const size_t eb = sizeof(uint32_t) * (size_t)std::max<int64_t>(E, 1);
    order.reserve(eb);
    keys.reserve(eb);
    st.meg_src.reserve(eb);
    st.meg_slot.reserve(eb);
    MB_CUDA(cudaMemcpyAsync(d_rank.p, rank.data(), sizeof(int32_t) * (size_t)V, cudaMemcpyHostToDevice, s));
    MB_CUDA(cudaMemcpyAsync(d_col.p, colstart.data(), sizeof(int32_t) * colstart.size(), cudaMemcpyHostToDevice, s));
    if (E > 0) {
        const int grid = grid_for(E, 256, ctx.num_sms * 16);
        k_meg_scatter<<<grid, 256, 0, s>>>(g.row.as<int32_t>(), g.esrc.as<int32_t>(), d_rank.as<int32_t>(),
                                           d_col.as<int32_t>(), E, order.as<uint32_t>());
        k_meg_keys<<<grid, 256, 0, s>>>(order.as<uint32_t>(), g.col.as<int32_t>(), E, keys.as<uint32_t>());
        MB_CHECK_LAUNCH();
        int bits = 1;
        while (bits < 32 && ((int64_t)1 << bits) < (int64_t)V) bits++;
        radix_sort_pairs(ctx, keys.as<uint32_t>(), order.as<uint32_t>(), E, bits, s);
        k_meg_finish<<<grid, 256, 0, s>>>(order.as<uint32_t>(), g.esrc.as<int32_t>(), E,
                                          st.meg_src.as<int32_t>(), st.meg_slot.as<int32_t>());
        MB_CHECK_LAUNCH();
    }
    MB_CUDA(cudaStreamSynchronize(s));
    d_rank.release(); d_col.release(); order.release(); keys.release();
    st.meg_built = true;
}

void PrState::ensure(Context &ctx, const Graph &g) {
    if (built && V == g.V && E == g.E) return;
    release();
    V = g.V;
    E = g.E;
    rank.reserve(sizeof(float) * (size_t)V);
    contrib[0].reserve(sizeof(float) * (size_t)V);
    contrib[1].reserve(sizeof(float) * (size_t)V);
    // contribution layout: by out-degree class, in-degree (or id) order within;
    // vertices without out-edges send nothing and have no position
    cudaStream_t s = ctx.stream;
    const int gridV = grid_for(V, 256, ctx.num_sms * 16);
    DevBuf key, val;
    try {
        key.reserve(sizeof(uint32_t) * (size_t)V);
        val.reserve(sizeof(uint32_t) * (size_t)V);
        pos.reserve(sizeof(int32_t) * (size_t)V);
        int in_bits = 0;
        while (by_indegree && in_bits < kInKeyBits && (g.max_indeg >> in_bits) != 0) in_bits++;
        k_deg_keys<<<gridV, 256, 0, s>>>(g.outdeg.as<int32_t>(), g.rrow.as<int32_t>(), V, g.max_outdeg <= 64, in_bits,
                                         key.as<uint32_t>(), val.as<uint32_t>());
        MB_CHECK_LAUNCH();
        radix_sort_pairs(ctx, key.as<uint32_t>(), val.as<uint32_t>(), V, 8 + in_bits, s);
        k_pos<<<gridV, 256, 0, s>>>(key.as<uint32_t>(), val.as<uint32_t>(), V, in_bits, pos.as<int32_t>());
        MB_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
        key.release(); val.release();
        throw;
    }
    key.release(); val.release();
    built = true;
}

void PrState::ensure_fixed(Context &ctx, const Graph &g) {
    if (fixed_built) return;
    // heavy-vertex work list, built once per graph from the in-degree offsets:
    // one item per block; hubs (more than one block) get block-sum slots
    std::vector<int32_t> rrow(V + 1);
    copy_sync(ctx.stream, rrow.data(), g.rrow.p, sizeof(int32_t) * (V + 1));
    std::vector<int4> it;
    std::vector<int32_t> hv, hf;
    int32_t slots = 0;
    for (int32_t v = 0; v < V; v++) {
        const int64_t d = (int64_t)rrow[v + 1] - rrow[v];
        if (d <= kPrLight) continue;
        if (d <= kPrBlock) {
            it.push_back(make_int4(rrow[v], rrow[v + 1], v, -1));
            continue;
        }
        hv.push_back(v);
        hf.push_back(slots);
        for (int64_t j0 = rrow[v]; j0 < rrow[v + 1]; j0 += kPrBlock)
            it.push_back(make_int4((int32_t)j0, (int32_t)std::min<int64_t>(rrow[v + 1], j0 + kPrBlock),
                                   v, slots++));
    }
    hf.push_back(slots);
    // longest blocks first: the warps that take hub blocks start earliest
    // (the order of the items does not change any sum)
    std::stable_sort(it.begin(), it.end(),
                     [](const int4 &x, const int4 &y) { return (x.y - x.x) > (y.y - y.x); });
    nitems = (int32_t)it.size();
    nhub = (int32_t)hv.size();
    nlong = 0;
    while (nlong < nitems && it[nlong].y - it[nlong].x > kPrShortItem) nlong++;
    items.reserve(sizeof(int4) * std::max<size_t>(it.size(), 1));
    hub_v.reserve(sizeof(int32_t) * std::max<size_t>(hv.size(), 1));
    hub_first.reserve(sizeof(int32_t) * hf.size());
    blk_sum.reserve(sizeof(float) * std::max<int32_t>(slots, 1));
    copy_sync(ctx.stream, items.p, it.data(), sizeof(int4) * it.size());
    copy_sync(ctx.stream, hub_v.p, hv.data(), 4 * hv.size());
    copy_sync(ctx.stream, hub_first.p, hf.data(), 4 * hf.size());
    if (nitems) {
        hcol.reserve(sizeof(int32_t) * (size_t)E);
        k_map_pos<<<grid_for(E, 256, ctx.num_sms * 16), 256, 0, ctx.stream>>>(
            g.rcol.as<int32_t>(), E, pos.as<int32_t>(), hcol.as<int32_t>());
        MB_CHECK_LAUNCH();
    }
    build_sell(ctx, g, kPrLight, g.rcol.as<int32_t>(), light, nullptr);
    fixed_built = true;
}

// The sliced ELL of the vertices with 1 to max_rows in-edges, the list of
// those without any, and (hubs, when not null) the others' {vertex, first
// slot, in-degree} in id order.
void PrState::build_sell(Context &ctx, const Graph &g, int32_t max_rows, const int32_t *src, PrSell &out,
                         std::vector<HubInfo> *hubs) {
    cudaStream_t s = ctx.stream;
    const int gridV = grid_for(V, 256, ctx.num_sms * 16);
    max_rows = std::min(max_rows, g.max_indeg);
    int bits = 1;
    while (bits < 32 && ((int64_t)1 << bits) < (int64_t)max_rows + 2) bits++;
    DevBuf key, val, cnt;
    auto drop = [&] { key.release(); val.release(); cnt.release(); };
    try {
        key.reserve(sizeof(uint32_t) * (size_t)V);
        val.reserve(sizeof(uint32_t) * (size_t)V);
        cnt.reserve(4 * sizeof(uint32_t));
        MB_CUDA(cudaMemsetAsync(cnt.p, 0, 4 * sizeof(uint32_t), s));
        k_sell_keys<<<gridV, 256, 0, s>>>(g.rrow.as<int32_t>(), V, max_rows, key.as<uint32_t>(), val.as<uint32_t>(),
                                          cnt.as<uint32_t>());
        MB_CHECK_LAUNCH();
        radix_sort_pairs(ctx, key.as<uint32_t>(), val.as<uint32_t>(), V, bits, s);
        uint32_t c[2] = {0, 0};
        copy_sync(s, c, cnt.p, sizeof(c));
        const int32_t nh = (int32_t)c[0], n = V - nh - (int32_t)c[1];
        const uint32_t *order = val.as<uint32_t>();
        out.nz = (int32_t)c[1];
        out.ngroups = (int32_t)(((int64_t)n + 31) / 32);
        out.nlong = 0;
        if (hubs) {
            hubs->resize((size_t)nh);
            if (nh) {
                std::vector<int32_t> hv((size_t)nh);
                std::vector<int2> info((size_t)nh);
                DevBuf hi;
                hi.reserve(sizeof(int2) * (size_t)nh);
                k_hub_info<<<grid_for(nh, 256, ctx.num_sms * 4), 256, 0, s>>>(order, nh, g.rrow.as<int32_t>(),
                                                                              hi.as<int2>());
                copy_sync(s, info.data(), hi.p, sizeof(int2) * (size_t)nh);
                copy_sync(s, hv.data(), order, sizeof(int32_t) * (size_t)nh);
                hi.release();
                for (int32_t i = 0; i < nh; i++) (*hubs)[i] = HubInfo{hv[i], info[i].x, info[i].y};
            }
        }
        if (out.ngroups) {
            out.rows.reserve(sizeof(int32_t) * (size_t)out.ngroups);
            out.base.reserve(sizeof(uint32_t) * (size_t)out.ngroups);
            out.v.reserve(sizeof(int32_t) * 32 * (size_t)out.ngroups);
            out.pd.reserve(sizeof(int2) * 32 * (size_t)out.ngroups);
            k_sell_rows<<<grid_for(out.ngroups, 256, ctx.num_sms * 16), 256, 0, s>>>(
                order + nh, n, out.ngroups, g.rrow.as<int32_t>(), out.rows.as<int32_t>(), cnt.as<uint32_t>() + 2);
            MB_CHECK_LAUNCH();
            scan_exclusive_u32(ctx, out.rows.as<uint32_t>(), out.base.as<uint32_t>(), out.ngroups,
                               cnt.as<uint32_t>() + 3, s);
            uint32_t t[2] = {0, 0};
            copy_sync(s, t, cnt.as<uint32_t>() + 2, sizeof(t));
            out.nlong = (int32_t)t[0];
            out.src.reserve(sizeof(int32_t) * 32 * (size_t)t[1]);
            k_sell_fill<<<grid_for((int64_t)out.ngroups * 32, 256, ctx.num_sms * 16), 256, 0, s>>>(
                order + nh, n, out.ngroups, out.rows.as<int32_t>(), out.base.as<uint32_t>(), g.rrow.as<int32_t>(),
                src, pos.as<int32_t>(), g.outdeg.as<int32_t>(), out.v.as<int32_t>(), out.pd.as<int2>(),
                out.src.as<int32_t>());
            MB_CHECK_LAUNCH();
        }
        if (out.nz) {
            out.zv.reserve(sizeof(int32_t) * (size_t)out.nz);
            out.zpd.reserve(sizeof(int2) * (size_t)out.nz);
            k_zero_fill<<<grid_for(out.nz, 256, ctx.num_sms * 16), 256, 0, s>>>(
                order + nh + n, out.nz, pos.as<int32_t>(), g.outdeg.as<int32_t>(), out.zv.as<int32_t>(),
                out.zpd.as<int2>());
            MB_CHECK_LAUNCH();
        }
        MB_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
        drop();
        throw;
    }
    drop();
}

void PrState::ensure_exact(Context &ctx, const Graph &g, int32_t hub_min) {
    if (exact_built && x_hub_min == hub_min) return;
    build_meg_order(ctx, g, *this);
    release_exact();
    cudaStream_t s = ctx.stream;
    std::vector<HubInfo> hubs;
    build_sell(ctx, g, hub_min, meg_src.as<int32_t>(), sell, &hubs);
    std::stable_sort(hubs.begin(), hubs.end(), [](const HubInfo &x, const HubInfo &y) { return x.n > y.n; });
    x_nhub = (int32_t)hubs.size();
    std::vector<int32_t> hv((size_t)x_nhub);
    for (int32_t h = 0; h < x_nhub; h++) hv[h] = hubs[h].v;
    x_hub_v.reserve(sizeof(int32_t) * std::max<size_t>(hubs.size(), 1));
    copy_sync(s, x_hub_v.p, hv.data(), 4 * hv.size());
    x_nbig = 0;  // the hubs are sorted: the big ones come first
    while (x_nbig < x_nhub && hubs[x_nbig].n > kHubBig) x_nbig++;
    // staging: hub h's run at a multiple of 4 floats, items of kStageItem slots
    std::vector<int64_t> soff((size_t)std::max<int32_t>(x_nhub, 1), 0);
    std::vector<int2> items;
    std::vector<int32_t> meg_off;
    int64_t staged = 0;
    for (int32_t h = 0; h < x_nhub; h++) {
        const int32_t n = hubs[h].n;
        soff[h] = staged;
        for (int32_t j0 = 0; j0 < n; j0 += kStageItem) {
            items.push_back(make_int2((int32_t)(staged + j0), std::min(kStageItem, n - j0)));
            meg_off.push_back(hubs[h].first + j0);
        }
        staged += ((int64_t)n + 3) & ~(int64_t)3;
    }
    if (staged > 0x7fffffffll) fail(MB_ERR_UNSUPPORTED, "PageRank: hub staging exceeds 2^31 slots");
    nstage_items = (int32_t)items.size();
    x_stage.reserve(sizeof(float) * (size_t)std::max<int64_t>(staged, 1));
    stage_off.reserve(sizeof(int64_t) * soff.size());
    stage_items.reserve(sizeof(int2) * std::max<size_t>(items.size(), 1));
    copy_sync(s, stage_off.p, soff.data(), 8 * soff.size());
    if (nstage_items) {
        stage_src.reserve(sizeof(int32_t) * (size_t)staged);
        copy_sync(s, stage_items.p, items.data(), sizeof(int2) * items.size());
        DevBuf off;
        off.reserve(sizeof(int32_t) * meg_off.size());
        try {
            copy_sync(s, off.p, meg_off.data(), sizeof(int32_t) * meg_off.size());
            k_stage_fill<<<std::min(nstage_items, ctx.num_sms * 8), 256, 0, s>>>(
                stage_items.as<int2>(), off.as<int32_t>(), nstage_items, meg_src.as<int32_t>(), pos.as<int32_t>(),
                stage_src.as<int32_t>());
            MB_CHECK_LAUNCH();
            MB_CUDA(cudaStreamSynchronize(s));
        } catch (...) {
            off.release();
            throw;
        }
        off.release();
    }
    MB_CUDA(cudaStreamSynchronize(s));
    x_hub_min = hub_min;
    exact_built = true;
}

void run_pagerank(Context &ctx, Graph &g, PrState &st, int32_t iters, float init, int sched,
                  mb_stats *stats, const float *init_vec) {
    st.ensure(ctx, g);
    const bool ref_order = ctx.pr_order == MB_PR_ORDER_REFERENCE;
    const bool unfused = sched == MB_SCHED_PUSH_UNFUSED;
    const int32_t hub_min = ctx.tunable[MB_TUNE_PR_HUB_MIN] > 0
                                ? (int32_t)std::min<int64_t>(ctx.tunable[MB_TUNE_PR_HUB_MIN], 0x7fffffff)
                                : (int32_t)std::min<int64_t>(std::max<int64_t>(g.E >> 14, kHubMinLeast), kHubMinMost);
    if (ref_order) build_meg_order(ctx, g, st);
    if (ref_order && !unfused) st.ensure_exact(ctx, g, hub_min);
    if (!ref_order) st.ensure_fixed(ctx, g);
    if (unfused) st.msg.reserve(sizeof(float) * (size_t)std::max<int64_t>(g.E, 1));
    // only for the hubs' scans and the heavy blocks
    if (!unfused && (ref_order ? st.x_nhub : st.nitems) > 0) st.ensure_streams();
    cudaStream_t s = ctx.stream;
    auto args = [&](int it) {
        const int parity = it & 1;
        PrArgs a;
        a.V = g.V;
        a.E = g.E;
        a.rrow = g.rrow.as<int32_t>();
        a.outdeg = g.outdeg.as<int32_t>();
        a.row = g.row.as<int32_t>();
        a.mslot = ref_order ? st.meg_slot.as<int32_t>() : g.mslot.as<int32_t>();
        a.contrib_in = st.contrib[parity].as<float>();
        a.contrib_out = st.contrib[parity ^ 1].as<float>();
        a.rank_out = it == iters - 1 ? st.rank.as<float>() : nullptr;
        a.pos = st.pos.as<int32_t>();
        a.hcol = st.hcol.as<int32_t>();
        a.msg = st.msg.as<float>();
        a.items = st.items.as<int4>();
        a.nitems = st.nitems;
        a.hub_v = st.hub_v.as<int32_t>();
        a.hub_first = st.hub_first.as<int32_t>();
        a.nhub = st.nhub;
        a.blk_sum = st.blk_sum.as<float>();
        a.nlong = st.nlong;
        return a;
    };
    // grids of exactly the resident blocks (grid-stride loops: no tail wave)
    auto resident = [&](const void *k, int threads) {
        int per_sm = 0;
        MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, 0));
        return ctx.num_sms * std::max(per_sm, 1);
    };
    const int grid_pull = resident((const void *)k_pr_pull<true>, kPrThreads);
    // short sliced-ELL groups a warp takes at once: the tunable, else 1, and 2 below
    // 8 edges per vertex, where one leaves a warp few gathers (1 / 2 / 4, us per
    // superstep: uniform 9 10^5 with 4 / 8 / 16 edges per vertex 17.9 / 16.8 / 20.7,
    // 30.4 / 30.7 / 38.7, 56.6 / 58.7 / 62.7; R-MAT 4 10^6 / 6 10^7 232 / 233 / 238, 3 10^6 /
    // 3 10^7 80 / 78 / 81; the 1448^2 grid 23.7 / 16.2 / 19.9, the 128^3 torus 24.6 / 17.5 /
    // 23.2, a binary tree of 2^19 6.9 / 5.2 / 6.6)
    const int vpl = ctx.tunable[MB_TUNE_PR_LIGHT_VPL] > 0 ? (int)ctx.tunable[MB_TUNE_PR_LIGHT_VPL]
                    : g.E < 8 * (int64_t)g.V               ? 2
                                                           : 1;
    const int pair = ctx.tunable[MB_TUNE_PR_SHORT_PAIR] > 0 ? (int)ctx.tunable[MB_TUNE_PR_SHORT_PAIR]
                                                             : kShortPairDefault;
    // each variant's grid is its own resident block count (registers differ)
    const void *heavy_fn[2][3] = {{(const void *)k_heavy_blocks<false, 1>, (const void *)k_heavy_blocks<false, 2>,
                                   (const void *)k_heavy_blocks<false, 4>},
                                  {(const void *)k_heavy_blocks<true, 1>, (const void *)k_heavy_blocks<true, 2>,
                                   (const void *)k_heavy_blocks<true, 4>}};
    const void *sell_fn[3] = {(const void *)k_pr_sell<1>, (const void *)k_pr_sell<2>, (const void *)k_pr_sell<4>};
    const int pi = pair == 1 ? 0 : pair == 2 ? 1 : 2, vi = vpl == 1 ? 0 : vpl == 2 ? 1 : 2;
    const int64_t heavy_threads = heavy_units(st.nitems, st.nlong, pair) * 32;
    const int grid_heavy[2] = {grid_for(heavy_threads, 256, resident(heavy_fn[0][pi], 256)),
                               grid_for(heavy_threads, 256, resident(heavy_fn[1][pi], 256))};
    auto heavy = [&](bool from_msg, cudaStream_t cs, const PrArgs &a) {
        PrArgs arg = a;
        void *params[] = {&arg};
        MB_CUDA(cudaLaunchKernel(heavy_fn[from_msg][pi], grid_heavy[from_msg], 256, params, 0, cs));
    };
    auto sell_args = [&](const PrSell &l) {
        SellArgs a{};
        a.v = l.v.as<int32_t>();
        a.pd = l.pd.as<int2>();
        a.rows = l.rows.as<int32_t>();
        a.base = l.base.as<uint32_t>();
        a.src = l.src.as<int32_t>();
        a.ngroups = l.ngroups;
        a.nlong = l.nlong;
        return a;
    };
    // one superstep of the vertices of a sliced ELL, those without in-edges included
    auto sell_step = [&](cudaStream_t cs, const PrSell &l, const PrArgs &p, int it) {
        SellArgs a = sell_args(l);
        a.contrib_in = p.contrib_in;
        a.contrib_out = p.contrib_out;
        a.rank_out = p.rank_out;
        a.zv = l.zv.as<int32_t>();
        a.zpd = l.zpd.as<int2>();
        a.nz = l.nz;
        a.zfirst = it < 2;
        if (!l.ngroups) {
            k_pr_zero<<<grid_for(l.nz, 256, ctx.num_sms * 8), 256, 0, cs>>>(a);
            MB_CHECK_LAUNCH();
            return;
        }
        void *params[] = {&a};
        const int64_t units = (int64_t)l.nlong + (l.ngroups - l.nlong + vpl - 1) / vpl;
        MB_CUDA(cudaLaunchKernel(sell_fn[vi], (unsigned)((units + 7) / 8), 256, params, 0, cs));
    };
    const int grid_vtx = ctx.num_sms * 8;
    const int hub_ctas = ctx.tunable[MB_TUNE_PR_HUB_CTAS] > 0 ? (int)ctx.tunable[MB_TUNE_PR_HUB_CTAS]
                                                               : std::max(ctx.num_sms / 4, 1);
    const int grid_hub_warp = std::max(resident((const void *)k_pr_hub_warp, 256) / 2, 1);
    const int grid_stage = resident((const void *)k_pr_hub_stage, 256);
    const int grid_hub_big = std::min(resident((const void *)k_pr_hub_exact<512, 512>, 512), hub_ctas);
    auto exact_args = [&](const PrArgs &a) {
        ExactArgs x;
        x.rrow = g.rrow.as<int32_t>();
        x.pos = st.pos.as<int32_t>();
        x.stage_src = st.stage_src.as<int32_t>();
        x.outdeg = g.outdeg.as<int32_t>();
        x.contrib_in = a.contrib_in;
        x.contrib_out = a.contrib_out;
        x.rank_out = a.rank_out;
        x.hub_v = st.x_hub_v.as<int32_t>();
        x.nhub = st.x_nhub;
        x.x_stage = st.x_stage.as<float>();
        x.stage_off = st.stage_off.as<int64_t>();
        x.stage_items = st.stage_items.as<int2>();
        x.nstage_items = st.nstage_items;
        return x;
    };
    // all supersteps in one launch (k_pr_resident)
    const PrSell &all = ref_order ? st.sell : st.light;
    int grid_res = 0, res_threads = kResThreads;
    const void *res_fn = (const void *)k_pr_resident<16>;
    int32_t *res_err = (int32_t *)ctx.ctrl_readback();
    *(volatile int32_t *)res_err = 0;
    // A superstep of a small sparse graph is shorter than the barrier between two
    // (us for ten, one launch / one each: 300 vertices with 2 / 4 edges 28 / 24, 28 / 24,
    // 3000 with 2 / 4 / 8 / 16 30 / 27, 30 / 28, 31 / 29, 34 / 40, 10^4 with 2 / 4 32 / 30, 32 / 30,
    // 4 10^4 34 / 34, 36 / 37, 7 10^4 35 / 38, 40 / 40).
    const bool by_launch = g.E < (1 << 15) && g.E < 12 * (int64_t)g.V;
    if (!unfused && iters > 1 && !by_launch && (ref_order ? st.x_nhub == 0 : st.nitems == 0) && all.ngroups > 0) {
        // the groups spread evenly over the SMs: small graphs in smaller CTAs, one
        // per SM (177 groups in 6 CTAs of 32 warps were bound by 6 SMs' gathers), more
        // than 32 groups per SM in two: with full CTAs some SMs had two and others one (us
        // per superstep, launches of their own / full CTAs / so, 21 edges per vertex: 155851
        // vertices 19.0 / 23.3 / 13.8, 215578 22.2 / 24.5 / 18.3, 2^18 28.4 / 25.3 / 22.5)
        const int64_t per_sm = (all.ngroups + ctx.num_sms - 1) / ctx.num_sms;
        const int64_t full = kResThreads / 32, ctas = per_sm > full ? 2 : 1;
        const int64_t warps = std::min<int64_t>(full, std::max<int64_t>(4, (per_sm + ctas - 1) / ctas));
        res_threads = (int)warps * 32;
        grid_res = (int)std::min<int64_t>((all.ngroups + warps - 1) / warps, INT32_MAX);
        if (grid_res > resident(res_fn, res_threads)) res_fn = (const void *)k_pr_resident<8>;
        if (grid_res > resident(res_fn, res_threads)) grid_res = 0;
    }
    if (grid_res && !st.bar.p) {
        st.bar.reserve(256);
        MB_CUDA(cudaMemsetAsync(st.bar.p, 0, 256, s));
    }
    auto emit = [&](cudaStream_t cs) {
        if (init_vec)
            k_pr_init_vec<<<grid_vtx, 256, 0, cs>>>(g.outdeg.as<int32_t>(), st.pos.as<int32_t>(), g.V, init_vec,
                                                    st.contrib[0].as<float>());
        else
            k_pr_init<<<grid_vtx, 256, 0, cs>>>(g.outdeg.as<int32_t>(), st.pos.as<int32_t>(), g.V, init,
                                                st.contrib[0].as<float>());
        MB_CHECK_LAUNCH();
        if (grid_res) {
            SellArgs a = sell_args(all);
            ResidentArgs r;
            r.contrib[0] = st.contrib[0].as<float>();
            r.contrib[1] = st.contrib[1].as<float>();
            r.rank = st.rank.as<float>();
            r.zv = all.zv.as<int32_t>();
            r.zpd = all.zpd.as<int2>();
            r.nz = all.nz;
            r.iters = iters;
            r.bar = st.bar.as<uint32_t>();
            r.err = res_err;
            r.polls = ctx.tunable[MB_TUNE_WAIT_POLLS] >= 0 ? (long)ctx.tunable[MB_TUNE_WAIT_POLLS] : 1l << 22;
            void *params[] = {&a, &r};
            MB_CUDA(cudaLaunchCooperativeKernel(res_fn, dim3(grid_res), dim3(res_threads), params,
                                                0, cs));
            return;
        }
        for (int it = 0; it < iters; it++) {
            PrArgs a = args(it);
            if (ref_order && unfused) {
                // the reference's send -> combine split over the message array,
                // each vertex folded serially in MEG order
                k_pr_send<<<grid_vtx, 256, 0, cs>>>(a);
                k_pr_pull<true, true><<<grid_pull, kPrThreads, 0, cs>>>(a);
                MB_CHECK_LAUNCH();
                continue;
            }
            if (ref_order) {
                ExactArgs x = exact_args(a);
                // the hubs' contributions staged by every SM, then their
                // scans on the side stream beside the rest
                const int32_t nbig = st.x_nbig, nsmall = st.x_nhub - st.x_nbig;
                if (st.x_nhub) {
                    k_pr_hub_stage<<<grid_stage, 256, 0, cs>>>(x);
                    MB_CHECK_LAUNCH();
                    MB_CUDA(cudaEventRecord(st.ev_fork, cs));
                    MB_CUDA(cudaStreamWaitEvent(st.side, st.ev_fork, 0));
                    // the scans beside the rest: the big hubs one CTA each on
                    // few CTAs, then the others one warp each
                    if (nbig)
                        k_pr_hub_exact<512, 512><<<std::min(nbig, grid_hub_big), 512, 0, st.side>>>(x, 0, nbig);
                    if (nsmall) {
                        // the warp scans beside the big hubs' CTAs when those
                        // take several rounds (more big hubs than CTAs);
                        // else after them (measured, 20 supersteps: C5, 301
                        // big hubs on 37 CTAs, 24.0 against 27.7 ms; the C5
                        // generator at 2^21, 22 big hubs, 4.10 against 3.79)
                        cudaStream_t hs = st.side;
                        if (nbig > grid_hub_big) {
                            MB_CUDA(cudaStreamWaitEvent(st.side3, st.ev_fork, 0));
                            hs = st.side3;
                        }
                        k_pr_hub_warp<<<grid_for((int64_t)nsmall * 32, 256, grid_hub_warp), 256, 0, hs>>>(
                            x, nbig, st.x_nhub);
                        if (hs == st.side3) {
                            MB_CUDA(cudaEventRecord(st.ev_join3, st.side3));
                            MB_CUDA(cudaStreamWaitEvent(st.side, st.ev_join3, 0));
                        }
                    }
                    MB_CHECK_LAUNCH();
                }
                sell_step(cs, st.sell, a, it);
                MB_CHECK_LAUNCH();
                if (st.x_nhub) {
                    MB_CUDA(cudaEventRecord(st.ev_join, st.side));
                    MB_CUDA(cudaStreamWaitEvent(cs, st.ev_join, 0));
                }
                continue;
            }
            if (unfused) {
                k_pr_send<<<grid_vtx, 256, 0, cs>>>(a);
                if (a.nitems) heavy(true, cs, a);
                k_pr_pull<true><<<grid_pull, kPrThreads, 0, cs>>>(a);
            } else {
                // the heavy blocks beside the light vertices: neither waits for
                // the other's last warps (us per superstep, in line / beside:
                // R-MAT 10^4 / 10^5 11.2 / 6.5, 1.3M / 17M 58.7 / 48.8, 2^23 / 2^26
                // 225 / 204)
                if (a.nitems) {
                    MB_CUDA(cudaEventRecord(st.ev_fork, cs));
                    MB_CUDA(cudaStreamWaitEvent(st.side, st.ev_fork, 0));
                }
                if (a.nitems) heavy(false, st.side, a);
                sell_step(cs, st.light, a, it);
                if (a.nitems) {
                    MB_CUDA(cudaEventRecord(st.ev_join, st.side));
                    MB_CUDA(cudaStreamWaitEvent(cs, st.ev_join, 0));
                }
            }
            if (a.nhub) k_hub_finalize<<<grid_for(a.nhub, 128, ctx.num_sms * 4), 128, 0, cs>>>(a);
            MB_CHECK_LAUNCH();
        }
        if (iters == 0) {  // no superstep: the ranks are the initial ranks
            if (init_vec) k_copy<<<grid_vtx, 256, 0, cs>>>(st.rank.as<float>(), init_vec, g.V);
            else k_fill<<<grid_vtx, 256, 0, cs>>>(st.rank.as<float>(), g.V, init);
            MB_CHECK_LAUNCH();
        }
    };
    cudaEvent_t e0, e1;
    MB_CUDA(cudaEventCreate(&e0));
    MB_CUDA(cudaEventCreate(&e1));
    try {
        if (ctx.use_graphs) {
            if (!st.exec || st.g_ctx != ctx.id || st.g_iters != iters || st.g_init != init || st.g_init_vec != init_vec ||
                st.g_sched != sched ||
                st.g_order != ctx.pr_order || st.g_tune != ctx.tune_gen) {
                st.drop_exec();
                cudaGraph_t gr;
                MB_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
                try {
                    emit(s);
                } catch (...) {
                    cudaStreamEndCapture(s, &gr);
                    throw;
                }
                MB_CUDA(cudaStreamEndCapture(s, &gr));
                cudaError_t e = cudaGraphInstantiate(&st.exec, gr, 0);
                cudaGraphDestroy(gr);
                MB_CUDA(e);
                st.g_ctx = ctx.id;
                st.g_iters = iters;
                st.g_init = init;
                st.g_init_vec = init_vec;
                st.g_sched = sched;
                st.g_order = ctx.pr_order;
                st.g_tune = ctx.tune_gen;
            }
            MB_CUDA(cudaEventRecord(e0, s));
            MB_CUDA(cudaGraphLaunch(st.exec, s));
            MB_CUDA(cudaEventRecord(e1, s));
        } else {
            MB_CUDA(cudaEventRecord(e0, s));
            emit(s);
            MB_CUDA(cudaEventRecord(e1, s));
        }
        MB_CUDA(cudaEventSynchronize(e1));
        if (grid_res && *(volatile int32_t *)res_err) {
            MB_CUDA(cudaMemsetAsync(st.bar.p, 0, 256, s));
            MB_CUDA(cudaStreamSynchronize(s));
            fail(MB_ERR_TIMEOUT, "pagerank: a barrier between two supersteps timed out");
        }
        float ms = 0;
        MB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (stats) {
            *stats = mb_stats{};
            stats->supersteps = iters;
            stats->edges_traversed = (int64_t)iters * g.E;
            stats->vertices_reached = g.V;
            stats->device_ms = ms;
            stats->schedule_count[unfused ? MB_SCHED_PUSH_UNFUSED : MB_SCHED_PUSH_EDGE_QUEUE] = iters;
            stats->edges_scanned = (int64_t)iters * g.E;
            const PrSell &l = ref_order ? st.sell : st.light;
            int64_t per_step;
            if (ref_order && unfused) per_step = 2;
            else if (unfused) per_step = 2 + (st.nitems > 0) + (st.nhub > 0);
            else {
                per_step = 1 + (ref_order ? (st.x_nhub > 0) + (st.x_nbig > 0) + (st.x_nhub > st.x_nbig)
                                                        : (st.nitems > 0) + (st.nhub > 0));
            }
            stats->kernel_launches = grid_res ? 2 : 1 + (int64_t)iters * per_step + (iters == 0);
        }
    } catch (...) {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
}

}  // namespace mb
