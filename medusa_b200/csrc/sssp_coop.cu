// sssp_coop.cu -- a whole SSSP in one launch, for graphs with hubs under the
// fixed rule.
//
// Frontier Bellman-Ford relaxes 3.7 to 6 edges per reached edge on R-MAT
// graphs.  Distance buckets (near-far: Davidson, Baxter, Garland & Owens,
// IPDPS 2014) cut that to 1.3 to 2, but need three to five times the
// supersteps, which the loop graph's 12-17 us per superstep made a loss.
// Here the supersteps follow one another inside one cooperative grid with one
// barrier each (6-8 us for a small one), so the buckets pay.  Where the steps
// stay small for long, the asynchronous kernel takes the rest (SsspRest).
//
// A superstep relaxes the out-edges of the near queue.  A vertex whose
// distance drops below the threshold T joins the next queue, once per
// superstep (a claim bit; two claim bitmaps in turn, so that a bit is cleared
// while the vertex is expanded and no superstep claims in it); one that drops
// to T or above gets a bit in the far bitmap.  When the queue runs dry, T
// rises by delta, past the least distance the last split kept (the same rules
// as choose_next, engine.cuh), and a split moves the far vertices now below T
// to the queue; one that is below the old T was expanded at that distance
// already and only loses its bit.  Every order reaches the same fixpoint,
// the exact distances; with weights that are not integers too, since a float
// sum along a path is monotone in its start.
// A superstep of at least kBmMin edges claims without asking for the result and
// builds the queue from the claim bitmap in a pass of its own: an append per
// tile costs more there than the pass.
//
// Several sources run in the same launch as (source, vertex) pairs, whatever
// the graph: a superstep's own cost is shared by all of them, and distances
// come out source by source.  The lines of 32 distances per vertex (mssssp.cu)
// relax an edge for all sources at once, but with buckets only 2 or 3 of the 32
// have it in their frontier.  32 sources on the mild R-MAT 2^20 / 2^24: 13.2 ms,
// against 29.4; uniform 5 10^5 / 6 10^6 x 9 1.5 against 5.8; grid 700^2 x 20 3.5 against 12.
#include "coop.cuh"
#include "sssp.cuh"
#include "sssp_coop.cuh"

namespace mb {
namespace {

constexpr int kThreads = 512;
constexpr int kItems = 2;
constexpr int kTileE = kThreads * kItems;
static_assert(kTileE >= kSsspCoopTile, "the tile tables are sized by it");
constexpr int kCtas = 3;  // per SM; 2: 0.82 / 4.3 ms, 4 (32 registers, spills): slower on both
constexpr uint32_t kInf = 0x7f800000u;
constexpr uint32_t kBmMin = 1 << 20;  // 2^19 and less: 2-4% slower
// Bucket width in mean weights.  0.5 / 0.7 / 0.85 / 1 / 1.5 / none, ms: mild R-MAT
// 2^20 / 2^24 0.90 / 0.79 / 0.79 / 0.86 / 1.08 / 1.22; 2^23 / 10^8 3.31 / 3.80 / 3.43 /
// 2.96 / 4.6 / 6.7; the skewed one 2^20 / 2^24 1.05 / 0.95 / 0.99 / 0.99 / 0.98 / 0.96.
// Below kBucketMinE edges the supersteps that buckets add cost more than the
// relaxations that they save, and where the edges per vertex are few there are
// few relaxations to save.  ms, 0.85 / 2 / none / the superstep loop: mild R-MAT 2^16 x 8
// edges per vertex 0.43 / 0.34 / 0.31 / 0.38, 2^18 x 4 0.65 / 0.52 / 0.41 / 0.45, 2^18 x 16
// 0.52 / 0.55 / 0.54 / 0.56, 2^20 x 2 0.96 / 0.69 / 0.48 / 0.50, x 4 0.84 / 0.60 / 0.58 / 0.61, x 6
// 0.81 / 0.68 / 0.74 / 0.72, x 8 0.79 / 0.79 / 0.94 / 0.88, 2^21 x 4 1.04 / 0.84 / 0.88 / 0.95, 2^24 x 4
// 3.8 / 3.6 / 5.8 / 5.3, x 8 5.2 / 6.2 / 10.2 / 8.3; a tree of 2^19 with a hub 1.58 / 0.99 /
// 0.39 / 0.47.
constexpr int64_t kBucketMinE = 1 << 22;
inline float single_width(const Graph &g) {
    if (g.E < kBucketMinE) return 0.f;
    return g.E < 7 * (int64_t)g.V ? 2.f : 0.85f;
}
// Bucket width in mean weights with several sources.  The more out-edges a
// run's frontiers hold, the less a superstep's own cost matters, and the
// narrower the best bucket; a sparse graph without hubs (roads) needs
// supersteps by the hundred at any width.  Measured best: mild R-MAT 2^20 and
// 2^22 x 32 0.4 (13.2 ms; 25.8 at 2.5), 10^5 x 32 0.7 (1.5; 1.6 at 1.2), uniform 5 10^5 x 9
// 1.2 (1.5; 1.7 at 0.4), 5 10^4 x 32 2.5 (0.63; 1.0 at 0.4), grid 700^2 x 20 5 (3.5; 10.3 at
// 0.4), skewed R-MAT 5 10^3 x 32 5 (0.24; 0.79 at 0.4).
inline float pairs_width(const Graph &g, int32_t nsrc) {
    const double e = (double)g.E * nsrc;
    if (async_by_default(g, true)) return 5.f;  // hub-free, at most 6 out-edges per vertex
    if (e >= (double)(1 << 27)) return 0.4f;
    if (e >= (double)(1 << 25)) return 0.9f;
    return e >= (double)(1 << 23) ? 2.5f : 5.f;
}

// The run stops when kHandSteps of its steps in a row have relaxed fewer than
// kHandEdges edges each on average: on a graph of a long diameter a step here
// is 5.4 us of barrier, where the asynchronous kernel follows each path by
// itself.  ms, the superstep loop with that kernel for its tail / here to the end /
// stopping: skewed R-MAT 2^18 with 64 lines of 2000 7.1 / 45 / 6.7, a line of 1.3 10^5
// with a hub 412 / 588 / 200, the 1448^2 grid with a hub of 1000 3.4 / 4.1 / 2.4.  R-MAT
// and uniform graphs have 10^5 edges a step and more in any such row; a ring of
// 2 10^5 vertices with 80 edges each (1.2 10^4) is faster here (3.4; 8.6 in the loop).
constexpr int kHandSteps = 64;
constexpr uint32_t kHandEdges = 4096;

__device__ __forceinline__ float inf_f() { return __uint_as_float(kInf); }

struct alignas(128) SCtr {  // one per iteration in turn, three in all
    unsigned long long q;  // queued vertices << 32 | their out-edges
    uint32_t far;          // a vertex was put off
    uint32_t far_min;      // split: float bits of the least distance kept
};
struct SShared {  // device memory of a run, zero before it
    SCtr ctr[3];
    unsigned long long reached, edges;
    uint32_t ticket;
    alignas(128) uint32_t bar[2];  // polled: a line of its own
};

// kMulti: nsrc sources at once.  A vertex is then a (source, vertex) pair,
// p = source * V + vertex: the index of its distance and of its bits.
struct SArgs {
    int32_t V;
    int64_t W;         // bitmap words, whole units of to_queue
    int32_t nsrc;
    const int32_t *sources;  // kMulti (device)
    uint8_t *qs[2];          // kMulti: the entries' sources
    unsigned long long *front;  // kMulti: the first queue's count << 32 | out-edges
    const int32_t *row, *col;
    const float *wt;
    float *dist;
    uint32_t *claim[2], *far;
    uint2 *q[2];      // {first edge less the out-edges queued before it, those}
    int32_t *qv[2];   // vertices
    int32_t *tf[2];   // first entry of each tile
    SShared *sh;
    SsspCoopOut *out;  // host memory
    int32_t source, cap;
    float delta;       // 0: no buckets
    bool hand;         // the run may stop (SsspRest)
    long polls;
};

template <bool kMulti>
struct SSmem {
    uint32_t off[kTileE + 1];
    int32_t row[kTileE + 1];
    float du[kTileE + 1];
    uint32_t pb[kMulti ? kTileE + 1 : 1];  // source * V
    uint2 out[kTileE];  // found vertices: {first edge, out-edges}
    int32_t outv[kTileE];
    uint8_t outs[kMulti ? kTileE : 1];
    uint32_t nout;
    uint32_t wtot[kThreads / 32];
    unsigned long long base;
};

template <bool kMulti>
__device__ __forceinline__ void write_entry(const SArgs &a, int nx, uint32_t pos, int32_t v, uint32_t src, uint32_t rs,
                                            uint32_t d, uint32_t off) {
    pick(a.q, nx)[pos] = make_uint2(rs - off, off);
    pick(a.qv, nx)[pos] = v;
    if (kMulti) pick(a.qs, nx)[pos] = (uint8_t)src;
    int32_t *tf = pick(a.tf, nx);
    const uint32_t t0 = (off + kTileE - 1) / kTileE, t1 = (off + d - 1) / kTileE;
    for (uint32_t t = t0; t <= t1; t++) tf[t] = (int32_t)pos;
}

template <bool kMulti>
__device__ __forceinline__ void found(SSmem<kMulti> &sm, bool pred, int32_t v, uint32_t src, int32_t rs, uint32_t d) {
    const unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (!mask) return;
    const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&sm.nout, (uint32_t)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) {
        const uint32_t i = base + __popc(mask & lanemask_lt());
        sm.out[i] = make_uint2((uint32_t)rs, d);
        sm.outv[i] = v;
        if (kMulti) sm.outs[i] = (uint8_t)src;
    }
}

// The tile's found vertices -> the next queue, one atomic per tile.
template <bool kMulti>
__device__ __forceinline__ void flush(const SArgs &a, SSmem<kMulti> &sm, unsigned long long *ctr, int nx) {
    __syncthreads();
    const uint32_t n = sm.nout;
    if (n == 0) return;  // the same for every thread
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t i0 = threadIdx.x * kItems;
    uint2 e[kItems];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        e[k] = i0 + k < n ? sm.out[i0 + k] : make_uint2(0u, 0u);
        sum += e[k].y;
    }
    const uint32_t incl = warp_incl_scan_u32(sum);
    if (lane == 31) sm.wtot[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        constexpr int kW = kThreads / 32;
        const uint32_t t = lane < kW ? sm.wtot[lane] : 0u;
        const uint32_t ti = warp_incl_scan_u32(t);
        if (lane < kW) sm.wtot[lane] = ti - t;
        if (lane == kW - 1) {
            sm.base = atomicAdd(ctr, ((unsigned long long)n << 32) | ti);
            sm.nout = 0;
        }
    }
    __syncthreads();
    const unsigned long long base = sm.base;
    uint32_t off = (uint32_t)base + sm.wtot[wid] + incl - sum;
#pragma unroll
    for (int k = 0; k < kItems; k++)
        if (i0 + k < n) {
            write_entry<kMulti>(a, nx, (uint32_t)(base >> 32) + i0 + k, sm.outv[i0 + k], kMulti ? sm.outs[i0 + k] : 0u,
                                e[k].x, e[k].y, off);
            off += e[k].y;
        }
}

// par: the claim bitmap of this superstep.
template <bool kMulti, bool kBm>
__device__ __forceinline__ void push(const SArgs &a, SSmem<kMulti> &sm, int cur, uint32_t n, uint32_t m, float T, int par,
                                     SCtr *ctr) {
    const uint32_t tiles = (m + kTileE - 1) / kTileE;
    const uint2 *q = pick(a.q, cur);
    const int32_t *qv = pick(a.qv, cur), *tf = pick(a.tf, cur);
    uint32_t *claim = pick(a.claim, par), *old = pick(a.claim, par ^ 1);
    bool far = false;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t c0 = t * kTileE, c1 = min(c0 + kTileE, m);
        const int32_t i0 = __ldcg(&tf[t]);
        const int32_t i1 = t + 1 < tiles ? __ldcg(&tf[t + 1]) : (int32_t)n - 1;
        const int k = i1 - i0 + 1;
        for (int j = threadIdx.x; j < k; j += kThreads) {
            const uint2 e = __ldcg(&q[i0 + j]);
            const int32_t u = __ldcg(&qv[i0 + j]);
            const uint32_t pb = kMulti ? (uint32_t)__ldcg(&pick(a.qs, cur)[i0 + j]) * (uint32_t)a.V : 0u;
            const uint32_t p = pb + (uint32_t)u;
            sm.off[j] = e.y;
            sm.row[j] = (int32_t)e.x;
            sm.du[j] = __ldcg(&a.dist[p]);
            if (kMulti) sm.pb[j] = pb;
            old[p >> 5] = 0u;  // every bit set there is of a vertex in this queue
        }
        __syncthreads();
        int32_t v[kItems];
        uint32_t pb[kItems];
        float nd[kItems], dv[kItems];
        {
            const uint32_t e0 = c0 + threadIdx.x * kItems;
            int j = e0 < c1 ? upper_bound_minus1(sm.off, k, e0) : 0;
#pragma unroll
            for (int r = 0; r < kItems; r++) {
                const uint32_t e = e0 + r;
                v[r] = -1;
                pb[r] = 0u;
                nd[r] = 0.f;
                if (e < c1) {
                    while (j + 1 < k && sm.off[j + 1] <= e) j++;
                    if (kMulti) pb[r] = sm.pb[j];
                    const int32_t at = sm.row[j] + (int32_t)e;
                    v[r] = __ldg(&a.col[at]);
                    nd[r] = sm.du[j] + __ldg(&a.wt[at]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kItems; r++) dv[r] = v[r] >= 0 ? __ldcg(&a.dist[pb[r] + (uint32_t)v[r]]) : 0.f;
#pragma unroll
        for (int r = 0; r < kItems; r++) {
            bool own = false;
            int32_t rs = 0, re = 0;
            if (nd[r] < dv[r]) {
                const uint32_t p = pb[r] + (uint32_t)v[r];
                atomicMin((unsigned *)&a.dist[p], __float_as_uint(nd[r]));
                const uint32_t bit = 1u << (p & 31);
                if (nd[r] >= T) {
                    far = true;
                    atomicOr(&a.far[p >> 5], bit);  // a test of the bit first costs more
                } else if (kBm) {
                    atomicOr(&claim[p >> 5], bit);
                } else {
                    rs = __ldg(&a.row[v[r]]);
                    re = __ldg(&a.row[v[r] + 1]);
                    own = !(atomicOr(&claim[p >> 5], bit) & bit);
                }
            }
            if (!kBm)
                found(sm, own && re > rs, v[r], kMulti && own ? pb[r] / (uint32_t)a.V : 0u, rs, (uint32_t)(re - rs));
        }
        if (kBm) __syncthreads();  // the tile's entries are reloaded next
        else flush(a, sm, &ctr->q, cur ^ 1);
    }
    // one store per CTA at most: the same address from every warp queues up
    if (__syncthreads_or(far) && threadIdx.x == 0) ctr->far = 1u;
}

// Vertices of a bitmap -> queue nx.  A warp takes four words (128 vertices) a
// round, their loads in flight together and the next round's words on their
// way; the CTA appends a round with one atomic.  (Word after word, each with
// its own chain of loads and an atomic, a warp's share of a 2^20-vertex bitmap
// took 30 to 60 us.)  kSplit: the far bitmap -- those below T leave it, and of
// these the ones not below T0 are queued; the least distance kept goes to
// ctr->far_min.  Else a claim bitmap, cleared.
template <bool kMulti, bool kSplit>
__device__ __forceinline__ void to_queue(const SArgs &a, CoopRound &cr, uint32_t *bm, float T0, float T, int nx,
                                         SCtr *ctr) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t units = a.W / 4, step = (int64_t)gridDim.x * (kThreads / 32);
    const int64_t first = (int64_t)blockIdx.x * (kThreads / 32);
    uint32_t kept = kInf;
    auto words = [&](int64_t u) {
        return u < units ? __ldcg(reinterpret_cast<const uint4 *>(bm) + u) : make_uint4(0u, 0u, 0u, 0u);
    };
    uint4 next = words(first + wid);
    for (int64_t c = first; c < units; c += step) {
        const int64_t u = c + wid;
        const uint32_t x[4] = {next.x, next.y, next.z, next.w};
        next = words(u + step);
        if (!__syncthreads_or((x[0] | x[1] | x[2] | x[3]) != 0u)) continue;
        const uint32_t p0 = (uint32_t)(u * 128) + lane;
        bool take[4];
        if (kSplit) {
            float d[4];
#pragma unroll
            for (int k = 0; k < 4; k++) d[k] = (x[k] >> lane) & 1u ? __ldcg(&a.dist[p0 + 32 * k]) : inf_f();
            uint32_t keep[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const bool has = (x[k] >> lane) & 1u;
                take[k] = has && d[k] < T && d[k] >= T0;
                const bool stay = has && !(d[k] < T);
                if (stay) kept = min(kept, __float_as_uint(d[k]));
                keep[k] = __ballot_sync(0xffffffffu, stay);
            }
            if (lane == 0 && (keep[0] != x[0] || keep[1] != x[1] || keep[2] != x[2] || keep[3] != x[3]))
                reinterpret_cast<uint4 *>(bm)[u] = make_uint4(keep[0], keep[1], keep[2], keep[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) take[k] = (x[k] >> lane) & 1u;
            if (lane == 0 && (x[0] | x[1] | x[2] | x[3]) != 0u)
                reinterpret_cast<uint4 *>(bm)[u] = make_uint4(0u, 0u, 0u, 0u);
        }
        int32_t rs[4], v[4];
        uint32_t dg[4], src[4], sum = 0, cnt = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            rs[k] = 0;
            dg[k] = 0;
            const uint32_t p = p0 + 32 * k;
            src[k] = kMulti ? p / (uint32_t)a.V : 0u;
            v[k] = (int32_t)(p - src[k] * (uint32_t)a.V);
            if (take[k]) {
                rs[k] = __ldg(&a.row[v[k]]);
                dg[k] = (uint32_t)(__ldg(&a.row[v[k] + 1]) - rs[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            sum += dg[k];
            cnt += dg[k] > 0;
        }
        const unsigned long long base = coop_round_append(cr, cnt, sum, &ctr->q);
        uint32_t pos = (uint32_t)(base >> 32), off = (uint32_t)base;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (dg[k] > 0) {
                write_entry<kMulti>(a, nx, pos, v[k], src[k], (uint32_t)rs[k], dg[k], off);
                pos++;
                off += dg[k];
            }
    }
    if (kSplit) {
        kept = __reduce_min_sync(0xffffffffu, kept);
        if (lane == 0 && kept < kInf) atomicMin(&ctr->far_min, kept);
    }
}

template <bool kMulti>
__global__ void __launch_bounds__(kThreads, kCtas) k_sssp_coop(SArgs a) {
    __shared__ SSmem<kMulti> sm;
    __shared__ CoopRound cr;
    __shared__ unsigned long long s_n[kThreads / 32], s_m[kThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t gt = (int64_t)blockIdx.x * kThreads + tid, gn = (int64_t)gridDim.x * kThreads;
    const float inf = inf_f();
    uint32_t barriers = 0;
    auto sync = [&] { return coop_barrier(a.sh->bar, ++barriers, a.polls, &a.out->err); };
    int cur = 0, par = 0, it = 0, supersteps = 0, splits = 0, err = 0;
    const uint32_t pairs = kMulti ? (uint32_t)a.nsrc * (uint32_t)a.V : (uint32_t)a.V;
    for (int64_t p = gt; p < pairs; p += gn) a.dist[p] = kMedusaMax;
    for (int64_t w = gt; w < a.W; w += gn) {
        a.claim[0][w] = 0u;
        a.claim[1][w] = 0u;
        a.far[w] = 0u;
    }
    if (tid == 0) sm.nout = 0;
    if (!sync()) return;
    // the sources' queue, by the first warp
    if (gt < 32) {
        uint32_t qn = 0, qm = 0;
        for (int32_t i0 = 0; i0 < a.nsrc; i0 += 32) {
            const int32_t i = i0 + lane;
            const int32_t v = i < a.nsrc ? (kMulti ? a.sources[i] : a.source) : -1;
            int32_t rs = 0, re = 0;
            if (v >= 0) {
                rs = __ldg(&a.row[v]);
                re = __ldg(&a.row[v + 1]);
                a.dist[(uint32_t)i * (uint32_t)a.V + (uint32_t)v] = 0.f;
            }
            const uint32_t d = (uint32_t)(re - rs);
            const unsigned in = __ballot_sync(0xffffffffu, d > 0);
            const uint32_t incl = warp_incl_scan_u32(d);
            if (d > 0)
                write_entry<kMulti>(a, 0, qn + __popc(in & lanemask_lt()), v, (uint32_t)i, (uint32_t)rs, d,
                                    qm + incl - d);
            qn += __popc(in);
            qm += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) {
            *a.front = ((unsigned long long)qn << 32) | qm;
            a.sh->ctr[0] = SCtr{0ull, 0u, kInf};
        }
    }
    if (!sync()) return;
    const unsigned long long f0 = __ldcg(a.front);
    uint32_t n = (uint32_t)(f0 >> 32), m = (uint32_t)f0;
    unsigned long long work = 0;
    float T = a.delta > 0.f ? a.delta : inf, fmin = inf;
    bool far = false;
    uint32_t mark = 0;  // work at the start of the row of steps
    for (;; it++) {
        if (n == 0 && !far) break;
        if (it >= a.cap) {
            err = ERR_STEP_CAP;
            break;
        }
        if (!kMulti && a.hand && it % kHandSteps == 0 && it > 0) {
            if ((uint32_t)work - mark < kHandSteps * kHandEdges) {
                if (gt == 0) {
                    a.out->supersteps = supersteps;
                    a.out->splits = splits;
                    a.out->work = work;
                    a.out->n = n;
                    a.out->cur = cur;
                    a.out->T = T;
                    a.out->handed = 1;
                }
                return;
            }
            mark = (uint32_t)work;
        }
        SCtr *ctr = &a.sh->ctr[it % 3];
        // last read before the barrier just passed
        if (gt == 0) a.sh->ctr[(it + 1) % 3] = SCtr{0ull, 0u, kInf};
        if (n == 0) {  // next bucket
            const float T0 = T;
            T = T0 + a.delta;
            if (fmin < inf) T = fmaxf(T, fmin + a.delta);
            if (!(T > T0)) T = __uint_as_float(__float_as_uint(T0) + 1u);
            if (fmin < inf && !(T > fmin)) T = __uint_as_float(__float_as_uint(fmin) + 1u);
            to_queue<kMulti, true>(a, cr, a.far, T0, T, cur, ctr);
            if (!sync()) return;
            fmin = __uint_as_float(__ldcg(&ctr->far_min));
            far = fmin < inf;
            splits++;
        } else {
            work += m;
            const bool bm = m >= kBmMin;
            if (bm) {
                push<kMulti, true>(a, sm, cur, n, m, T, par, ctr);
                if (!sync()) return;
                to_queue<kMulti, false>(a, cr, pick(a.claim, par), 0.f, 0.f, cur ^ 1, ctr);
            } else {
                push<kMulti, false>(a, sm, cur, n, m, T, par, ctr);
            }
            if (!sync()) return;
            far = far || __ldcg(&ctr->far) != 0u;
            cur ^= 1;
            par ^= 1;
            supersteps++;
        }
        const unsigned long long c = __ldcg(&ctr->q);
        n = (uint32_t)(c >> 32);
        m = (uint32_t)c;
    }
    // reached vertices and their out-edges
    unsigned long long rn = 0, rm = 0;
    for (int64_t v = gt; v < a.V; v += gn) {
        uint32_t c = 0;
        for (int32_t i = 0; i < a.nsrc; i++) c += __ldcg(&a.dist[(uint32_t)i * (uint32_t)a.V + (uint32_t)v]) < kMedusaMax;
        rn += c;
        if (c) rm += (unsigned long long)c * (uint32_t)(__ldg(&a.row[v + 1]) - __ldg(&a.row[v]));
    }
    rn = warp_sum(rn);
    rm = warp_sum(rm);
    if (lane == 0) {
        s_n[tid >> 5] = rn;
        s_m[tid >> 5] = rm;
    }
    __syncthreads();
    if (tid == 0) {
        rn = rm = 0;
        for (int w = 0; w < kThreads / 32; w++) {
            rn += s_n[w];
            rm += s_m[w];
        }
        if (rn) {
            atomicAdd(&a.sh->reached, rn);
            atomicAdd(&a.sh->edges, rm);
        }
        __threadfence();
        if (atomicAdd(&a.sh->ticket, 1u) == gridDim.x - 1) {  // the last CTA reports
            a.out->supersteps = supersteps;
            a.out->splits = splits;
            a.out->reached = atomicAdd(&a.sh->reached, 0ull);
            a.out->edges = atomicAdd(&a.sh->edges, 0ull);
            a.out->work = work;
            if (err) a.out->err = err;
        }
    }
}

}  // namespace

void SsspCoopState::ensure(const Graph &g, int32_t nsrc) {
    if (!built) {
        sh.reserve(sizeof(SShared));
        front.reserve(sizeof(unsigned long long));
        srcs.reserve(sizeof(int32_t) * kSsspCoopSources);
        double mean = 0.0;
        bool bad = false;
        sssp_weight_stats(g, &mean, &bad);
        mean_w = (float)mean;
        weights_ok = !bad;
        built = true;
    }
    if (nsrc <= room) return;
    const size_t pairs = (size_t)nsrc * (size_t)g.V, tiles = (size_t)nsrc * (size_t)g.E / kSsspCoopTile + 2;
    const size_t W = ((pairs + 31) / 32 + 3) & ~(size_t)3;
    for (int i = 0; i < 2; i++) {
        claim[i].reserve(sizeof(uint32_t) * W);
        q[i].reserve(sizeof(uint2) * pairs);
        qv[i].reserve(sizeof(int32_t) * pairs);
        if (nsrc > 1) qs[i].reserve(pairs);
        tf[i].reserve(sizeof(int32_t) * tiles);
    }
    far.reserve(sizeof(uint32_t) * W);
    room = nsrc;
}

int32_t sssp_coop_sources(const Graph &g) { return pairs_sources(g.V, g.E); }

bool sssp_coop_applies(const Context &ctx, const Graph &g, SsspCoopState &st, int32_t nsrc) {
    // the loop graph's and the asynchronous kernel's own parameters ask for them
    for (int t : {MB_TUNE_SSSP_BM_PUSH_MIN, MB_TUNE_PUSH_BLOCKS_PER_SM, MB_TUNE_VERTEX_BLOCKS_PER_SM,
                  MB_TUNE_TAIL_EDGES, MB_TUNE_BULK_STAGE, MB_TUNE_SMALL_PUSH_EDGES, MB_TUNE_SSSP_ASYNC,
                  MB_TUNE_ASYNC_DELTA, MB_TUNE_ASYNC_BLOCKS_PER_SM, MB_TUNE_ASYNC_BELOW})
        if (ctx.tunable[t] >= 0) return false;
    if (ctx.schedule_policy != MB_POLICY_FIXED || !ctx.use_graphs || ctx.tracing || ctx.persist || !ctx.tail ||
        ctx.max_step >= 0 || ctx.sssp_delta != 0.f)
        return false;
    const bool small = sssp_small(g);
    if (nsrc == 1 && !small && async_by_default(g, false)) return false;  // hub-free graphs: the asynchronous kernel
    const bool skewed = g.max_outdeg > g.E / 1024;
    // On the largest skewed graphs a few supersteps hold nearly all edges, which
    // the loop's push and its asynchronous tail take faster, and buckets save
    // nothing (ms, loop / here with buckets / without: R-MAT 2^24 / 2^28 5.7-5.9 /
    // 6.1-7.0 / 7.5; 2^24 / 2^27 4.7 / 4.6 / 5.4; 2^23 / 2^27 4.0 / 3.8 / 4.2).
    if (nsrc == 1 && skewed && g.E > ((int64_t)1 << 27)) return false;
    if (nsrc > 1) {
        if (ctx.tunable[MB_TUNE_MSS_DELTA] >= 0) return false;  // the lines' buckets
        // On a graph with a huge hub most sources' frontiers meet in a few
        // supersteps, and a line of 32 distances per edge is the cheaper form
        // once there is enough of them: from 2^22 edges, or 2^25 of a run's sources
        // together, on (ms, lines / pairs: skewed R-MAT 2^20 / 2^24 x 16 sources 7.0 /
        // 8.8-9.9, 2^17 / 2^21 x 16 1.36 / 1.80, x 4 0.85 / 0.34, 2^16 / 2^20 x 32 1.05 / 1.40,
        // x 16 0.99 / 0.69, 2^19 / 2^21 x 32 1.88 / 2.24; a star of 2^20 x 32 0.78 / 1.56, x 8
        // 0.72 / 0.35).
        const int64_t run = g.E * std::min(nsrc, kSsspCoopSources);  // out-edges of a run
        if (skewed && !small && (g.E >= (1 << 22) || run >= (1 << 25))) return false;
    }
    st.ensure(g, 1);
    return st.weights_ok;
}

bool run_sssp_coop(Context &ctx, Graph &g, SsspCoopState &st, const int32_t *sources, int32_t nsrc, float *dist,
                   mb_stats *stats, const EmitFn *after, SsspRest *rest) {
    static_assert(sizeof(SsspCoopOut) <= Context::kSmallBytes - Context::kCtrlOff, "readback too small");
    cudaStream_t s = ctx.stream;
    volatile SsspCoopOut *out = (volatile SsspCoopOut *)ctx.ctrl_readback();
    out->err = 0;
    out->handed = 0;
    st.ensure(g, nsrc);
    const bool multi = nsrc > 1;
    SArgs a{};
    a.V = g.V;
    a.W = ((((int64_t)g.V * nsrc + 31) / 32) + 3) & ~3ll;
    a.nsrc = nsrc;
    a.sources = st.srcs.as<int32_t>();
    a.front = st.front.as<unsigned long long>();
    a.row = g.row.as<int32_t>();
    a.col = g.col.as<int32_t>();
    a.wt = g.wt.as<float>();
    a.dist = dist;
    for (int i = 0; i < 2; i++) {
        a.claim[i] = st.claim[i].as<uint32_t>();
        a.q[i] = st.q[i].as<uint2>();
        a.qv[i] = st.qv[i].as<int32_t>();
        a.qs[i] = st.qs[i].as<uint8_t>();
        a.tf[i] = st.tf[i].as<int32_t>();
    }
    a.far = st.far.as<uint32_t>();
    a.sh = st.sh.as<SShared>();
    a.out = (SsspCoopOut *)ctx.ctrl_readback();
    a.source = sources[0];
    a.cap = step_cap(ctx, ((int64_t)g.V * 4 + 16) * nsrc);
    a.delta = multi ? pairs_width(g, nsrc) * st.mean_w : single_width(g) * st.mean_w;
    a.polls = ctx.tunable[MB_TUNE_WAIT_POLLS] >= 0 ? (long)ctx.tunable[MB_TUNE_WAIT_POLLS] : kBarrierSpins;
    // a caller's step cap counts supersteps, which the asynchronous kernel has none of
    a.hand = rest && ctx.tunable[MB_TUNE_STEP_CAP] < 0;
    int per_sm = 0;
    const void *kernel = multi ? (const void *)k_sssp_coop<true> : (const void *)k_sssp_coop<false>;
    MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0));
    if (per_sm < 1) fail(MB_ERR_UNSUPPORTED, "cooperative SSSP kernel does not fit on an SM");
    // no more CTAs than tiles: fewer arrive at the barriers of small graphs
    const int grid = (int)std::min<int64_t>(ctx.num_sms * std::min(per_sm, kCtas), std::max<int64_t>(g.E * nsrc / kTileE, 16));
    const cudaEvent_t e0 = ctx.event(0), e1 = ctx.event(1);
    if (multi)
        MB_CUDA(cudaMemcpyAsync(st.srcs.p, sources, sizeof(int32_t) * (size_t)nsrc, cudaMemcpyHostToDevice, s));
    MB_CUDA(cudaEventRecord(e0, s));
    MB_CUDA(cudaMemsetAsync(st.sh.p, 0, sizeof(SShared), s));
    void *params[] = {&a};
    MB_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kThreads), params, 0, s));
    MB_CUDA(cudaEventRecord(e1, s));
    if (after) (*after)(s);
    MB_CUDA(cudaStreamSynchronize(s));
    float ms = 0;
    MB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (out->err & ERR_BARRIER) fail(MB_ERR_TIMEOUT, "sssp: a grid barrier timed out");
    if (out->err & ERR_STEP_CAP) fail(MB_ERR_TIMEOUT, "sssp: superstep cap reached");
    if (stats) {
        *stats = mb_stats{};
        stats->supersteps = out->supersteps + out->splits;
        stats->edges_traversed = (int64_t)out->edges;
        stats->vertices_reached = (int64_t)out->reached;
        stats->device_ms = ms;
        stats->schedule_count[MB_SCHED_PUSH_EDGE_QUEUE] = out->supersteps;
        stats->kernel_launches = 1;
        stats->edges_scanned = (int64_t)out->work;
    }
    if (!out->handed) return false;
    *rest = SsspRest{dist, a.qv[out->cur], out->n, a.far, out->T};
    if (stats) stats->edges_traversed = stats->vertices_reached = 0;  // counted at the end
    return true;
}

}  // namespace mb
