// sssp_small.cu -- SSSP on a graph that fits one CTA, under the fixed rule.
//
// The queues, the distances and (kStaged) the graph itself live in shared
// memory and one __syncthreads stands between two supersteps: 1.2 us each,
// where one of the cooperative grid costs 6 us and a phase of the asynchronous
// kernel 27.  The rules are sssp_coop.cu's: a near queue, a claim bit per
// vertex and superstep, a far bitmap that a split empties below the next
// threshold.  One CTA per source.  Bound by the barrier and its chain of
// shared-memory accesses where the frontiers are small, by the CTA's 2 clocks
// per relaxed edge where they are large: hence kSsspSmallE.
// Measured (ms, the kernels these graphs had before / here; 1 and 32 sources):
// 10^4 vertices in a line 18.8 / 8.4 and 127 / 13.5, 100 x 100 grid 0.73 / 0.35 and
// 2.6 / 0.48, uniform 10^3 / 4 10^3 0.144 / 0.036 and 0.21 / 0.04, mild R-MAT
// 10^3 / 2 10^4 0.084 / 0.05 and 0.18 / 0.06.  With 6.5 10^4 edges: uniform 10^4
// 0.176 / 0.198, skewed R-MAT 3200 0.096 / 0.119 -- left where they were.
#include "sssp.cuh"
#include "sssp_coop.cuh"

namespace mb {
namespace {

constexpr int kThreads = 1024;
constexpr int kItems = 4;  // consecutive edges of a thread, at most
constexpr size_t kSmem = 220 << 10;
constexpr int kShift = 17;
constexpr uint32_t kMask = (1u << kShift) - 1u;
static_assert(kSsspSmallE <= kMask && kSsspSmallV < (1 << (32 - kShift)), "counts share a word");
constexpr uint32_t kInf = 0x7f800000u;

// Bucket width in mean weights, 1 / 2 / 5 / none: 100 x 100 grid 0.59 / 0.46 / 0.35 / 0.39 ms,
// 100 x 100 torus 0.50 / 0.39 / 0.31 / 0.37; mild R-MAT 3000 / 3 10^4 0.070 / 0.084 / 0.096 /
// 0.095, uniform 3000 / 3 10^4 0.073 / 0.071 / 0.105 / 0.108.  Wide buckets for road-like
// graphs (hub-free, at most 4 out-edges per vertex).
inline float small_width(const Graph &g) {
    return g.max_outdeg <= 64 && g.E <= 4 * (int64_t)g.V ? 5.f : 1.5f;
}

struct SmallArgs {
    int32_t V, E, W;
    const int32_t *row, *col;
    const float *wt;
    float *dist;
    SsspCoopOut *out;  // host memory, one per source
    int32_t cap;
    float delta;  // 0: no buckets
    int32_t sources[kSsspSmallSources];
};

__host__ __device__ inline size_t small_words(int32_t V, int64_t E, bool staged) {
    const size_t v4 = ((size_t)V + 3) & ~(size_t)3, w4 = ((size_t)((V + 31) / 32) + 3) & ~(size_t)3;
    return 3 * w4 + 5 * v4 + (staged ? v4 + 4 + 2 * (size_t)E : 0);
}

template <bool kStaged>
__global__ void __launch_bounds__(kThreads, 1) k_sssp_small(const __grid_constant__ SmallArgs a) {
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t v4 = ((uint32_t)a.V + 3u) & ~3u, w4 = ((uint32_t)a.W + 3u) & ~3u;
    uint32_t *claim0 = smem, *claim1 = claim0 + w4, *farbm = claim1 + w4;
    volatile uint32_t *dist = farbm + w4;  // float bits: not negative, so they order as integers
    uint2 *q0 = reinterpret_cast<uint2 *>(farbm + w4 + v4);  // {vertex, out-edges queued before it}
    uint2 *q1 = q0 + v4;
    int32_t *srow = reinterpret_cast<int32_t *>(q1 + v4), *scol = srow + v4 + 4;
    float *swt = reinterpret_cast<float *>(scol + a.E);
    // one slot per superstep in turn: it fills the slot after its own, which the
    // one before cleared, so one barrier a superstep is enough
    __shared__ uint32_t s_q[3];  // queued vertices << kShift | their out-edges
    __shared__ uint32_t s_far[3], s_min[3], s_reached, s_edges;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int32_t source = a.sources[blockIdx.x];
    const int32_t deg0 = __ldg(&a.row[source + 1]) - __ldg(&a.row[source]);
    if (kStaged) {
        for (int32_t i = tid; i <= a.V; i += kThreads) srow[i] = __ldg(&a.row[i]);
#pragma unroll 4
        for (int32_t i = tid; i < a.E; i += kThreads) {
            scol[i] = __ldg(&a.col[i]);
            swt[i] = __ldg(&a.wt[i]);
        }
    }
    const int32_t *row = kStaged ? srow : a.row, *col = kStaged ? scol : a.col;
    const float *wt = kStaged ? swt : a.wt;
    for (int i = tid; i < a.W; i += kThreads) claim0[i] = claim1[i] = farbm[i] = 0u;
    for (int32_t v = tid; v < a.V; v += kThreads) dist[v] = v == source ? 0u : __float_as_uint(kMedusaMax);
    if (tid == 0) {
        s_reached = s_edges = 0u;
        for (int i = 0; i < 3; i++) {
            s_q[i] = s_far[i] = 0u;
            s_min[i] = kInf;
        }
        q0[0] = make_uint2((uint32_t)source, 0u);
        s_q[0] = deg0 > 0 ? (1u << kShift) + (uint32_t)deg0 : 0u;
    }
    __syncthreads();
    int32_t supersteps = 0, splits = 0, err = 0;
    unsigned long long work = 0;
    const float inf = __uint_as_float(kInf);
    float T = a.delta > 0.f ? a.delta : inf, fmin = inf;
    bool far = false;
    int slot = 0, next = 1;
    for (int32_t it = 0;; it++) {
        const uint2 *q = it & 1 ? q1 : q0;
        uint2 *qn = it & 1 ? q0 : q1;
        uint32_t *claim = it & 1 ? claim1 : claim0, *old = it & 1 ? claim0 : claim1;
        uint32_t *ctr = &s_q[next];
        const int after = next == 2 ? 0 : next + 1;
        const uint32_t c = s_q[slot], n = c >> kShift, m = c & kMask;
        if (n == 0 && !far) break;
        if (it >= a.cap) {
            err = ERR_STEP_CAP;
            break;
        }
        // the claims of the superstep before end: this one reads each queued
        // distance now, and a later drop claims again, in the other bitmap
        for (int i = tid; i < a.W; i += kThreads) old[i] = 0u;
        if (tid == 0) {
            s_q[after] = s_far[after] = 0u;
            s_min[after] = kInf;
        }
        // a warp's vertices -> the next queue, one scan and one atomic
        auto append = [&](uint32_t mine) {
            const uint32_t incl = warp_incl_scan_u32(mine);
            uint32_t base = 0;
            if (lane == 31 && incl) base = atomicAdd(ctr, incl);
            return __shfl_sync(0xffffffffu, base, 31) + incl - mine;
        };
        if (n == 0) {  // next bucket
            const float T0 = T;
            T = T0 + a.delta;
            if (fmin < inf) T = fmaxf(T, fmin + a.delta);
            if (!(T > T0)) T = __uint_as_float(__float_as_uint(T0) + 1u);
            if (fmin < inf && !(T > fmin)) T = __uint_as_float(__float_as_uint(fmin) + 1u);
            uint32_t kept = kInf;
            for (int w = wid; w < a.W; w += kThreads / 32) {
                const uint32_t x = farbm[w];
                if (x == 0u) continue;
                const int32_t v = w * 32 + lane;
                const bool has = (x >> lane) & 1u;
                const float d = has ? __uint_as_float(dist[v]) : inf;
                const bool stay = has && !(d < T), take = has && d < T && d >= T0;
                if (stay) kept = min(kept, __float_as_uint(d));
                const uint32_t keep = __ballot_sync(0xffffffffu, stay);
                if (lane == 0) farbm[w] = keep;
                const uint32_t dg = take ? (uint32_t)(row[v + 1] - row[v]) : 0u;
                const uint32_t base = append(dg ? (1u << kShift) + dg : 0u);
                if (dg) qn[base >> kShift] = make_uint2((uint32_t)v, base & kMask);
            }
            kept = __reduce_min_sync(0xffffffffu, kept);
            if (lane == 0 && kept < kInf) atomicMin(&s_min[next], kept);
            splits++;
        } else {
            // few edges: one each; many: consecutive ones, one search for all
            const uint32_t per = min((m + kThreads - 1) / kThreads, (uint32_t)kItems);
            bool put_off = false;
            // a warp without edges goes to the barrier: 32 idle warps took 1700 clocks
            for (uint32_t b = 0; b + (uint32_t)wid * 32u * per < m; b += kThreads * per) {
                const uint32_t e0 = b + tid * per;
                int32_t v[kItems];
                uint32_t nd[kItems] = {}, mine = 0, dg[kItems];
                uint32_t lo = 0;
                if (e0 < m) {
                    uint32_t hi = n;  // q[lo].y <= e0 < q[hi].y
                    while (hi - lo > 1) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (q[mid].y <= e0) lo = mid; else hi = mid;
                    }
                }
                uint2 u = q[lo];
                uint32_t end = lo + 1 < n ? q[lo + 1].y : m;
                int32_t at = row[u.x] - (int32_t)u.y;
                float du = __uint_as_float(dist[u.x]);
#pragma unroll
                for (int r = 0; r < kItems; r++) {
                    const uint32_t e = e0 + r;
                    v[r] = -1;
                    if (r < per && e < m) {
                        if (e >= end) {
                            lo++;  // every queued vertex has out-edges
                            u = q[lo];
                            end = lo + 1 < n ? q[lo + 1].y : m;
                            at = row[u.x] - (int32_t)u.y;
                            du = __uint_as_float(dist[u.x]);
                        }
                        v[r] = col[at + (int32_t)e];
                        nd[r] = __float_as_uint(du + wt[at + (int32_t)e]);
                    }
                }
#pragma unroll
                for (int r = 0; r < kItems; r++) {
                    dg[r] = 0u;
                    if (v[r] >= 0 && nd[r] < dist[v[r]] &&
                        nd[r] < atomicMin(const_cast<uint32_t *>(&dist[v[r]]), nd[r])) {
                        const uint32_t bit = 1u << (v[r] & 31);
                        if (__uint_as_float(nd[r]) >= T) {
                            put_off = true;
                            if (!(farbm[v[r] >> 5] & bit)) atomicOr(&farbm[v[r] >> 5], bit);
                        } else if (!(atomicOr(&claim[v[r] >> 5], bit) & bit)) {
                            dg[r] = (uint32_t)(row[v[r] + 1] - row[v[r]]);
                            if (dg[r]) mine += (1u << kShift) + dg[r];
                        }
                    }
                }
                if (!__any_sync(0xffffffffu, mine != 0u)) continue;
                uint32_t base = append(mine);
#pragma unroll
                for (int r = 0; r < kItems; r++)
                    if (dg[r]) {
                        qn[base >> kShift] = make_uint2((uint32_t)v[r], base & kMask);
                        base += (1u << kShift) + dg[r];
                    }
            }
            if (put_off) s_far[next] = 1u;
            work += m;
            supersteps++;
        }
        __syncthreads();
        if (n == 0) {
            fmin = __uint_as_float(s_min[next]);
            far = fmin < inf;
        } else {
            far = far || s_far[next] != 0u;
        }
        slot = next;
        next = after;
    }
    uint32_t rn = 0, rm = 0;
    float *out = a.dist + (size_t)blockIdx.x * (size_t)a.V;
    for (int32_t v = tid; v < a.V; v += kThreads) {
        const float d = __uint_as_float(dist[v]);
        out[v] = d;
        if (d < kMedusaMax) {
            rn++;
            rm += (uint32_t)(row[v + 1] - row[v]);
        }
    }
    rn = warp_sum(rn);
    rm = warp_sum(rm);
    if (lane == 0 && rn) {
        atomicAdd(&s_reached, rn);
        atomicAdd(&s_edges, rm);
    }
    __syncthreads();
    if (tid == 0) {
        SsspCoopOut &o = a.out[blockIdx.x];
        o.supersteps = supersteps;
        o.splits = splits;
        o.reached = s_reached;
        o.edges = s_edges;
        o.work = work;
        o.err = err;
    }
}

}  // namespace

// Without hubs the other side is the asynchronous kernel, slower by more (20^3
// cube, 45600 edges: 0.32 against 0.19 ms).
bool sssp_small(const Graph &g) {
    return g.V <= kSsspSmallV && g.E <= (g.max_outdeg <= 64 ? kSsspSmallE : kSsspSmallHubE);
}

void run_sssp_small(Context &ctx, Graph &g, SsspCoopState &st, const int32_t *sources, int32_t nsrc, float *dist,
                    mb_stats *stats, const EmitFn *after) {
    static_assert(sizeof(SsspCoopOut) * kSsspSmallSources <= Context::kSmallBytes - Context::kCtrlOff,
                  "readback too small");
    cudaStream_t s = ctx.stream;
    SsspCoopOut *out = (SsspCoopOut *)ctx.ctrl_readback();
    SmallArgs a{};
    a.V = g.V;
    a.E = (int32_t)g.E;
    a.W = (g.V + 31) / 32;
    a.row = g.row.as<int32_t>();
    a.col = g.col.as<int32_t>();
    a.wt = g.wt.as<float>();
    a.dist = dist;
    a.out = out;
    a.cap = step_cap(ctx, (int64_t)g.V * 4 + 16);
    a.delta = small_width(g) * st.mean_w;
    for (int32_t i = 0; i < nsrc; i++) a.sources[i] = sources[i];
    const bool staged = small_words(g.V, g.E, true) * 4 <= kSmem;
    const size_t smem = small_words(g.V, g.E, staged) * 4;
    const void *fn = staged ? (const void *)k_sssp_small<true> : (const void *)k_sssp_small<false>;
    MB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    const cudaEvent_t e0 = ctx.event(0), e1 = ctx.event(1);
    MB_CUDA(cudaEventRecord(e0, s));
    void *params[] = {&a};
    MB_CUDA(cudaLaunchKernel(fn, dim3(nsrc), dim3(kThreads), params, smem, s));
    MB_CUDA(cudaEventRecord(e1, s));
    if (after) (*after)(s);
    MB_CUDA(cudaStreamSynchronize(s));
    float ms = 0;
    MB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    mb_stats total{};
    for (int32_t i = 0; i < nsrc; i++) {
        const SsspCoopOut &o = out[i];
        if (o.err & ERR_STEP_CAP) fail(MB_ERR_TIMEOUT, "sssp: superstep cap reached");
        total.supersteps = std::max(total.supersteps, o.supersteps + o.splits);
        total.edges_traversed += (int64_t)o.edges;
        total.vertices_reached += (int64_t)o.reached;
        total.schedule_count[MB_SCHED_PUSH_EDGE_QUEUE] = std::max<decltype(+total.schedule_count[0])>(
            total.schedule_count[MB_SCHED_PUSH_EDGE_QUEUE], o.supersteps);
        total.edges_scanned += (int64_t)o.work;
    }
    total.device_ms = ms;
    total.kernel_launches = 1;
    if (stats) *stats = total;
}

}  // namespace mb
