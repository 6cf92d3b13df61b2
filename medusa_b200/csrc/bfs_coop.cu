// bfs_coop.cu -- a whole BFS in one launch, under the fixed rule.
//
// The loop graph (bfs.cu, loopgraph.cuh) pays 12-17 us per superstep: the
// select kernel, the conditional nodes and one or two launches, however small
// the frontier is.  Here the supersteps follow one another inside one kernel:
//   k_bfs_small: one CTA, the frontier queues and the visited bits in shared
//     memory, __syncthreads between supersteps.  Graphs of at most
//     kBfsSmallV vertices and kBfsSmallE edges (push only: one CTA relaxes
//     about an edge per clock, so larger graphs are faster on the whole GPU),
//     0.75 us per superstep; several sources take a CTA each (ms, 32 sources,
//     the batched kernels / here: 10^4 vertices in a line 220 / 6.7, 100 x 100 grid
//     3.8 / 0.22, mild R-MAT 10^4 / 6.5 10^4 0.29 / 0.09, 10^3 / 4 10^3 0.28 / 0.02);
//   k_bfs_coop: one cooperative grid, one grid barrier per superstep.  Every
//     CTA reads the superstep's counters after the barrier and takes the same
//     decision, so no thread decides for the others between two barriers.
// The supersteps, their directions and their counts are those of the loop
// graph under the fixed rule (engine.cuh, fixed_rule).  Two things differ.
// A pull needs no frontier bitmap: an unvisited vertex with any visited
// in-neighbour has one on the frontier (else it would have been reached
// before), so it tests the visited bits as they were before the superstep,
// and writes the new ones to a second bitmap.  The frontier after a pull,
// when a push follows, is what the two bitmaps differ in.  And queue entries
// hold a vertex's first edge, not its number: a push loads no offsets for its
// tiles.  Levels go straight to the caller's device array; vertices not
// reached get -1 at the end instead of a fill before.
// Long runs of small frontiers go on in a second launch, of the kernel whose
// CTA 0 runs them alone (coop_solo, bfs_coop_dev.cuh).
// Measured (calls): R-MAT 2^10 / 2^13 161 -> 41 us; 2^24 / 2^28 596 -> 453 us
// (a small superstep 6-7 us; the large ones push 57 G edges/s and pull at the
// latency of their first list entries); first calls 5.9 -> 0.6 ms, for there is
// no graph to instantiate.
#include "bfs_coop_dev.cuh"

namespace mb {
namespace {

constexpr int kSmallThreads = 1024;
constexpr int kSmallU = 4;  // edges per thread in flight
constexpr size_t kSmallSmem = 220 << 10;
constexpr int kSmallShift = 17;
constexpr uint32_t kSmallMask = (1u << kSmallShift) - 1u;
static_assert(kBfsSmallE <= kSmallMask && kBfsSmallV < (1 << (32 - kSmallShift)), "counts share a word");

// ---- one CTA ----------------------------------------------------------------------

struct SmallArgs {
    int32_t V, E, W, cap;
    const int32_t *row, *col;
    int32_t *level;
    BfsCoopOut *out;  // host memory, one per source
    int32_t sources[kBfsSmallSources];
};

// Shared memory: the visited bits, the levels, two queues, and with kStaged
// the graph itself (offsets and columns, read once): a superstep then waits
// for no memory outside the SM.
__host__ __device__ inline size_t small_words(int32_t V, int64_t E, bool staged) {
    const size_t v4 = ((size_t)V + 3) & ~(size_t)3, w4 = ((size_t)((V + 31) / 32) + 3) & ~(size_t)3;
    return w4 + 5 * v4 + (staged ? v4 + 4 + (size_t)E : 0);
}
template <bool kStaged>
__global__ void __launch_bounds__(kSmallThreads, 1) k_bfs_small(const __grid_constant__ SmallArgs a) {
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t v4 = ((uint32_t)a.V + 3u) & ~3u;
    uint32_t *vis = smem;  // W words
    int32_t *level = reinterpret_cast<int32_t *>(smem + (((uint32_t)a.W + 3u) & ~3u));
    uint2 *q0 = reinterpret_cast<uint2 *>(level + v4);
    uint2 *q1 = q0 + v4;
    int32_t *srow = reinterpret_cast<int32_t *>(q1 + v4), *scol = srow + v4 + 4;
    // queued vertices << kSmallShift | their out-edges; a superstep fills the
    // slot after its own, which the one before cleared, so one barrier is enough
    __shared__ uint32_t s_q[3];
    __shared__ uint32_t s_reached;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int32_t source = a.sources[blockIdx.x];
    const int32_t rs0 = __ldg(&a.row[source]), deg0 = __ldg(&a.row[source + 1]) - rs0;
    if (kStaged) {
        for (int32_t i = tid; i <= a.V; i += kSmallThreads) srow[i] = __ldg(&a.row[i]);
#pragma unroll 8
        for (int32_t i = tid; i < a.E; i += kSmallThreads) scol[i] = __ldg(&a.col[i]);
    }
    const int32_t *row = kStaged ? srow : a.row, *col = kStaged ? scol : a.col;
    for (int i = tid; i < a.W; i += kSmallThreads) vis[i] = i == (source >> 5) ? 1u << (source & 31) : 0u;
    for (int32_t v = tid; v < a.V; v += kSmallThreads) level[v] = v == source ? 0 : -1;
    if (tid == 0) {
        s_reached = 0;
        q0[0] = make_uint2((uint32_t)rs0, 0u);
        s_q[0] = deg0 > 0 ? (1u << kSmallShift) + (uint32_t)deg0 : 0u;
        s_q[1] = s_q[2] = 0u;
    }
    __syncthreads();
    int32_t step = 0, err = 0;
    int slot = 0, next = 1;
    unsigned long long edges = 0;  // of every vertex queued, so of every one reached
    for (;;) {
        const uint2 *q = step & 1 ? q1 : q0;
        uint2 *qn = step & 1 ? q0 : q1;
        const uint32_t c = s_q[slot], n = c >> kSmallShift, m = c & kSmallMask;
        if (n == 0) break;
        if (step >= a.cap) {
            err = ERR_STEP_CAP;
            break;
        }
        uint32_t *ctr = &s_q[next];
        const int after = next == 2 ? 0 : next + 1;
        if (tid == 0) s_q[after] = 0u;
        // a warp without edges goes to the barrier: 32 idle warps took 1700 clocks
        for (uint32_t b = 0; b + (uint32_t)wid * 32u < m; b += kSmallThreads * kSmallU) {
            int32_t v[kSmallU], rs[kSmallU], re[kSmallU];
            bool own[kSmallU];
#pragma unroll
            for (int r = 0; r < kSmallU; r++) {
                const uint32_t e = b + r * kSmallThreads + tid;
                v[r] = -1;
                if (e < m) {
                    uint32_t lo = 0, hi = n;  // q[lo].y <= e < q[hi].y
                    while (hi - lo > 1) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (q[mid].y <= e) lo = mid; else hi = mid;
                    }
                    v[r] = col[q[lo].x + (e - q[lo].y)];
                }
            }
#pragma unroll
            for (int r = 0; r < kSmallU; r++) {
                own[r] = false;
                rs[r] = re[r] = 0;
                if (v[r] >= 0) {
                    const uint32_t bit = 1u << (v[r] & 31);
                    if (!(vis[v[r] >> 5] & bit) && !(atomicOr(&vis[v[r] >> 5], bit) & bit)) {
                        own[r] = true;
                        rs[r] = row[v[r]];
                        re[r] = row[v[r] + 1];
                        level[v[r]] = step + 1;
                    }
                }
            }
            // one scan and one atomic for the warp's finds, counts and
            // out-edges in one word
            uint32_t mine = 0;
#pragma unroll
            for (int r = 0; r < kSmallU; r++)
                if (own[r] && re[r] > rs[r]) mine += (1u << kSmallShift) + (uint32_t)(re[r] - rs[r]);
            const uint32_t incl = warp_incl_scan_u32(mine);
            uint32_t base = 0;
            if (lane == 31 && incl) base = atomicAdd(ctr, incl);
            base = __shfl_sync(0xffffffffu, base, 31) + incl - mine;
#pragma unroll
            for (int r = 0; r < kSmallU; r++)
                if (own[r] && re[r] > rs[r]) {
                    qn[base >> kSmallShift] = make_uint2((uint32_t)rs[r], base & kSmallMask);
                    base += (1u << kSmallShift) + (uint32_t)(re[r] - rs[r]);
                }
        }
        edges += m;
        step++;
        __syncthreads();
        slot = next;
        next = after;
    }
    uint32_t reached = 0;
    int32_t *out = a.level + (size_t)blockIdx.x * (size_t)a.V;
    for (int i = tid; i < a.W; i += kSmallThreads) reached += __popc(vis[i]);
    reached = warp_sum(reached);
    if (lane == 0 && reached) atomicAdd(&s_reached, reached);
    for (int32_t v = tid; v < a.V; v += kSmallThreads) out[v] = level[v];
    __syncthreads();
    if (tid == 0) {
        BfsCoopOut &o = a.out[blockIdx.x];
        o.supersteps = step;
        o.err = err;
        o.reached = s_reached;
        o.edges = edges;
    }
}

// kSolo: the rest of a run that the kernel without left (CoopResume).
template <bool kSolo>
__global__ void __launch_bounds__(kCoopThreads, kBfsCoopCtas) k_bfs_coop(CoopArgs a) {
    __shared__ CoopSmem sm;
    uint32_t barriers = 0;
    if (kSolo) {
        if (threadIdx.x == 0) sm.nout = 0;
        __syncthreads();
        coop_bfs<true>(a, sm, barriers, 0u, 0ull, &a.sh->resume);
        return;
    }
    const int64_t gt = (int64_t)blockIdx.x * kCoopThreads + threadIdx.x, gn = (int64_t)gridDim.x * kCoopThreads;
    const int32_t rs0 = __ldg(&a.row[a.source]), deg0 = __ldg(&a.row[a.source + 1]) - rs0;
    for (int64_t w = gt; w < a.W; w += gn) a.vis[0][w] = w == (a.source >> 5) ? 1u << (a.source & 31) : 0u;
    for (int64_t t = gt; t * kCoopTile < deg0; t += gn) a.tf[0][t] = 0;
    if (gt == 0) {
        a.q[0][0] = make_uint2((uint32_t)rs0, 0u);
        a.level[a.source] = 0;
    }
    if (threadIdx.x == 0) sm.nout = 0;
    if (!coop_sync(a, ++barriers)) return;
    coop_bfs<false>(a, sm, barriers, deg0 > 0 ? 1u : 0u, (uint32_t)deg0, nullptr);
}

}  // namespace

void BfsCoopState::ensure(const Graph &g) {
    if (built) return;
    const size_t tiles = (size_t)(g.E / kBfsCoopTile) + 2, W = ((size_t)g.V + 31) / 32;
    for (int i = 0; i < 2; i++) {
        vis[i].reserve(sizeof(uint32_t) * W);
        q[i].reserve(sizeof(uint2) * (size_t)g.V);
        tf[i].reserve(sizeof(int32_t) * tiles);
    }
    sh.reserve(sizeof(CoopShared));
    built = true;
}

bool bfs_coop_applies(const Context &ctx) {
    // the loop graph's own parameters and its other ways to run ask for the loop
    for (int t : {MB_TUNE_PUSH_BLOCKS_PER_SM, MB_TUNE_VERTEX_BLOCKS_PER_SM, MB_TUNE_TAIL_EDGES,
                  MB_TUNE_SMALL_PUSH_EDGES})
        if (ctx.tunable[t] >= 0) return false;
    return ctx.schedule_policy == MB_POLICY_FIXED && ctx.use_graphs && !ctx.tracing && !ctx.persist && ctx.tail &&
           ctx.max_step < 0;
}

void run_bfs_small(Context &ctx, Graph &g, const int32_t *sources, int32_t nsrc, int32_t *levels, mb_stats *stats,
                   const EmitFn *after) {
    static_assert(sizeof(BfsCoopOut) * kBfsSmallSources <= Context::kSmallBytes - Context::kCtrlOff,
                  "readback too small");
    cudaStream_t s = ctx.stream;
    BfsCoopOut *out = (BfsCoopOut *)ctx.ctrl_readback();
    SmallArgs a{};
    a.V = g.V;
    a.E = (int32_t)g.E;
    a.W = (g.V + 31) / 32;
    a.cap = step_cap(ctx, (int64_t)g.V + 4);
    a.row = g.row.as<int32_t>();
    a.col = g.col.as<int32_t>();
    a.level = levels;
    a.out = out;
    for (int32_t i = 0; i < nsrc; i++) a.sources[i] = sources[i];
    const bool staged = small_words(g.V, g.E, true) * 4 <= kSmallSmem;
    const size_t smem = small_words(g.V, g.E, staged) * 4;
    const void *fn = staged ? (const void *)k_bfs_small<true> : (const void *)k_bfs_small<false>;
    MB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
    const cudaEvent_t e0 = ctx.event(0), e1 = ctx.event(1);
    MB_CUDA(cudaEventRecord(e0, s));
    void *params[] = {&a};
    MB_CUDA(cudaLaunchKernel(fn, dim3(nsrc), dim3(kSmallThreads), params, smem, s));
    MB_CUDA(cudaEventRecord(e1, s));
    if (after) (*after)(s);
    MB_CUDA(cudaStreamSynchronize(s));
    float ms = 0;
    MB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    mb_stats total{};
    for (int32_t i = 0; i < nsrc; i++) {
        const BfsCoopOut &o = out[i];
        if (o.err & ERR_STEP_CAP) fail(MB_ERR_TIMEOUT, "bfs: superstep cap reached");
        total.supersteps = std::max(total.supersteps, o.supersteps);
        total.edges_traversed += (int64_t)o.edges;
        total.vertices_reached += (int64_t)o.reached;
    }
    total.device_ms = ms;
    total.schedule_count[MB_SCHED_PUSH_EDGE_QUEUE] = total.supersteps;
    total.kernel_launches = 1;
    total.edges_scanned = total.edges_traversed;  // each once
    if (stats) *stats = total;
}

void run_bfs_coop(Context &ctx, Graph &g, BfsCoopState &st, int32_t source, int32_t *level, mb_stats *stats,
                  const EmitFn *after) {
    static_assert(sizeof(BfsCoopOut) <= Context::kSmallBytes - Context::kCtrlOff, "readback too small");
    cudaStream_t s = ctx.stream;
    volatile BfsCoopOut *out = (volatile BfsCoopOut *)ctx.ctrl_readback();
    out->err = 0;
    out->handed = 0;
    CoopArgs a{};
    a.V = g.V;
    a.E = g.E;
    a.W = ((int64_t)g.V + 31) / 32;
    a.row = g.row.as<int32_t>();
    a.col = g.col.as<int32_t>();
    a.rrow = g.rrow.as<int32_t>();
    a.rcol = g.rcol.as<int32_t>();
    a.level = level;
    a.out = (BfsCoopOut *)ctx.ctrl_readback();
    a.source = source;
    a.alpha = ctx.tunable[MB_TUNE_BFS_ALPHA] >= 0 ? (int32_t)ctx.tunable[MB_TUNE_BFS_ALPHA] : 15;
    a.beta = ctx.tunable[MB_TUNE_BFS_BETA] > 0 ? (int32_t)ctx.tunable[MB_TUNE_BFS_BETA] : 20;
    a.gamma = ctx.tunable[MB_TUNE_BFS_GAMMA] >= 0 ? (int32_t)ctx.tunable[MB_TUNE_BFS_GAMMA] : kBfsGammaDefault;
    a.cap = step_cap(ctx, (int64_t)g.V + 4);
    a.polls = ctx.tunable[MB_TUNE_WAIT_POLLS] >= 0 ? (long)ctx.tunable[MB_TUNE_WAIT_POLLS] : kBarrierSpins;
    const cudaEvent_t e0 = ctx.event(0), e1 = ctx.event(1);
    st.ensure(g);
    for (int i = 0; i < 2; i++) {
        a.vis[i] = st.vis[i].as<uint32_t>();
        a.q[i] = st.q[i].as<uint2>();
        a.tf[i] = st.tf[i].as<int32_t>();
    }
    a.sh = st.sh.as<CoopShared>();
    auto launch = [&](const void *kernel) {
        int per_sm = 0;
        MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kCoopThreads, 0));
        if (per_sm < 1) fail(MB_ERR_UNSUPPORTED, "cooperative BFS kernel does not fit on an SM");
        // no more CTAs than tiles: fewer arrive at the barriers of small graphs
        const int grid = (int)std::min<int64_t>(ctx.num_sms * std::min(per_sm, kBfsCoopCtas),
                                                std::max<int64_t>(g.E / kCoopTile, 16));
        MB_CUDA(cudaMemsetAsync(st.sh.p, 0, offsetof(CoopShared, resume), s));
        void *params[] = {&a};
        MB_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kCoopThreads), params, 0, s));
        MB_CUDA(cudaEventRecord(e1, s));
        if (after) (*after)(s);
        MB_CUDA(cudaStreamSynchronize(s));
    };
    MB_CUDA(cudaEventRecord(e0, s));
    launch((const void *)k_bfs_coop<false>);
    const bool handed = !out->err && out->handed;
    if (handed) launch((const void *)k_bfs_coop<true>);
    float ms = 0;
    MB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (out->err & ERR_BARRIER) fail(MB_ERR_TIMEOUT, "bfs: a grid barrier timed out");
    if (out->err & ERR_STEP_CAP) fail(MB_ERR_TIMEOUT, "bfs: superstep cap reached");
    if (stats) {
        *stats = mb_stats{};
        stats->supersteps = out->supersteps;
        stats->edges_traversed = (int64_t)out->edges;
        stats->vertices_reached = (int64_t)out->reached;
        stats->device_ms = ms;
        stats->schedule_count[MB_SCHED_PUSH_EDGE_QUEUE] = out->pushes;
        stats->schedule_count[MB_SCHED_PULL_THREAD] = out->pulls;
        stats->kernel_launches = 1 + handed;
        stats->edges_scanned = (int64_t)out->work;
    }
}

}  // namespace mb
