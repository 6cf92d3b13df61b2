// bfs_coop_dev.cuh -- device code of the one-launch cooperative BFS, shared by
// bfs_coop.cu and the many-graph kernel (multigraph.cu).
#pragma once
#include "bfs_coop.cuh"
#include "coop.cuh"

namespace mb {

constexpr int kCoopThreads = 512;
constexpr int kCoopItems = 2;
constexpr int kCoopTile = kCoopThreads * kCoopItems;  // edges of a tile
static_assert(kCoopTile == kBfsCoopTile, "the tile tables are sized by it");

struct alignas(128) CoopCtr {  // one per superstep in turn, three in all
    unsigned long long q;  // queued vertices << 32 | their out-edges
    uint32_t n, pad;       // a pull's new vertices
    unsigned long long m;  // and their out-edges
};
struct CoopSolo {  // what coop_solo leaves to the grid
    uint32_t n, m, steps, pad;       // the frontier, and the supersteps run
    unsigned long long edges, work;  // of those: out-edges found, edges looked at
};
struct CoopResume {  // where a run stands between two supersteps, the frontier in a queue
    int32_t vb, cur, step, pushes, pulls;
    uint32_t n, prev_n, pad;
    unsigned long long m, edges, work;
    int64_t unvisited;
};
struct CoopShared {  // device memory of a run, zero before each launch up to resume
    CoopCtr ctr[3];
    CoopSolo solo[2];  // in turn
    unsigned long long toq;  // the queue built from a pull's vertices
    unsigned long long reached;
    uint32_t ticket;
    alignas(128) uint32_t bar[2];  // polled: a line of its own
    alignas(128) CoopResume resume;
};

struct CoopArgs {
    int32_t V;
    int64_t E, W;
    const int32_t *row, *col, *rrow, *rcol;
    int32_t *level;
    uint32_t *vis[2];
    uint2 *q[2];     // {first edge, out-edges queued before it}
    int32_t *tf[2];  // first entry of each tile
    CoopShared *sh;
    BfsCoopOut *out;  // host memory
    int32_t source, alpha, beta, gamma, cap;
    long polls;
};

// ---- one cooperative grid -----------------------------------------------------------

__device__ __forceinline__ bool coop_sync(const CoopArgs &a, uint32_t k) {
    return coop_barrier(a.sh->bar, k, a.polls, &a.out->err);
}

struct CoopSmem {
    uint32_t off[kCoopTile + 1];
    int32_t row[kCoopTile + 1];  // first edge less the edges before it
    uint2 out[kCoopTile];        // found vertices: {first edge, out-edges}
    uint32_t nout;
    uint32_t wtot[kCoopThreads / 32];
    unsigned long long base;
};

// The tile's found vertices -> the next queue, one atomic per tile.
__device__ __forceinline__ void coop_flush(CoopSmem &sm, unsigned long long *ctr, uint2 *q, int32_t *tf) {
    __syncthreads();
    const uint32_t n = sm.nout;
    if (n == 0) return;  // the same for every thread
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t i0 = threadIdx.x * kCoopItems;
    uint2 e[kCoopItems];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kCoopItems; k++) {
        e[k] = i0 + k < n ? sm.out[i0 + k] : make_uint2(0u, 0u);
        sum += e[k].y;
    }
    const uint32_t incl = warp_incl_scan_u32(sum);
    if (lane == 31) sm.wtot[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        constexpr int kW = kCoopThreads / 32;
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
    for (int k = 0; k < kCoopItems; k++) {
        if (i0 + k < n) {
            const uint32_t pos = (uint32_t)(base >> 32) + i0 + k, d = e[k].y;
            q[pos] = make_uint2(e[k].x, off);
            const uint32_t t0 = (off + kCoopTile - 1) / kCoopTile, t1 = (off + d - 1) / kCoopTile;
            for (uint32_t t = t0; t <= t1; t++) tf[t] = (int32_t)pos;
            off += d;
        }
    }
}

__device__ __forceinline__ void coop_found(CoopSmem &sm, bool pred, int32_t rs, uint32_t d) {
    const unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (!mask) return;
    const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&sm.nout, (uint32_t)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) sm.out[base + __popc(mask & lanemask_lt())] = make_uint2((uint32_t)rs, d);
}

__device__ __forceinline__ void coop_push(const CoopArgs &a, CoopSmem &sm, const uint2 *q, const int32_t *tf,
                                          uint32_t n, uint32_t m, uint32_t *vis, int32_t lvl, CoopCtr *ctr,
                                          uint2 *qn, int32_t *tfn) {
    const uint32_t tiles = (m + kCoopTile - 1) / kCoopTile;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t c0 = t * kCoopTile, c1 = min(c0 + kCoopTile, m);
        const int32_t i0 = __ldcg(&tf[t]);
        const int32_t i1 = t + 1 < tiles ? __ldcg(&tf[t + 1]) : (int32_t)n - 1;
        const int k = i1 - i0 + 1;
        for (int j = threadIdx.x; j < k; j += kCoopThreads) {
            const uint2 e = __ldcg(&q[i0 + j]);
            sm.off[j] = e.y;
            sm.row[j] = (int32_t)(e.x - e.y);
        }
        __syncthreads();
        int32_t v[kCoopItems];
        {
            const uint32_t e0 = c0 + threadIdx.x * kCoopItems;
            int j = e0 < c1 ? upper_bound_minus1(sm.off, k, e0) : 0;
#pragma unroll
            for (int r = 0; r < kCoopItems; r++) {
                const uint32_t e = e0 + r;
                v[r] = -1;
                if (e < c1) {
                    while (j + 1 < k && sm.off[j + 1] <= e) j++;
                    v[r] = __ldg(&a.col[sm.row[j] + (int32_t)e]);
                }
            }
        }
        // through L1: bits are only ever set, so a stale word costs an atomic
        // that finds the bit set, never a wrong claim (5.2M frontier edges on
        // R-MAT 2^24 / 2^28: 91 us, against 151 reading at L2)
        uint32_t w[kCoopItems];
#pragma unroll
        for (int r = 0; r < kCoopItems; r++) w[r] = v[r] >= 0 ? __ldca(&vis[v[r] >> 5]) : ~0u;
        bool own[kCoopItems];
#pragma unroll
        for (int r = 0; r < kCoopItems; r++) {
            const uint32_t bit = 1u << (v[r] & 31);
            own[r] = !(w[r] & bit) && !(atomicOr(&vis[v[r] >> 5], bit) & bit);
        }
#pragma unroll
        for (int r = 0; r < kCoopItems; r++) {
            int32_t rs = 0, re = 0;
            if (own[r]) {
                rs = __ldg(&a.row[v[r]]);
                re = __ldg(&a.row[v[r] + 1]);
                a.level[v[r]] = lvl;
            }
            coop_found(sm, re > rs, rs, (uint32_t)(re - rs));
        }
        coop_flush(sm, &ctr->q, qn, tfn);
    }
}

// A warp owns a word of the bitmaps; a lane scans kPullCap in-edges of its
// vertex alone, four at a time (their tests do not wait for one another), the
// warp the rest of longer lists.
constexpr int kPullCap = 32;
__device__ __forceinline__ void coop_pull(const CoopArgs &a, const uint32_t *vis, uint32_t *visn, int32_t lvl,
                                          CoopCtr *ctr) {
    __shared__ uint32_t s_n[kCoopThreads / 32];
    __shared__ unsigned long long s_m[kCoopThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t warps = (int64_t)gridDim.x * (kCoopThreads / 32);
    uint32_t cn = 0;
    unsigned long long cm = 0;
    for (int64_t w = (int64_t)blockIdx.x * (kCoopThreads / 32) + wid; w < a.W; w += warps) {
        const uint32_t word = vis[w];
        const int32_t v = (int32_t)(w * 32 + lane);
        const uint32_t todo = ~word & tail_mask(w, a.V);
        if (!todo) {
            if (lane == 0) visn[w] = word;
            continue;
        }
        bool found = false;
        int32_t j = 0, je = 0;
        if ((todo >> lane) & 1u) {
            j = __ldg(&a.rrow[v]);
            je = __ldg(&a.rrow[v + 1]);
            const int32_t jcap = min(je, j + kPullCap);
            // the first alone: where the frontier is large, it mostly is a hit
            if (j < jcap) found = test_bit(vis, __ldg(&a.rcol[j++]));
            while (j < jcap && !found) {
                int32_t u[4];
                const int32_t jb = load4_from(a.rcol, j, jcap, a.E, u);
                uint32_t x[4];
#pragma unroll
                for (int r = 0; r < 4; r++) x[r] = u[r] >= 0 ? vis[u[r] >> 5] : 0u;
#pragma unroll
                for (int r = 0; r < 4; r++) found |= (x[r] >> (u[r] & 31)) & 1u;
                j = min(jb + 4, jcap);
            }
        }
        unsigned pend = __ballot_sync(0xffffffffu, !found && j < je);
        while (pend) {
            const int l = __ffs(pend) - 1;
            pend &= pend - 1;
            const int32_t pj = __shfl_sync(0xffffffffu, j, l), pje = __shfl_sync(0xffffffffu, je, l);
            bool hit = false;
            for (int32_t b = pj; b < pje && !hit; b += 128) {
                uint32_t x[4];
                int32_t u[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int32_t jj = b + 32 * r + lane;
                    u[r] = jj < pje ? __ldg(&a.rcol[jj]) : -1;
                }
#pragma unroll
                for (int r = 0; r < 4; r++) x[r] = u[r] >= 0 ? vis[u[r] >> 5] : 0u;
                bool h = false;
#pragma unroll
                for (int r = 0; r < 4; r++) h |= (x[r] >> (u[r] & 31)) & 1u;
                hit = __any_sync(0xffffffffu, h);
            }
            if (lane == l) found = hit;
        }
        const uint32_t mask = __ballot_sync(0xffffffffu, found);
        if (lane == 0) visn[w] = word | mask;
        if (found) {
            a.level[v] = lvl;
            cn++;
            cm += (uint32_t)(__ldg(&a.row[v + 1]) - __ldg(&a.row[v]));
        }
    }
    cn = warp_sum(cn);
    cm = warp_sum(cm);
    if (lane == 0) {
        s_n[wid] = cn;
        s_m[wid] = cm;
    }
    __syncthreads();
    if (wid == 0) {
        constexpr int kW = kCoopThreads / 32;
        cn = warp_sum(lane < kW ? s_n[lane] : 0u);
        cm = warp_sum(lane < kW ? s_m[lane] : 0ull);
        if (lane == 0 && cn) {
            atomicAdd(&ctr->n, cn);
            atomicAdd(&ctr->m, cm);
        }
    }
}

// The vertices a pull added (now, not before) -> queue: every warp gathers
// them in a buffer of its own and appends full buffers with one atomic (260k
// vertices of 2^24: 28 us; four words a round and one atomic per CTA and round,
// as sssp_coop.cu does on its denser bitmaps: 52).
constexpr int kToqBuf = 64;
__device__ __forceinline__ void coop_toq(const CoopArgs &a, CoopSmem &sm, const uint32_t *now, const uint32_t *before,
                                         unsigned long long *ctr, uint2 *q, int32_t *tf) {
    static_assert(kToqBuf * (kCoopThreads / 32) <= kCoopTile, "the warps' buffers share sm.out");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint2 *buf = sm.out + wid * kToqBuf;
    uint32_t nb = 0;  // warp-uniform, below 32 between two words
    auto flush = [&](uint32_t cnt) {
        __syncwarp();
        const uint2 e = lane < (int)cnt ? buf[lane] : make_uint2(0u, 0u);
        const uint2 rest = lane + cnt < nb ? buf[lane + cnt] : make_uint2(0u, 0u);
        const uint32_t incl = warp_incl_scan_u32(e.y);
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(ctr, ((unsigned long long)cnt << 32) | total);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < (int)cnt) {
            const uint32_t pos = (uint32_t)(base >> 32) + lane, off = (uint32_t)base + incl - e.y;
            q[pos] = make_uint2(e.x, off);
            const uint32_t t0 = (off + kCoopTile - 1) / kCoopTile, t1 = (off + e.y - 1) / kCoopTile;
            for (uint32_t t = t0; t <= t1; t++) tf[t] = (int32_t)pos;
        }
        __syncwarp();
        if (lane + cnt < nb) buf[lane] = rest;
        nb -= cnt;
        __syncwarp();
    };
    const int64_t warps = (int64_t)gridDim.x * (kCoopThreads / 32);
    for (int64_t b = ((int64_t)blockIdx.x * (kCoopThreads / 32) + wid) * 32; b < a.W; b += warps * 32) {
        // a lane loads a word: 32 words per round
        const int64_t wl = b + lane;
        const uint32_t xl = wl < a.W ? (now[wl] & ~before[wl]) : 0u;
        unsigned nz = __ballot_sync(0xffffffffu, xl != 0u);
        while (nz) {
            const int l = __ffs(nz) - 1;
            nz &= nz - 1;
            const uint32_t x = __shfl_sync(0xffffffffu, xl, l);
            int32_t rs = 0, re = 0;
            if ((x >> lane) & 1u) {
                const int32_t v = (int32_t)((b + l) * 32 + lane);
                rs = __ldg(&a.row[v]);
                re = __ldg(&a.row[v + 1]);
            }
            const unsigned in = __ballot_sync(0xffffffffu, re > rs);
            if (re > rs) buf[nb + __popc(in & lanemask_lt())] = make_uint2((uint32_t)rs, (uint32_t)(re - rs));
            nb += __popc(in);
            if (nb >= 32) flush(32);
        }
    }
    if (nb) flush(nb);
    __syncthreads();  // sm.out is the pushes' next
}

// Supersteps of a frontier of at most a tile of out-edges, by this CTA alone:
// a superstep of the grid costs 5 us, nearly all of it the barrier, however
// small the frontier is.  Here __syncthreads stands between two of them, the
// frontier stays in shared memory, and what is left is a chain of two L2 round
// trips and a search.  Until the frontier has more out-edges, the rule asks for
// a pull, nothing is left, or kSoloSteps supersteps have run: the other CTAs
// wait at the barrier meanwhile, and their wait is bounded.
// (Without it graphs of a long diameter with one hub, which the superstep loop
// runs in its own one-CTA kernel, took twice as long as there: ms, loop / grid
// alone / here, a line of 40,000 with a hub 77 / 147 / 27, grid 300 x 300 2.3 /
// 3.0 / 1.95, 2^18 skewed R-MAT with 64 lines of 2000 7.3 / 11.7 / 3.1; 64 lines of
// 10,000 in one batch, teams / grid alone / here, 28 / 53 / 14.5.)
constexpr uint32_t kSoloSteps = 1024;
// Small supersteps of the grid before it: one alone costs 3 us more here than
// there, and a graph of a short diameter has but a few at each end (2^17 / 2^21
// skewed R-MAT 74 us; 84 where one was enough).
constexpr int kSoloAfter = 8;
__device__ __forceinline__ bool coop_pull_next(unsigned long long m, int64_t unvisited, int32_t alpha, int32_t gamma,
                                               int64_t E) {
    return alpha > 0 && (int64_t)m * alpha > unvisited && (gamma == 0 || (int64_t)m * gamma >= E);
}
struct SoloArgs {  // in shared memory: what a call of its own needs, so that it takes no register of its caller
    const int32_t *row, *col;
    int32_t *level, *tf;  // tf, qn: the frontier it leaves
    uint32_t *vis;
    const uint2 *q;
    uint2 *qn;
    CoopSolo *out;
    int64_t E, unvisited;
    int32_t alpha, gamma, cap, step;
    uint32_t n, m;
};
// A call, not inlined: inlined, its registers pushed the grid's pull and push
// into spills.
static __device__ __noinline__ void coop_solo(const SoloArgs &a, CoopSmem &sm) {
    static_assert(sizeof(sm.off) + sizeof(sm.row) >= kCoopTile * sizeof(uint2) &&
                      offsetof(CoopSmem, row) == sizeof(sm.off) && offsetof(CoopSmem, off) == 0,
                  "two frontiers of a tile's vertices");
    uint2 *buf[2] = {reinterpret_cast<uint2 *>(sm.off), sm.out};  // {first edge less off, off}
    // queued vertices << 32 | their out-edges; a superstep fills the slot after
    // its own, which the one before cleared, so one barrier is enough
    __shared__ unsigned long long s_q[3];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint32_t n = a.n, m = a.m;
    int64_t unvisited = a.unvisited;
    const int32_t step = a.step;
    for (uint32_t i = tid; i < n; i += kCoopThreads) {
        const uint2 e = __ldcg(&a.q[i]);
        buf[0][i] = make_uint2(e.x - e.y, e.y);
    }
    if (tid < 3) s_q[tid] = tid == 0 ? ((unsigned long long)n << 32) | m : 0ull;
    __syncthreads();
    uint32_t steps = 0;
    unsigned long long edges = 0, work = 0;
    int next = 1;
    for (;;) {
        const uint2 *f = steps & 1 ? buf[1] : buf[0];
        uint2 *fn = steps & 1 ? buf[0] : buf[1];
        const int after = next == 2 ? 0 : next + 1;
        if (tid == 0) s_q[after] = 0ull;
        const int32_t lvl = step + (int32_t)steps + 1;
        work += m;
        // a warp without edges goes to the barrier
        for (uint32_t b = 0; b + (uint32_t)wid * 32u < m; b += kCoopThreads) {
            const uint32_t e = b + tid;
            int32_t v = -1, rs = 0;
            uint32_t d = 0;
            if (e < m) {
                uint32_t lo = 0, hi = n;  // f[lo].y <= e < f[hi].y
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (f[mid].y <= e) lo = mid; else hi = mid;
                }
                v = __ldg(&a.col[(int32_t)(f[lo].x + e)]);
                // the offsets load beside the claim, found or not
                rs = __ldg(&a.row[v]);
                const int32_t re = __ldg(&a.row[v + 1]);
                const uint32_t bit = 1u << (v & 31);
                if (!(atomicOr(&a.vis[v >> 5], bit) & bit)) {
                    a.level[v] = lvl;
                    d = (uint32_t)(re - rs);
                }
            }
            const unsigned in = __ballot_sync(0xffffffffu, d > 0);
            if (!in) continue;
            const uint32_t incl = warp_incl_scan_u32(d);
            unsigned long long base = 0;
            if (lane == 31) base = atomicAdd(&s_q[next], ((unsigned long long)__popc(in) << 32) | incl);
            base = __shfl_sync(0xffffffffu, base, 31);
            if (d > 0) {
                const uint32_t off = (uint32_t)base + incl - d;
                fn[(uint32_t)(base >> 32) + __popc(in & lanemask_lt())] = make_uint2((uint32_t)rs - off, off);
            }
        }
        __syncthreads();
        steps++;
        const unsigned long long c = s_q[next];
        n = (uint32_t)(c >> 32);
        m = (uint32_t)c;
        edges += m;
        unvisited -= (int64_t)m;
        next = after;
        if (n == 0 || m > kCoopTile || steps >= kSoloSteps || step + (int32_t)steps >= a.cap ||
            coop_pull_next(m, unvisited, a.alpha, a.gamma, a.E))
            break;
    }
    // the frontier to the other queue, with its tile table
    const uint2 *f = steps & 1 ? buf[1] : buf[0];
    for (uint32_t i = tid; i < n; i += kCoopThreads) {
        const uint32_t off = f[i].y, end = i + 1 < n ? f[i + 1].y : m;
        a.qn[i] = make_uint2(f[i].x + off, off);
        const uint32_t t0 = (off + kCoopTile - 1) / kCoopTile, t1 = (end - 1) / kCoopTile;
        for (uint32_t t = t0; t <= t1; t++) a.tf[t] = (int32_t)i;
    }
    if (tid == 0) {
        a.out->n = n;
        a.out->m = m;
        a.out->steps = steps;
        a.out->edges = edges;
        a.out->work = work;
    }
    __syncthreads();  // sm.out is the pushes' next
}

// The supersteps from the frontier in q[0] (n vertices, m out-edges, levels and
// visited bits set, tile table filled), then -1 for the vertices not reached and
// the report; false if a barrier gave up.  sm.nout is 0 and the frontier
// visible to every CTA (a barrier passed).  kSolo: small frontiers by one CTA;
// without it a run that has come to them stops there (CoopResume), for a
// kernel with it to go on from: both in one kernel cost the large supersteps
// of R-MAT 2^24 / 2^28 4% in registers.
template <bool kSolo>
__device__ __forceinline__ bool coop_bfs(const CoopArgs &a, CoopSmem &sm, uint32_t &barriers, uint32_t n,
                                         unsigned long long m, const CoopResume *from) {
    __shared__ unsigned long long s_r[kCoopThreads / 32];
    __shared__ SoloArgs s_solo;
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t gt = (int64_t)blockIdx.x * kCoopThreads + tid;
    int vb = 0, cur = 0, step = 0, pushes = 0, pulls = 0, err = 0;
    uint32_t it = 0, solos = 0;  // supersteps of the grid, calls of coop_solo
    int small = 0;               // supersteps in a row with a tile of edges or less
    bool queue = true;  // the frontier is in q[cur]; else what a pull added
    uint32_t prev_n = n;
    unsigned long long edges = m, work = 0;
    int64_t unvisited = a.E - (int64_t)m;
    if (kSolo && from) {
        vb = from->vb;
        cur = from->cur;
        step = from->step;
        pushes = from->pushes;
        pulls = from->pulls;
        n = from->n;
        prev_n = from->prev_n;
        m = from->m;
        edges = from->edges;
        work = from->work;
        unvisited = from->unvisited;
        small = kSoloAfter;
    }
    while (n > 0 && m > 0) {
        if (step >= a.cap) {
            err = ERR_STEP_CAP;
            break;
        }
        // the fixed rule (engine.cuh)
        bool pull;
        if (queue) pull = coop_pull_next(m, unvisited, a.alpha, a.gamma, a.E);
        else pull = !((int64_t)n * a.beta < (int64_t)a.V && n < prev_n);
        small = !pull && queue && m <= kCoopTile ? small + 1 : 0;
        if (!kSolo && small > kSoloAfter) {
            if (gt == 0) {
                a.sh->resume = CoopResume{vb, cur, step, pushes, pulls, n, prev_n, 0u, m, edges, work, unvisited};
                a.out->handed = 1ull;
            }
            return true;
        }
        if (kSolo && small > kSoloAfter) {
            // read by every CTA before the barrier after the next solo
            CoopSolo *so = &a.sh->solo[solos & 1];
            if (blockIdx.x == 0) {
                if (tid == 0)
                    s_solo = SoloArgs{a.row,  a.col,     a.level, a.tf[cur ^ 1], a.vis[vb], a.q[cur], a.q[cur ^ 1],
                                      so,     a.E,       unvisited, a.alpha,     a.gamma,   a.cap,    step,
                                      n,      (uint32_t)m};
                __syncthreads();
                coop_solo(s_solo, sm);
            }
            if (!coop_sync(a, ++barriers)) return false;
            prev_n = n = __ldcg(&so->n);
            m = __ldcg(&so->m);
            const uint32_t k = __ldcg(&so->steps);
            const unsigned long long found = __ldcg(&so->edges);
            edges += found;
            unvisited -= (int64_t)found;
            work += __ldcg(&so->work);
            step += (int)k;
            pushes += (int)k;
            cur ^= 1;
            solos++;
            continue;
        }
        CoopCtr *ctr = &a.sh->ctr[it % 3];
        it++;
        if (gt == 0) a.sh->ctr[it % 3] = CoopCtr{0ull, 0u, 0u, 0ull};  // last read before the barrier just passed
        const int32_t lvl = step + 1;
        if (pull) {
            coop_pull(a, a.vis[vb], a.vis[vb ^ 1], lvl, ctr);
            if (!coop_sync(a, ++barriers)) return false;
            prev_n = n;
            n = __ldcg(&ctr->n);
            m = __ldcg(&ctr->m);
            vb ^= 1;
            queue = false;
            pulls++;
            work += (unsigned long long)a.E;
        } else {
            if (!queue) {
                coop_toq(a, sm, a.vis[vb], a.vis[vb ^ 1], &a.sh->toq, a.q[cur], a.tf[cur]);
                if (!coop_sync(a, ++barriers)) return false;
                const unsigned long long c = __ldcg(&a.sh->toq);
                n = (uint32_t)(c >> 32);
                queue = true;
            }
            work += m;
            coop_push(a, sm, a.q[cur], a.tf[cur], n, (uint32_t)m, a.vis[vb], lvl, ctr, a.q[cur ^ 1], a.tf[cur ^ 1]);
            if (!coop_sync(a, ++barriers)) return false;
            if (gt == 0) a.sh->toq = 0ull;  // read by every CTA before this barrier
            const unsigned long long c = __ldcg(&ctr->q);
            n = (uint32_t)(c >> 32);
            m = (uint32_t)c;
            prev_n = n;
            cur ^= 1;
            pushes++;
        }
        edges += m;
        unvisited -= (int64_t)m;
        step++;
    }
    // vertices not reached, and the number of those that were
    const uint32_t *vis = a.vis[vb];
    unsigned long long reached = 0;
    for (int64_t w = (int64_t)blockIdx.x * (kCoopThreads / 32) + (tid >> 5); w < a.W;
         w += (int64_t)gridDim.x * (kCoopThreads / 32)) {
        const uint32_t word = vis[w];
        const int32_t v = (int32_t)(w * 32 + lane);
        if (lane == 0) reached += __popc(word);
        if (v < a.V && !((word >> lane) & 1u)) a.level[v] = -1;
    }
    reached = warp_sum(reached);
    if (lane == 0) s_r[tid >> 5] = reached;
    __syncthreads();
    if (tid == 0) {
        reached = 0;
        for (int w = 0; w < kCoopThreads / 32; w++) reached += s_r[w];
        if (reached) atomicAdd(&a.sh->reached, reached);
        __threadfence();
        if (atomicAdd(&a.sh->ticket, 1u) == gridDim.x - 1) {  // the last CTA reports
            a.out->supersteps = step;
            a.out->pushes = pushes;
            a.out->pulls = pulls;
            a.out->reached = atomicAdd(&a.sh->reached, 0ull);
            a.out->edges = edges;
            a.out->work = work;
            if (err) a.out->err = err;
        }
    }
    return true;
}

}  // namespace mb
