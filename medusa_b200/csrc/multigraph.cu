// multigraph.cu -- many independent graphs of uneven sizes in ONE persistent
// launch, fed by a device-side work queue.
//
// Each graph g gets a team of T_g CTAs, T_g growing with its edge count (the
// edges per CTA and the CTA size are tunables the autotuner sets).  The work
// queue is a list of (graph, member) entries, largest graph first, handed
// out by one atomic counter; a CTA that takes an entry runs its share of the
// graph -- `pr_iters` PageRank supersteps, then one BFS -- and synchronises
// with its team mates through a barrier in the graph's team state.  The
// launch is cooperative, so every CTA is resident: entries are handed out
// in order and a team's entries are consecutive, so at most one team is
// ever incomplete and the CTAs of complete teams always come back for more
// -- every barrier wait ends.  Every wait is also bounded: past kTeamSpins
// polls the CTA sets the batch's error flag and every CTA leaves.
//
// PageRank follows the fixed summation order of pr_order.cuh, so each
// graph's ranks equal mb_pagerank's on that graph bit for bit.  The BFS is
// level-synchronous and direction-optimising per level (top-down from the
// queue while the frontier holds fewer than V/20 vertices, else bottom-up),
// which gives the reference's levels (Algorithm/CPUFunctorHoster.cpp:16-65).
// No reference counterpart exists for the batching itself.
//
// That is the form with its parameters set (MB_TUNE_BATCH_*), and for batches
// of 2^31 edges or vertices.  By default the batch runs as ONE graph, the
// disjoint union of its graphs (k_union): teams leave a warp the 32 vertices of
// a group, hubs of thousands of in-edges one after another, and CTAs idle
// behind the largest graphs.  The union's vertices go through the sliced ELL
// and the heavy blocks of pagerank.cu, whatever graph they belong to, with one
// grid barrier per superstep, and its BFS has one source per graph, or, on small
// sparse graphs without hubs, runs graph by graph (union_by_graph).  The first
// run builds the union; where there is no memory for it, the teams run.  The sums'
// order is per vertex, so the ranks are the same bits.  64 graphs of 2^10 to
// 2^16 vertices, 21.6M edges, 20 supersteps and one BFS each: 2.28 ms,
// against 8.0.
#include <algorithm>
#include <cmath>
#include "frontier.cuh"
#include "bfs_coop_dev.cuh"
#include "multigraph.cuh"
#include "pr_sell.cuh"

namespace mb {
void graph_generate(Context &ctx, Graph &g, const mb_gen_params &p, uint32_t flags);

namespace {

constexpr long kTeamSpins = 1l << 24;  // polls (64 ns apart) before a barrier gives up (default)

struct MultiArgs {
    const GDesc *desc;
    TeamState *team;
    const int2 *entries;  // (graph, member), largest graph first
    int32_t nentries;
    int32_t pr_iters;
    float *contrib[2];    // batch-wide, graph g at desc[g].vbase
    int32_t *queue[2];
    float *rank;          // outputs, batch-wide
    int32_t *level;
    unsigned *work;       // [0] next entry, [1] error flag, [2] launches
    long wait_polls;      // polls before a team barrier gives up
};

// Team barrier (all threads of the CTA call it).  False if it gave up or
// another CTA reported an error.
__device__ bool team_sync(TeamState *ts, int t, unsigned *err, long polls) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        __threadfence();
        if (t > 1) {
            const unsigned gen = __ldcg(&ts->bar_gen);
            const unsigned arrived = atomicAdd(&ts->bar_count, 1u);
            if (arrived == (unsigned)t - 1) {
                atomicExch(&ts->bar_count, 0u);
                __threadfence();
                atomicAdd(&ts->bar_gen, 1u);
            } else {
                ok = 0;
                for (long it = 0; it < polls; it++) {
                    if (__ldcg(&ts->bar_gen) != gen) {
                        ok = 1;
                        break;
                    }
                    if (__ldcg(err)) break;
                    __nanosleep(64);
                }
                if (!ok) atomicExch(err, 1u);
            }
            __threadfence();
        }
        s_ok = ok && !__ldcg(err);
    }
    __syncthreads();
    return s_ok;
}

// Append v (where pred) to the team's next queue; all lanes call it.
__device__ __forceinline__ void append_warp(bool pred, int32_t v, unsigned *count, int32_t *q) {
    const unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (!mask) return;
    const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) q[base + __popc(mask & lanemask_lt())] = v;
}

struct Member {
    int k, t;             // member index, team size
    int64_t tid, nthr;    // thread index and count across the team
    int64_t warp, nwarp;  // warp index and count across the team
};

__device__ bool pr_phase(const MultiArgs &a, const GDesc &d, TeamState *ts, const Member &m) {
    const float init = 1.0f / (float)d.V;
    float *c0 = a.contrib[0] + d.vbase, *c1 = a.contrib[1] + d.vbase;
    float *rank = a.rank + d.vbase;
    for (int64_t v = m.tid; v < d.V; v += m.nthr) {
        const int32_t deg = d.row[v + 1] - d.row[v];
        c0[v] = deg > 0 ? init / (float)deg : 0.0f;
        if (a.pr_iters == 0) rank[v] = init;
    }
    if (!team_sync(ts, m.t, &a.work[1], a.wait_polls)) return false;
    const int lane = threadIdx.x & 31;
    const int64_t ngroups = ((int64_t)d.V + 31) / 32;
    for (int it = 0; it < a.pr_iters; it++) {
        const float *cin = (it & 1) ? c1 : c0;
        float *cout = (it & 1) ? c0 : c1;
        for (int64_t grp = m.warp; grp < ngroups; grp += m.nwarp) {
            const int32_t v = (int32_t)(grp * 32 + lane);
            const bool valid = v < d.V;
            int32_t b = 0, e = 0;
            if (valid) {
                b = __ldg(&d.rrow[v]);
                e = __ldg(&d.rrow[v + 1]);
            }
            const bool heavy = valid && (e - b) > kPrLight;
            float sum = 0.f;
            if (valid && !heavy) {
#pragma unroll 4
                for (int32_t j = b; j < e; j++) sum += __ldcg(&cin[__ldg(&d.rcol[j])]);
            }
            for (unsigned hm = __ballot_sync(0xffffffffu, heavy); hm; hm &= hm - 1) {
                const int owner = __ffs(hm) - 1;
                const int32_t hb = __shfl_sync(0xffffffffu, b, owner);
                const int32_t he = __shfl_sync(0xffffffffu, e, owner);
                float tot = 0.f;
                for (int64_t j0 = hb; j0 < he; j0 += kPrBlock) {
                    const int64_t j1 = min((int64_t)he, j0 + kPrBlock);
                    tot += pr_warp_block_sum(j0, j1, [&](int64_t j) { return __ldcg(&cin[__ldg(&d.rcol[j])]); });
                }
                if (lane == owner) sum = tot;
            }
            if (valid) {
                const float r = pr_update(sum);
                rank[v] = r;
                const int32_t deg = __ldg(&d.row[v + 1]) - __ldg(&d.row[v]);
                cout[v] = deg > 0 ? r / (float)deg : 0.0f;
            }
        }
        if (!team_sync(ts, m.t, &a.work[1], a.wait_polls)) return false;
    }
    return true;
}

__device__ bool bfs_phase(const MultiArgs &a, const GDesc &d, TeamState *ts, const Member &m) {
    int32_t *lv = a.level + d.vbase;
    int32_t *q[2] = {a.queue[0] + d.vbase, a.queue[1] + d.vbase};
    for (int64_t v = m.tid; v < d.V; v += m.nthr) lv[v] = -1;
    if (!team_sync(ts, m.t, &a.work[1], a.wait_polls)) return false;
    if (m.k == 0 && threadIdx.x == 0) {
        lv[d.source] = 0;
        q[0][0] = d.source;
        ts->qn[0] = 1;
    }
    if (!team_sync(ts, m.t, &a.work[1], a.wait_polls)) return false;
    const int lane = threadIdx.x & 31;
    for (int32_t L = 0;; L++) {
        const int cur = L % 3, nxt = (L + 1) % 3, clr = (L + 2) % 3;
        const unsigned n = __ldcg(&ts->qn[cur]);
        if (n == 0) break;  // every member reads the same count
        // the counter of level L-1 is read by nobody any more
        if (m.k == 0 && threadIdx.x == 0) ts->qn[clr] = 0;
        const int32_t *qc = q[L & 1];
        int32_t *qx = q[(L + 1) & 1];
        unsigned *cnt = &ts->qn[nxt];
        if ((int64_t)n * 20 > (int64_t)d.V) {
            // bottom-up: each unvisited vertex looks for a parent at level L
            for (int64_t base = m.warp * 32; base < d.V; base += m.nwarp * 32) {
                const int32_t v = (int32_t)(base + lane);
                bool found = false;
                if (v < d.V && __ldcg(&lv[v]) == -1) {
                    const int32_t jb = __ldg(&d.rrow[v]), je = __ldg(&d.rrow[v + 1]);
                    for (int32_t j = jb; j < je; j++) {
                        if (__ldcg(&lv[__ldg(&d.rcol[j])]) == L) {
                            found = true;
                            break;
                        }
                    }
                    if (found) lv[v] = L + 1;
                }
                append_warp(found, v, cnt, qx);
            }
        } else {
            // top-down from the queue: warps for lists of 32 or more, lanes below
            auto visit = [&](bool valid, int32_t v) {
                const bool claim = valid && __ldcg(&lv[v]) == -1 && atomicCAS(&lv[v], -1, L + 1) == -1;
                append_warp(claim, v, cnt, qx);
            };
            for (int64_t base = m.warp * 32; base < n; base += m.nwarp * 32) {
                const int64_t i = base + lane;
                int32_t st = 0, deg = 0;
                if (i < n) {
                    const int32_t u = __ldcg(&qc[i]);
                    st = __ldg(&d.row[u]);
                    deg = __ldg(&d.row[u + 1]) - st;
                }
                for (unsigned big = __ballot_sync(0xffffffffu, deg >= 32); big; big &= big - 1) {
                    const int l = __ffs(big) - 1;
                    const int32_t bst = __shfl_sync(0xffffffffu, st, l);
                    const int32_t bdeg = __shfl_sync(0xffffffffu, deg, l);
                    for (int32_t k = 0; k < bdeg; k += 32)
                        visit(k + lane < bdeg, k + lane < bdeg ? __ldg(&d.col[bst + k + lane]) : 0);
                }
                const int32_t sd = deg < 32 ? deg : 0;
                int32_t maxd = sd;
#pragma unroll
                for (int off = 16; off; off >>= 1) maxd = max(maxd, __shfl_xor_sync(0xffffffffu, maxd, off));
                for (int32_t r = 0; r < maxd; r++) visit(r < sd, r < sd ? __ldg(&d.col[st + r]) : 0);
            }
        }
        if (!team_sync(ts, m.t, &a.work[1], a.wait_polls)) return false;
    }
    // reached vertices and their out-edges (the traversal count)
    unsigned long long nr = 0, er = 0;
    for (int64_t v = m.tid; v < d.V; v += m.nthr) {
        if (__ldcg(&lv[v]) >= 0) {
            nr++;
            er += (unsigned)(__ldg(&d.row[v + 1]) - __ldg(&d.row[v]));
        }
    }
    nr = warp_sum(nr);
    er = warp_sum(er);
    if (lane == 0 && nr) {
        atomicAdd(&ts->reached, nr);
        atomicAdd(&ts->reached_edges, er);
    }
    return true;
}

__global__ void k_multi(MultiArgs a) {
    __shared__ int s_e;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.work[2], 1u);
    const int wpc = blockDim.x >> 5;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_e = (int)atomicAdd(&a.work[0], 1u);
        __syncthreads();
        const int e = s_e;
        if (e >= a.nentries || __ldcg(&a.work[1])) break;
        const int2 en = a.entries[e];
        const GDesc d = a.desc[en.x];
        TeamState *ts = &a.team[en.x];
        Member m;
        m.k = en.y;
        m.t = d.team;
        m.tid = (int64_t)m.k * blockDim.x + threadIdx.x;
        m.nthr = (int64_t)m.t * blockDim.x;
        m.warp = (int64_t)m.k * wpc + (threadIdx.x >> 5);
        m.nwarp = (int64_t)m.t * wpc;
        if (!pr_phase(a, d, ts, m)) continue;  // the error flag ends the loop
        bfs_phase(a, d, ts, m);
    }
}

// ---- the batch as one graph -------------------------------------------------------

struct UnionSrc {  // one graph of the union
    const int32_t *row, *col, *rrow, *rcol;
    int64_t vbase, ebase;
    int32_t V, E;
};

// Every graph's offsets and columns into the union's arrays, and its part of
// the first superstep's contributions.
__global__ void k_union_fill(const UnionSrc *src, int32_t n, int32_t *row, int32_t *col, int32_t *rrow, int32_t *rcol,
                             int32_t *outdeg) {
    for (int32_t i = blockIdx.y; i < n; i += gridDim.y) {
        const UnionSrc g = src[i];
        const int32_t t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
        const int32_t vb = (int32_t)g.vbase, eb = (int32_t)g.ebase;
        for (int64_t v = t; v < g.V; v += step) {
            row[g.vbase + v] = eb + g.row[v];
            rrow[g.vbase + v] = eb + g.rrow[v];
            outdeg[g.vbase + v] = g.row[v + 1] - g.row[v];
        }
        for (int64_t e = t; e < g.E; e += step) {
            col[g.ebase + e] = vb + g.col[e];
            rcol[g.ebase + e] = vb + g.rcol[e];
        }
        if (i == n - 1 && t == 0) {
            row[g.vbase + g.V] = eb + g.E;
            rrow[g.vbase + g.V] = eb + g.E;
        }
    }
}
__global__ void k_union_init(const UnionSrc *src, int32_t n, const int32_t *outdeg, const int32_t *pos, float *contrib) {
    for (int32_t i = blockIdx.y; i < n; i += gridDim.y) {
        const UnionSrc g = src[i];
        const float init = 1.0f / (float)g.V;
        for (int64_t v = g.vbase + blockIdx.x * blockDim.x + threadIdx.x; v < g.vbase + g.V;
             v += (int64_t)gridDim.x * blockDim.x)
            if (pos[v] >= 0) contrib[pos[v]] = init / (float)outdeg[v];
    }
}

struct UnionArgs {
    SellArgs sell;
    // heavy blocks (PrState): {j0, j1, vertex, hub slot or -1}
    const int4 *items;
    const int32_t *hcol, *pos, *outdeg, *slot_hub, *hub_first;
    float *blk_sum;
    uint32_t *hub_done;  // blocks of a hub summed; zero before and after a superstep
    int32_t nitems, nlong;
    const float *c0;     // the first superstep's contributions
    float *c[2], *rank;
    int32_t iters;
    uint32_t *ctr;       // units taken, one counter per superstep
    const int32_t *sources;  // vertices of the union, one per graph
    int32_t nsrc;
    unsigned long long *front;  // their queue's count << 32 | out-edges
    CoopArgs bfs;
    bool by_graph;       // the BFS graph by graph (union_by_graph), in `one`
    MultiArgs one;
};

// The BFS of every graph by one CTA, as a team of one.  A level then is a
// __syncthreads where the union's is a grid barrier, for a frontier that is
// small in each graph but not in all of them together (sparse graphs of a long
// diameter; ms, one superstep and the BFS, union / here: 200 grids of 30 x 30 0.53
// / 0.36, 16 of 100 x 100 1.28 / 1.00).
static __device__ __noinline__ void union_by_graph(const MultiArgs &a, CoopShared *sh, BfsCoopOut *out) {
    __shared__ int s_g;
    unsigned long long reached = 0, edges = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_g = (int)atomicAdd(&a.work[0], 1u);
        __syncthreads();
        const int i = s_g;
        if (i >= a.nentries) break;
        const GDesc d = a.desc[i];
        TeamState *ts = &a.team[i];
        Member m;
        m.k = 0;
        m.t = 1;
        m.tid = threadIdx.x;
        m.nthr = blockDim.x;
        m.warp = threadIdx.x >> 5;
        m.nwarp = blockDim.x >> 5;
        bfs_phase(a, d, ts, m);
        __syncthreads();
        reached += __ldcg(&ts->reached);
        edges += __ldcg(&ts->reached_edges);
    }
    if (threadIdx.x != 0) return;
    atomicAdd(&sh->reached, reached);
    atomicAdd(&sh->toq, edges);  // unused otherwise here
    __threadfence();
    if (atomicAdd(&sh->ticket, 1u) == gridDim.x - 1) {
        out->reached = atomicAdd(&sh->reached, 0ull);
        out->edges = atomicAdd(&sh->toq, 0ull);
    }
}

constexpr int kUnionCtas = 3;
constexpr int kUnionU = 8;

struct HeavyOut {  // pr_write's view of a superstep
    const int32_t *pos, *outdeg;
    float *contrib_out, *rank_out;
};

// One block of a heavy vertex, in the order of pr_warp_block_sum.  A hub's
// block sums are folded in order by the warp that finishes the last of them.
__device__ __forceinline__ void union_block(const UnionArgs &a, const HeavyOut &o, const float *cin, int32_t i) {
    const int lane = threadIdx.x & 31;
    const int4 it = __ldg(&a.items[i]);
    const int32_t len = it.y - it.x;
    float acc = 0.f;
    for (int32_t k0 = 0; k0 < len; k0 += 32 * kUnionU) {
        int32_t idx[kUnionU];
        float x[kUnionU];
#pragma unroll
        for (int q = 0; q < kUnionU; q++) {
            const int32_t k = k0 + lane + 32 * q;
            idx[q] = k < len ? ld_stream(&a.hcol[(int64_t)it.x + k]) : -1;
        }
#pragma unroll
        for (int q = 0; q < kUnionU; q++) x[q] = idx[q] >= 0 ? cin[idx[q]] : 0.f;
#pragma unroll
        for (int q = 0; q < kUnionU; q++)
            if (idx[q] >= 0) acc += x[q];
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane != 0) return;
    if (it.w < 0) {
        pr_write(o, it.z, 0.f + acc);
        return;
    }
    a.blk_sum[it.w] = acc;
    const int32_t h = a.slot_hub[it.w], f = a.hub_first[h], l = a.hub_first[h + 1];
    __threadfence();
    if (atomicAdd(&a.hub_done[h], 1u) != (uint32_t)(l - f) - 1u) return;
    __threadfence();
    a.hub_done[h] = 0u;
    float sum = 0.f;
    for (int32_t k = f; k < l; k++) sum += __ldcg(&a.blk_sum[k]);
    pr_write(o, it.z, sum);
}

__global__ void __launch_bounds__(kCoopThreads, kUnionCtas) k_union(UnionArgs a) {
    __shared__ CoopSmem sm;
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t gt = (int64_t)blockIdx.x * kCoopThreads + tid, gn = (int64_t)gridDim.x * kCoopThreads;
    const uint32_t warps = (uint32_t)(gn >> 5);
    uint32_t barriers = 0;
    for (int64_t w = gt; w < a.bfs.W; w += gn) a.bfs.vis[0][w] = 0u;
    if (tid == 0) sm.nout = 0;
    // 1. PageRank
    const uint32_t nsell = (uint32_t)a.sell.nlong + (uint32_t)(a.sell.ngroups - a.sell.nlong + 1) / 2;
    const uint32_t units = (uint32_t)a.nitems + nsell;
    // A warp's first unit.  The units are in order of their length: where there
    // are fewer than warps, next to each other the longest groups kept a few SMs
    // at work long after the others (1000 graphs of 2^6 vertices and 2^10 edges 36 us
    // per superstep, spread over the CTAs 8; 64 of 2^10 to 2^16, with 40,000 units,
    // 1% slower spread).
    const uint32_t gw = units < warps ? (uint32_t)(tid >> 5) * gridDim.x + blockIdx.x : (uint32_t)(gt >> 5);
    for (int it = 0; it < a.iters; it++) {
        SellArgs s = a.sell;
        s.contrib_in = it == 0 ? a.c0 : (it & 1) ? a.c[1] : a.c[0];
        s.contrib_out = (it & 1) ? a.c[0] : a.c[1];
        s.rank_out = it == a.iters - 1 ? a.rank : nullptr;
        s.zfirst = it < 2;
        const HeavyOut o{a.pos, a.outdeg, s.contrib_out, s.rank_out};
        zero_vertices(s);
        // the next units come from the counter
        uint32_t u = gw;
        while (u < units) {
            uint32_t t = 0;
            if (lane == 0) t = atomicAdd(&a.ctr[it], 1u);
            if (u < (uint32_t)a.nitems) {
                union_block(a, o, s.contrib_in, (int32_t)u);
            } else {
                const uint32_t k = u - (uint32_t)a.nitems;
                if (k < (uint32_t)s.nlong) sell_long<kUnionU, false>(s, k);
                else sell_short<2, false>(s, s.nlong + (int64_t)(k - s.nlong) * 2);
            }
            u = warps + __shfl_sync(0xffffffffu, t, 0);
        }
        if (!coop_sync(a.bfs, ++barriers)) return;
    }
    if (a.by_graph) {
        __shared__ MultiArgs s_one;
        if (tid == 0) s_one = a.one;
        __syncthreads();
        union_by_graph(s_one, a.bfs.sh, a.bfs.out);
        return;
    }
    // 2. one BFS from every graph's source; CTA 0 makes the frontier
    if (blockIdx.x == 0 && tid < 32) {
        uint32_t n = 0, m = 0;
        for (int32_t i0 = 0; i0 < a.nsrc; i0 += 32) {
            const int32_t v = i0 + lane < a.nsrc ? a.sources[i0 + lane] : -1;
            int32_t rs = 0, re = 0;
            if (v >= 0) {
                rs = __ldg(&a.bfs.row[v]);
                re = __ldg(&a.bfs.row[v + 1]);
                a.bfs.level[v] = 0;
                atomicOr(&a.bfs.vis[0][v >> 5], 1u << (v & 31));
            }
            const uint32_t d = (uint32_t)(re - rs);
            const unsigned in = __ballot_sync(0xffffffffu, d > 0);
            const uint32_t incl = warp_incl_scan_u32(d);
            if (d > 0) {
                const uint32_t pos = n + __popc(in & lanemask_lt()), off = m + incl - d;
                a.bfs.q[0][pos] = make_uint2((uint32_t)rs, off);
                for (uint32_t t = (off + kCoopTile - 1) / kCoopTile; t <= (off + d - 1) / kCoopTile; t++)
                    a.bfs.tf[0][t] = (int32_t)pos;
            }
            n += __popc(in);
            m += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) *a.front = ((unsigned long long)n << 32) | m;
    }
    if (!coop_sync(a.bfs, ++barriers)) return;
    const unsigned long long f = __ldcg(a.front);
    coop_bfs<true>(a.bfs, sm, barriers, (uint32_t)(f >> 32), (uint32_t)f, nullptr);
}

}  // namespace

// Keep the CSR and the reverse CSR of graph i (all the batch kernel reads)
// and count it into the batch's vertex offsets.
static void batch_take(Batch &b, int32_t i) {
    b.graphs[i].esrc.release();
    b.graphs[i].wt.release();
    b.graphs[i].rwt.release();
    b.graphs[i].mslot.release();
    b.vbase.push_back(b.vbase.back() + b.graphs[i].V);
    b.total_E += b.graphs[i].E;
}

void batch_generate(Context &ctx, Batch &b, const mb_gen_params *params, int32_t n) {
    b.release();
    b.graphs.resize(n);
    b.vbase.assign(1, 0);
    for (int32_t i = 0; i < n; i++) {
        graph_generate(ctx, b.graphs[i], params[i], MB_ORDER_REFERENCE);
        batch_take(b, i);
    }
    batch_finish(b);
}

void batch_from_edges(Context &ctx, Batch &b, int32_t n, const int32_t *nv, const int64_t *ne,
                      const int32_t *src, const int32_t *dst) {
    b.release();
    b.graphs.resize(n);
    b.vbase.assign(1, 0);
    int64_t e0 = 0;
    for (int32_t i = 0; i < n; i++) {
        DevBuf bs, bd;
        try {
            const size_t eb = sizeof(uint32_t) * (size_t)std::max<int64_t>(ne[i], 1);
            bs.reserve(eb);
            bd.reserve(eb);
            copy_sync(ctx.stream, bs.p, src + e0, 4 * (size_t)ne[i]);
            copy_sync(ctx.stream, bd.p, dst + e0, 4 * (size_t)ne[i]);
            graph_build_from_device_edges(ctx, b.graphs[i], nv[i], ne[i], bs.as<uint32_t>(),
                                          bd.as<uint32_t>(), nullptr, MB_ORDER_REFERENCE);
        } catch (...) {
            bs.release();
            bd.release();
            throw;
        }
        bs.release();
        bd.release();
        batch_take(b, i);
        e0 += ne[i];
    }
    batch_finish(b);
}

void batch_finish(Batch &b) {
    const int32_t n = (int32_t)b.graphs.size();
    b.total_V = b.vbase.back();
    const size_t vb = (size_t)std::max<int64_t>(b.total_V, 1);
    for (int i = 0; i < 2; i++) {
        b.contrib[i].reserve(sizeof(float) * vb);
        b.queue[i].reserve(sizeof(int32_t) * vb);
    }
    b.desc.reserve(sizeof(GDesc) * std::max(n, 1));
    b.team.reserve(sizeof(TeamState) * std::max(n, 1));
    b.work.reserve(4 * sizeof(unsigned));
    b.desc_gen = -1;
}

// The union of the batch's graphs and its lists (once).
static void union_build(Context &ctx, Batch &b) {
    if (b.uni) return;
    const int32_t n = (int32_t)b.graphs.size();
    cudaStream_t s = ctx.stream;
    std::unique_ptr<BatchUnion> u(new BatchUnion());
    Graph &g = u->g;
    g.V = (int32_t)b.total_V;
    g.E = b.total_E;
    g.device = ctx.device;
    const size_t eb = sizeof(int32_t) * (size_t)std::max<int64_t>(g.E, 1), vb = sizeof(int32_t) * (size_t)g.V;
    g.row.reserve(vb + 4);
    g.rrow.reserve(vb + 4);
    g.outdeg.reserve(vb);
    g.col.reserve(eb);
    g.rcol.reserve(eb);
    std::vector<UnionSrc> src((size_t)n);
    int64_t ebase = 0;
    for (int32_t i = 0; i < n; i++) {
        const Graph &x = b.graphs[i];
        src[i] = UnionSrc{x.row.as<int32_t>(), x.col.as<int32_t>(), x.rrow.as<int32_t>(), x.rcol.as<int32_t>(),
                          b.vbase[i], ebase, x.V, (int32_t)x.E};
        ebase += x.E;
        g.max_outdeg = std::max(g.max_outdeg, x.max_outdeg);
        g.max_indeg = std::max(g.max_indeg, x.max_indeg);
    }
    u->src.reserve(sizeof(UnionSrc) * (size_t)n);
    copy_sync(s, u->src.p, src.data(), sizeof(UnionSrc) * (size_t)n);
    const dim3 grid(32, (unsigned)std::min(n, 4096));
    k_union_fill<<<grid, 256, 0, s>>>(u->src.as<UnionSrc>(), n, g.row.as<int32_t>(), g.col.as<int32_t>(),
                                      g.rrow.as<int32_t>(), g.rcol.as<int32_t>(), g.outdeg.as<int32_t>());
    MB_CHECK_LAUNCH();
    MB_CUDA(cudaStreamSynchronize(s));
    PrState &pr = u->pr;
    // by id within a class: a graph's contributions stay together (64 graphs of
    // 2^10 to 2^16 vertices 2.24 against 2.39 ms)
    pr.by_indegree = false;
    pr.ensure(ctx, g);
    pr.ensure_fixed(ctx, g);
    u->c0.reserve(sizeof(float) * (size_t)g.V);
    k_union_init<<<grid, 256, 0, s>>>(u->src.as<UnionSrc>(), n, g.outdeg.as<int32_t>(), pr.pos.as<int32_t>(),
                                      u->c0.as<float>());
    MB_CHECK_LAUNCH();
    std::vector<int32_t> first((size_t)pr.nhub + 1);
    copy_sync(s, first.data(), pr.hub_first.p, sizeof(int32_t) * first.size());
    std::vector<int32_t> hub((size_t)std::max(first[(size_t)pr.nhub], 1), 0);
    for (int32_t h = 0; h < pr.nhub; h++)
        for (int32_t k = first[h]; k < first[(size_t)h + 1]; k++) hub[k] = h;
    u->slot_hub.reserve(sizeof(int32_t) * hub.size());
    copy_sync(s, u->slot_hub.p, hub.data(), sizeof(int32_t) * hub.size());
    u->hub_done.reserve(sizeof(uint32_t) * (size_t)std::max(pr.nhub, 1));
    MB_CUDA(cudaMemsetAsync(u->hub_done.p, 0, sizeof(uint32_t) * (size_t)std::max(pr.nhub, 1), s));
    u->bfs.ensure(g);
    u->front.reserve(sizeof(unsigned long long));
    u->sources.reserve(sizeof(int32_t) * (size_t)n);
    MB_CUDA(cudaStreamSynchronize(s));
    b.uni = std::move(u);
}

// Graph i as the teams' kernel reads it, without its team and source.
static GDesc graph_desc(const Batch &b, int32_t i) {
    const Graph &g = b.graphs[i];
    GDesc d{};
    d.V = g.V;
    d.E = (int32_t)g.E;
    d.row = g.row.as<int32_t>();
    d.col = g.col.as<int32_t>();
    d.rrow = g.rrow.as<int32_t>();
    d.rcol = g.rcol.as<int32_t>();
    d.vbase = b.vbase[i];
    return d;
}

// Whether the union's BFS goes graph by graph: graphs that had a CTA each in
// the teams' form, without hubs and with 2 to 6 edges per vertex (grids).  Lines and
// trees have fewer: their frontiers stay small in the union too (64 lines of 1000
// 1.45 ms there, 3.4 by graph), and denser graphs have short diameters.
static bool union_bfs_by_graph(const Batch &b) {
    for (const Graph &g : b.graphs)
        if (g.E + g.V > (1 << 16) || g.max_outdeg > 64 || g.E < 2 * (int64_t)g.V || g.E > 6 * (int64_t)g.V) return false;
    return b.graphs.size() > 1;
}

static void union_run(Context &ctx, Batch &b, int32_t pr_iters, const int32_t *sources, float *ranks_dev,
                      int32_t *levels_dev, mb_stats *stats) {
    const int32_t n = (int32_t)b.graphs.size();
    cudaStream_t s = ctx.stream;
    std::vector<int32_t> src((size_t)n);
    for (int32_t i = 0; i < n; i++) {
        const int32_t v = sources ? sources[i] : 0;
        if (v < 0 || v >= b.graphs[i].V) fail(MB_ERR_INVALID, "batch: source vertex out of range");
        src[i] = (int32_t)(b.vbase[i] + v);
    }
    BatchUnion &u = *b.uni;
    const Graph &g = u.g;
    PrState &pr = u.pr;
    MB_CUDA(cudaMemcpyAsync(u.sources.p, src.data(), sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, s));
    volatile BfsCoopOut *out = (volatile BfsCoopOut *)ctx.ctrl_readback();
    out->err = 0;
    UnionArgs a{};
    const PrSell &l = pr.light;
    a.sell.v = l.v.as<int32_t>();
    a.sell.pd = l.pd.as<int2>();
    a.sell.rows = l.rows.as<int32_t>();
    a.sell.base = l.base.as<uint32_t>();
    a.sell.src = l.src.as<int32_t>();
    a.sell.ngroups = l.ngroups;
    a.sell.nlong = l.nlong;
    a.sell.zv = l.zv.as<int32_t>();
    a.sell.zpd = l.zpd.as<int2>();
    a.sell.nz = l.nz;
    a.items = pr.items.as<int4>();
    a.nitems = pr.nitems;
    a.hcol = pr.hcol.as<int32_t>();
    a.pos = pr.pos.as<int32_t>();
    a.outdeg = g.outdeg.as<int32_t>();
    a.slot_hub = u.slot_hub.as<int32_t>();
    a.hub_first = pr.hub_first.as<int32_t>();
    a.blk_sum = pr.blk_sum.as<float>();
    a.hub_done = u.hub_done.as<uint32_t>();
    a.c0 = u.c0.as<float>();
    a.c[0] = pr.contrib[0].as<float>();
    a.c[1] = pr.contrib[1].as<float>();
    a.rank = ranks_dev;
    a.iters = pr_iters;
    const size_t ctr_bytes = sizeof(uint32_t) * (size_t)pr_iters;
    a.ctr = (uint32_t *)pr.ctr.reserve(ctr_bytes);
    a.sources = u.sources.as<int32_t>();
    a.nsrc = n;
    a.front = u.front.as<unsigned long long>();
    CoopArgs &f = a.bfs;
    f.V = g.V;
    f.E = g.E;
    f.W = ((int64_t)g.V + 31) / 32;
    f.row = g.row.as<int32_t>();
    f.col = g.col.as<int32_t>();
    f.rrow = g.rrow.as<int32_t>();
    f.rcol = g.rcol.as<int32_t>();
    f.level = levels_dev;
    for (int i = 0; i < 2; i++) {
        f.vis[i] = u.bfs.vis[i].as<uint32_t>();
        f.q[i] = u.bfs.q[i].as<uint2>();
        f.tf[i] = u.bfs.tf[i].as<int32_t>();
    }
    f.sh = u.bfs.sh.as<CoopShared>();
    f.out = (BfsCoopOut *)ctx.ctrl_readback();
    f.alpha = 15;  // fixed_rule's defaults
    f.beta = 20;
    f.gamma = kBfsGammaDefault;
    f.cap = INT32_MAX;  // every superstep reaches a vertex
    f.polls = ctx.tunable[MB_TUNE_WAIT_POLLS] >= 0 ? (long)ctx.tunable[MB_TUNE_WAIT_POLLS] : kBarrierSpins;
    a.by_graph = union_bfs_by_graph(b);
    std::vector<GDesc> desc;
    if (a.by_graph) {
        for (int32_t i = 0; i < n; i++) {
            desc.push_back(graph_desc(b, i));
            desc.back().source = sources ? sources[i] : 0;
        }
        MB_CUDA(cudaMemcpyAsync(b.desc.p, desc.data(), sizeof(GDesc) * n, cudaMemcpyHostToDevice, s));
        MB_CUDA(cudaMemsetAsync(b.team.p, 0, sizeof(TeamState) * n, s));
        MB_CUDA(cudaMemsetAsync(b.work.p, 0, 4 * sizeof(unsigned), s));
        a.one.desc = b.desc.as<GDesc>();
        a.one.team = b.team.as<TeamState>();
        a.one.nentries = n;
        a.one.queue[0] = b.queue[0].as<int32_t>();
        a.one.queue[1] = b.queue[1].as<int32_t>();
        a.one.level = levels_dev;
        a.one.work = b.work.as<unsigned>();
        a.one.wait_polls = f.polls;
        out->edges = out->reached = 0;
    }
    int per_sm = 0;
    MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_union, kCoopThreads, 0));
    if (per_sm < 1) fail(MB_ERR_UNSUPPORTED, "batch kernel does not fit on an SM");
    // no more CTAs than tiles: fewer arrive at the barriers of small batches
    const int grid = (int)std::min<int64_t>(ctx.num_sms * std::min(per_sm, kUnionCtas),
                                            std::max<int64_t>(g.E / kCoopTile, 16));
    const cudaEvent_t e0 = ctx.event(0), e1 = ctx.event(1);
    MB_CUDA(cudaEventRecord(e0, s));
    MB_CUDA(cudaMemsetAsync(f.sh, 0, sizeof(CoopShared), s));
    MB_CUDA(cudaMemsetAsync(a.ctr, 0, ctr_bytes, s));
    void *params[] = {(void *)&a};
    MB_CUDA(cudaLaunchCooperativeKernel((const void *)k_union, dim3(grid), dim3(kCoopThreads), params, 0, s));
    MB_CUDA(cudaEventRecord(e1, s));
    MB_CUDA(cudaStreamSynchronize(s));
    if (out->err) {  // a superstep may have been left half way
        MB_CUDA(cudaMemsetAsync(a.hub_done, 0, sizeof(uint32_t) * (size_t)std::max(pr.nhub, 1), s));
        MB_CUDA(cudaStreamSynchronize(s));
        fail(MB_ERR_TIMEOUT, "batch: a grid barrier timed out");
    }
    float ms = 0;
    MB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (stats) {
        *stats = mb_stats{};
        stats->supersteps = pr_iters;
        stats->edges_traversed = (int64_t)pr_iters * b.total_E + (int64_t)out->edges;
        stats->vertices_reached = (int64_t)out->reached;
        stats->device_ms = ms;
        stats->kernel_launches = 1;
        stats->edges_scanned = (int64_t)out->edges;
    }
}

void batch_run(Context &ctx, Batch &b, int32_t pr_iters, const int32_t *sources, float *ranks_dev,
               int32_t *levels_dev, mb_stats *stats) {
    const int32_t n = (int32_t)b.graphs.size();
    if (pr_iters > 0 && b.total_V <= INT32_MAX && b.total_E <= INT32_MAX &&
        ctx.tunable[MB_TUNE_BATCH_THREADS] < 0 && ctx.tunable[MB_TUNE_BATCH_EDGES_PER_CTA] < 0 && !b.no_union) {
        b.no_union = !memory_for([&] { union_build(ctx, b); }, [] {});
        if (!b.no_union) {
            union_run(ctx, b, pr_iters, sources, ranks_dev, levels_dev, stats);
            return;
        }
    }
    cudaStream_t s = ctx.stream;
    const int threads = (int)(ctx.tunable[MB_TUNE_BATCH_THREADS] > 0 ? ctx.tunable[MB_TUNE_BATCH_THREADS] : 256);
    const int64_t epc = ctx.tunable[MB_TUNE_BATCH_EDGES_PER_CTA] > 0 ? ctx.tunable[MB_TUNE_BATCH_EDGES_PER_CTA]
                                                                     : (int64_t)1 << 16;
    int per_sm = 0;
    MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)k_multi, threads, 0));
    if (per_sm < 1) fail(MB_ERR_UNSUPPORTED, "batch kernel does not fit on an SM");
    const int grid = ctx.num_sms * per_sm;
    // descriptors and the work queue (largest graph first)
    std::vector<GDesc> desc(n);
    std::vector<int32_t> order(n);
    int64_t nent = 0;
    for (int32_t i = 0; i < n; i++) {
        const Graph &g = b.graphs[i];
        GDesc &d = desc[i];
        d = graph_desc(b, i);
        d.team = (int32_t)std::min<int64_t>(std::max<int64_t>(1, (g.E + g.V + epc - 1) / epc), grid);
        d.source = sources ? sources[i] : 0;
        if (d.source < 0 || d.source >= g.V) fail(MB_ERR_INVALID, "batch: source vertex out of range");
        order[i] = i;
        nent += d.team;
    }
    std::stable_sort(order.begin(), order.end(),
                     [&](int32_t x, int32_t y) { return desc[x].E + desc[x].V > desc[y].E + desc[y].V; });
    std::vector<int2> ent;
    ent.reserve((size_t)nent);
    for (int32_t i : order)
        for (int32_t k = 0; k < desc[i].team; k++) ent.push_back(make_int2(i, k));
    b.entries.reserve(sizeof(int2) * std::max<size_t>(ent.size(), 1));
    b.nentries = (int32_t)ent.size();
    MB_CUDA(cudaMemcpyAsync(b.desc.p, desc.data(), sizeof(GDesc) * n, cudaMemcpyHostToDevice, s));
    MB_CUDA(cudaMemcpyAsync(b.entries.p, ent.data(), sizeof(int2) * ent.size(), cudaMemcpyHostToDevice, s));
    MultiArgs a;
    a.desc = b.desc.as<GDesc>();
    a.team = b.team.as<TeamState>();
    a.entries = b.entries.as<int2>();
    a.nentries = b.nentries;
    a.pr_iters = pr_iters;
    a.contrib[0] = b.contrib[0].as<float>();
    a.contrib[1] = b.contrib[1].as<float>();
    a.queue[0] = b.queue[0].as<int32_t>();
    a.queue[1] = b.queue[1].as<int32_t>();
    a.rank = ranks_dev;
    a.level = levels_dev;
    a.work = b.work.as<unsigned>();
    a.wait_polls = ctx.tunable[MB_TUNE_WAIT_POLLS] >= 0 ? (long)ctx.tunable[MB_TUNE_WAIT_POLLS] : kTeamSpins;
    cudaEvent_t e0, e1;
    MB_CUDA(cudaEventCreate(&e0));
    MB_CUDA(cudaEventCreate(&e1));
    try {
        MB_CUDA(cudaEventRecord(e0, s));
        MB_CUDA(cudaMemsetAsync(b.team.p, 0, sizeof(TeamState) * n, s));
        MB_CUDA(cudaMemsetAsync(b.work.p, 0, 4 * sizeof(unsigned), s));
        void *params[] = {(void *)&a};
        MB_CUDA(cudaLaunchCooperativeKernel((const void *)k_multi, dim3(grid), dim3(threads), params, 0, s));
        MB_CUDA(cudaEventRecord(e1, s));
        MB_CUDA(cudaEventSynchronize(e1));
        float ms = 0;
        MB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        unsigned work[4];
        MB_CUDA(cudaMemcpy(work, b.work.p, sizeof(work), cudaMemcpyDeviceToHost));
        if (work[1]) fail(MB_ERR_TIMEOUT, "batch: a team barrier timed out");
        std::vector<TeamState> ts(n);
        MB_CUDA(cudaMemcpy(ts.data(), b.team.p, sizeof(TeamState) * n, cudaMemcpyDeviceToHost));
        if (stats) {
            *stats = mb_stats{};
            int64_t reached = 0, redges = 0;
            for (const auto &t : ts) {
                reached += (int64_t)t.reached;
                redges += (int64_t)t.reached_edges;
            }
            stats->supersteps = pr_iters;
            stats->edges_traversed = (int64_t)pr_iters * b.total_E + redges;
            stats->vertices_reached = reached;
            stats->device_ms = ms;
            stats->kernel_launches = work[2];
            stats->edges_scanned = redges;
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
