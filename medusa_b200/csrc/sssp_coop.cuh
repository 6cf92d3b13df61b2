// sssp_coop.cuh -- a whole SSSP in one launch (internal).
#pragma once
#include "engine.cuh"
#include "pairs_limit.h"

namespace mb {

constexpr int kSsspCoopTile = 512;
constexpr int32_t kSsspSmallV = 10240;  // 20 bytes of shared memory per vertex
constexpr int64_t kSsspSmallE = 49152, kSsspSmallHubE = 40960;  // without hubs, with
constexpr int32_t kSsspSmallSources = 128;  // at most, in one launch

struct SsspCoopOut {
    int32_t supersteps, splits, err;
    int32_t handed;  // 1: the run stopped, its frontiers long small (SsspRest)
    unsigned long long reached, edges, work;
    uint32_t n;      // handed: the near queue's entries,
    int32_t cur;     // which queue it is,
    float T;         // and the threshold
};

// What a run that stopped has left to do: the distances so far, and the vertices
// whose out-edges are not relaxed from theirs -- n of the near queue, and those
// of the far bitmap at T or above.
struct SsspRest {
    const float *dist;
    const int32_t *near;
    uint32_t n;
    const uint32_t *far;
    float T;
};

struct SsspCoopState {
    bool built = false;
    bool weights_ok = false;  // no negative or NaN weight
    float mean_w = 0.f;
    int32_t room = 0;  // sources the buffers below hold at once
    DevBuf claim[2], far, q[2], qv[2], qs[2], tf[2], sh, front, srcs;
    ~SsspCoopState() { release(); }
    void release_room() {
        for (int i = 0; i < 2; i++) {
            claim[i].release();
            q[i].release();
            qv[i].release();
            qs[i].release();
            tf[i].release();
        }
        far.release();
        room = 0;
    }
    void release() {
        release_room();
        sh.release();
        front.release();
        srcs.release();
        built = false;
    }
    void ensure(const Graph &g, int32_t nsrc);
};

// Whether the context's settings and the graph leave SSSP from nsrc sources to
// run_sssp_coop (makes the state when they do).
bool sssp_coop_applies(const Context &ctx, const Graph &g, SsspCoopState &st, int32_t nsrc);

// Sources that one run takes at a time.
int32_t sssp_coop_sources(const Graph &g);

// SSSP from nsrc sources (host array) into dist[s * V + v] (device memory).
// after: queued behind the run, before its host synchronisation.  rest, for one
// source: the run may stop where the asynchronous kernel is the better one for
// what is left; it then returns true, with that in *rest (valid until the
// next run) and the statistics of its own part (run_sssp takes it on).
bool run_sssp_coop(Context &ctx, Graph &g, SsspCoopState &st, const int32_t *sources, int32_t nsrc, float *dist,
                   mb_stats *stats, const EmitFn *after, SsspRest *rest = nullptr);

// A graph that fits one CTA, nsrc <= kSsspSmallSources sources (a CTA each):
// the same, but the distances are stored in one sweep, so `dist` may also be
// pinned host memory.
bool sssp_small(const Graph &g);
void run_sssp_small(Context &ctx, Graph &g, SsspCoopState &st, const int32_t *sources, int32_t nsrc, float *dist,
                    mb_stats *stats, const EmitFn *after);

}  // namespace mb
