// sssp_coop.cuh -- a whole SSSP in one launch (internal).
#pragma once
#include "engine.cuh"

namespace mb {

constexpr int kSsspCoopTile = 512;

struct SsspCoopOut {
    int32_t supersteps, splits, err, pad;
    unsigned long long reached, edges, work;
};

struct SsspCoopState {
    bool built = false;
    bool weights_ok = false;  // no negative or NaN weight
    float mean_w = 0.f;
    DevBuf dist, claim[2], far, q[2], qv[2], tf[2], sh;
    ~SsspCoopState() { release(); }
    void release() {
        for (int i = 0; i < 2; i++) {
            claim[i].release();
            q[i].release();
            qv[i].release();
            tf[i].release();
        }
        dist.release();
        far.release();
        sh.release();
        built = false;
    }
    void ensure(const Graph &g);
};

// Whether the context's settings and the graph leave a whole SSSP to
// run_sssp_coop (makes the state when they do).
bool sssp_coop_applies(const Context &ctx, const Graph &g, SsspCoopState &st);

// One SSSP from `source` into `dist` (device memory, V entries).
// after: queued behind the run, before its host synchronisation.
void run_sssp_coop(Context &ctx, Graph &g, SsspCoopState &st, int32_t source, float *dist, mb_stats *stats,
                   const EmitFn *after);

}  // namespace mb
