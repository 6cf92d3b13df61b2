// bfs_coop.cuh -- a whole BFS in one launch (internal).
#pragma once
#include "engine.cuh"

namespace mb {

constexpr int kBfsCoopTile = 1024;
constexpr int kBfsCoopCtas = 4;  // CTAs per SM of the cooperative grid
constexpr int32_t kBfsSmallV = 10240;  // 20 bytes of shared memory per vertex
constexpr int64_t kBfsSmallE = 1 << 16;

struct BfsCoopOut {
    int32_t supersteps, pushes, pulls, err;
    unsigned long long reached, edges, work;
};

struct BfsCoopState {
    bool built = false;
    DevBuf vis[2], q[2], tf[2], sh;
    ~BfsCoopState() { release(); }
    void release() {
        for (int i = 0; i < 2; i++) {
            vis[i].release();
            q[i].release();
            tf[i].release();
        }
        sh.release();
        built = false;
    }
    void ensure(const Graph &g);
};

// Whether the one-CTA kernel runs the graph; it stores the levels in one
// sweep, so `level` may also be pinned host memory then.
inline bool bfs_small(const Graph &g) { return g.V <= kBfsSmallV && g.E <= kBfsSmallE; }

// Whether the context's settings leave a whole BFS to run_bfs_coop.
bool bfs_coop_applies(const Context &ctx);

// One BFS from `source` into `level` (device memory, V entries).
// after: queued behind the run, before its host synchronisation.
void run_bfs_coop(Context &ctx, Graph &g, BfsCoopState &st, int32_t source, int32_t *level, mb_stats *stats,
                  const EmitFn *after);

}  // namespace mb
