// bfs_coop.cuh -- a whole BFS in one launch (internal).
#pragma once
#include "engine.cuh"

namespace mb {

constexpr int kBfsCoopTile = 1024;
constexpr int kBfsCoopCtas = 4;  // CTAs per SM of the cooperative grid
constexpr int32_t kBfsSmallV = 10240;  // 20 bytes of shared memory per vertex
constexpr int64_t kBfsSmallE = 1 << 16;
constexpr int32_t kBfsSmallSources = 128;  // at most, in one launch

struct BfsCoopOut {
    int32_t supersteps, pushes, pulls, err;
    unsigned long long reached, edges, work;
    unsigned long long handed;  // left to the kernel with supersteps of one CTA
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

// Whether the graph fits the one-CTA kernel.
inline bool bfs_small(const Graph &g) { return g.V <= kBfsSmallV && g.E <= kBfsSmallE; }

// Whether the context's settings leave a whole BFS to run_bfs_coop.
bool bfs_coop_applies(const Context &ctx);

// A graph that fits one CTA: BFS from nsrc <= kBfsSmallSources sources (host
// array), a CTA each, into levels[s * V + v], which is written in one sweep and
// so may also be pinned host memory.
void run_bfs_small(Context &ctx, Graph &g, const int32_t *sources, int32_t nsrc, int32_t *levels, mb_stats *stats,
                   const EmitFn *after);

// One BFS from `source` into `level` (device memory, V entries).
// after: queued behind the run, before its host synchronisation.
void run_bfs_coop(Context &ctx, Graph &g, BfsCoopState &st, int32_t source, int32_t *level, mb_stats *stats,
                  const EmitFn *after);

}  // namespace mb
