"""Batched BFS, pull supersteps: in-lists at the edges of the pull's mappings
(a lane's own edges, the whole warp, one CTA), sources that die out, and a
list covered by its last edge only."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# a lane alone takes 16 in-edges, a warp lists up to 4096, a CTA (2048 per round) the rest
DEGREES = [0, 1, 4, 15, 16, 17, 79, 80, 81, 4095, 4096, 4097, 6144, 8193]


def star_graph(rng, first_hit):
    """Vertex d of the first len(DEGREES) has DEGREES[d] in-edges from distinct
    leaves; every source reaches one leaf; isolated and dead-end sources too."""
    n, leaves, nsrc = len(DEGREES), max(DEGREES), 40
    src, dst = [], []
    for d, deg in enumerate(DEGREES):
        src.append(n + np.arange(deg))
        dst.append(np.full(deg, d))
    base = n + leaves
    for s in range(nsrc - 3):
        # first_hit: the leaf every list starts with; else one that only the longest lists hold
        leaf = 0 if first_hit else int(rng.integers(4090, leaves))
        src.append([base + s])
        dst.append([n + leaf])
    src.append([base + nsrc - 3])  # a dead end: its only edge leaves the graph's rest
    dst.append([base + nsrc - 2])
    src.append(np.arange(n))       # the lists' owners lead back to a leaf
    dst.append(n + np.arange(n))
    V = base + nsrc
    src, dst = np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)
    order = rng.permutation(len(src))
    return V, src[order], dst[order], list(range(base, V))


@pytest.mark.parametrize("direction", [None, 4], ids=["fixed", "pull"])
@pytest.mark.parametrize("first_hit", [True, False], ids=["first", "late"])
def test_pull_list_lengths(gpu_ctx, direction, first_hit):
    V, src, dst, sources = star_graph(np.random.default_rng(5), first_hit)
    g = gpu_ctx.graph_from_edges(V, src, dst)
    if direction is not None:
        gpu_ctx.set_policy(api.MB_POLICY_FORCED, direction)
    try:
        levels, st = g.bfs(sources)
    finally:
        gpu_ctx.set_policy(api.MB_POLICY_FIXED)
    aa = O.AAGraph(V, src, dst, None)
    for i, s in enumerate(sources):
        want, _ = O.bfs(V, aa, None, [s])
        np.testing.assert_array_equal(levels[i], want, err_msg="source %d" % s)
    assert st["vertices_reached"] == int((levels >= 0).sum())
    g.close()
