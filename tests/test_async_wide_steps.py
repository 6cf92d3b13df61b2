"""The asynchronous kernel's threshold steps on graphs of fewer than 4 edges per
vertex: narrow where the frontier multiplies, wide where it is a front that moves
along; distances and levels against the oracle."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def uniform(V, E, seed):
    r = np.random.default_rng(seed)
    return V, r.integers(0, V, E).astype(np.int32), r.integers(0, V, E).astype(np.int32)


def grid(rows, cols, random_edges=0):
    i = np.arange(rows * cols).reshape(rows, cols)
    a = np.concatenate([i[:-1].ravel(), i[:, :-1].ravel()])
    b = np.concatenate([i[1:].ravel(), i[:, 1:].ravel()])
    t = np.random.default_rng(5).integers(0, rows * cols, (2, random_edges))
    s, d = np.concatenate([a, b, t[0]]), np.concatenate([b, a, t[1]])
    return rows * cols, s.astype(np.int32), d.astype(np.int32)


def run(ctx, graph, weights):
    V, s, d = graph
    r = np.random.default_rng(len(s))
    w = (r.integers(1, 101, len(s)) if weights == "int" else r.random(len(s)) * 10).astype(np.float32)
    g = ctx.graph_from_edges(V, s, d, w)
    dist, st = g.sssp([0])
    want, _ = O.sssp(V, s, d, w, 0)
    np.testing.assert_array_equal(dist[0].view(np.uint32), want.view(np.uint32))
    level, sb = g.bfs([0])
    want, _ = O.bfs(V, s, d, 0)
    np.testing.assert_array_equal(level[0], want)
    g.close()
    return st, sb


# about the size where the narrow step changes, and at the least and most edges per vertex
@pytest.mark.parametrize("V,E", [(1 << 21, 3 << 21), ((1 << 21) - 1, 3 << 21), (1 << 21, 5 << 20), (1 << 21, (5 << 20) - 1),
                                 (1 << 20, (4 << 20) - 1), (70001, 90000)])
def test_multiplying_frontiers_take_narrow_steps(gpu_ctx, V, E):
    st, _ = run(gpu_ctx, uniform(V, E, 3), "int")
    # relaxations per edge: about 1.3 with steps of 5 mean weights; wide ones
    # (24 mean weights) cover the whole graph at once
    if E >= 1 << 22:
        assert st["edges_scanned"] < 2 * st["edges_traversed"], st


@pytest.mark.parametrize("weights", ["int", "fraction"])
@pytest.mark.parametrize("rows,cols,random_edges", [(300, 300, 0), (1, 30000, 0), (2, 20000, 20), (700, 900, 3000)])
def test_moving_fronts_take_wide_steps(gpu_ctx, rows, cols, random_edges, weights):
    graph = grid(rows, cols, random_edges)
    st, sb = run(gpu_ctx, graph, weights)
    if (rows, cols) == (300, 300):  # 600 hops: 76 phases of 8, and some 28 of 24
        assert sb["supersteps"] < 50 and st["supersteps"] < 40, (st, sb)


@pytest.mark.parametrize("V,fan", [(70001, 2), (550000, 40), (1 << 20, 3)])
def test_trees(gpu_ctx, V, fan):
    v = np.arange(1, V)
    p = (v - 1) // fan
    s, d = np.concatenate([p, v]).astype(np.int32), np.concatenate([v, p]).astype(np.int32)
    st, sb = run(gpu_ctx, (V, s, d), "int")
    # every vertex has one path: nothing is relaxed twice
    assert st["edges_scanned"] == sb["edges_scanned"] == 2 * (V - 1)
