"""Batched BFS on sparse graphs of a long diameter and on graphs with hubs: the
supersteps that list their vertices, those that pass over all of them (from V
out-edges, or with hubs from 16 V over the sources on), pulls with a few sources
per vertex and none, more dense supersteps than are kept."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def torus(k):
    i = np.arange(k ** 3).reshape(k, k, k)
    s = np.concatenate([i.ravel()] * 6)
    d = np.concatenate([np.roll(i, r, ax).ravel() for ax in range(3) for r in (1, -1)])
    return k ** 3, s, d


def ring(V, k, hub):
    v = np.arange(V)
    s = np.concatenate([v] * (2 * k) + [np.full(hub, 3)])
    d = np.concatenate([(v + r) % V for j in range(1, k + 1) for r in (j, -j)] + [np.arange(hub) * 101 % V])
    return V, s, d


def skewed(V, E):
    rng = np.random.default_rng(E)
    return V, (rng.random(E) ** 3 * V).astype(np.int64), (rng.random(E) ** 2 * V).astype(np.int64)


SHAPES = {"torus": torus(23), "ring": ring(12001, 4, 0), "ring, hub": ring(12001, 8, 400), "skewed": skewed(20001, 300000),
          "uniform": (30001,) + tuple(np.random.default_rng(2).integers(0, 30001, (2, 150000)))}


@pytest.mark.parametrize("nsrc", [2, 8, 33, 64])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_every_source_equals_the_oracle(gpu_ctx, name, nsrc):
    V, src, dst = SHAPES[name]
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    g = gpu_ctx.graph_from_edges(V, src, dst)
    assert V > 10240
    sources = np.random.default_rng(nsrc).integers(0, V, nsrc).astype(np.int32)
    got, st = g.bfs(sources)
    degree = np.bincount(src, minlength=V)
    reached = edges = 0
    for i, s in enumerate(sources):
        want, _ = O.bfs(V, src, dst, [int(s)])
        np.testing.assert_array_equal(got[i], want)
        hit = want >= 0
        reached += int(hit.sum())
        edges += int(degree[hit].sum())
    assert st["vertices_reached"] == reached
    assert st["edges_traversed"] == edges
    g.close()
