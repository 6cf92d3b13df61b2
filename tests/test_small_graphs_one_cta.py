"""SSSP and many-source runs of graphs that fit one CTA: both sides of its vertex
and edge limits, the graph staged in shared memory or not, long diameters, zero
and fractional weights, more sources than one launch takes, host and device
results."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def lattice(rows, cols):
    i = np.arange(rows * cols, dtype=np.int32).reshape(rows, cols)
    a = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    b = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    return rows * cols, np.concatenate([a, b]), np.concatenate([b, a])


def random_edges(V, E, power):
    rng = np.random.default_rng(V + E)
    src = np.minimum((rng.random(E) ** power * V).astype(np.int64), V - 1).astype(np.int32)
    dst = np.minimum((rng.random(E) ** power * V).astype(np.int64), V - 1).astype(np.int32)
    return V, src, dst


# one CTA: V <= 10240 and E <= 40960 (49152 without hubs; BFS 65536); staged where 24 V + 8 E bytes and the bitmaps fit in 220 KB
GRAPHS = {"one": (1, np.zeros(0, np.int32), np.zeros(0, np.int32)), "loop": (1, np.zeros(2, np.int32), np.zeros(2, np.int32)),
          "pair": lattice(1, 2), "word": lattice(1, 32), "line": lattice(1, 2000), "grid": lattice(100, 102),
          "at_v": lattice(64, 160), "past_v": lattice(7, 1463), "staged": random_edges(1000, 24000, 1),
          "hubs": random_edges(1000, 25000, 3), "at_e": random_edges(5000, 40960, 2),
          "past_e": random_edges(5000, 40961, 2), "flat_at_e": random_edges(5000, 49152, 1),
          "flat_past_e": random_edges(5000, 49153, 1), "thin": random_edges(10240, 12000, 1)}


@pytest.mark.parametrize("weights", ["integer", "zero", "fraction"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_distances_equal_the_oracle(gpu_ctx, name, weights):
    V, src, dst = GRAPHS[name]
    rng = np.random.default_rng(3)
    w = rng.integers(1, 101, len(src)).astype(np.float32)
    if weights == "zero":
        w[rng.random(len(src)) < 0.5] = 0
    elif weights == "fraction":
        w = rng.random(len(src), dtype=np.float32)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    torch = pytest.importorskip("torch")
    out = torch.empty((2, V), dtype=torch.float32, device="cuda")
    degree = np.bincount(src, minlength=V)
    sources = [V // 3, V - 1]
    both, stats = g.sssp(sources, out=out)
    reached = edges = 0
    for i, s in enumerate(sources):
        want = O.sssp(V, src, dst, w, s)[0]
        got, st = g.sssp([s])
        np.testing.assert_array_equal(got[0].view(np.uint32), want.view(np.uint32))
        np.testing.assert_array_equal(out.cpu().numpy()[i].view(np.uint32), want.view(np.uint32))
        hit = want < api.MEDUSA_MAX
        assert st["vertices_reached"] == int(hit.sum())
        assert st["edges_traversed"] == int(degree[hit].sum())
        reached += int(hit.sum())
        edges += int(degree[hit].sum())
    assert stats["vertices_reached"] == reached and stats["edges_traversed"] == edges
    g.close()


@pytest.mark.parametrize("nsrc", [2, 64, 128, 129, 300])
@pytest.mark.parametrize("name", ["pair", "grid", "hubs", "at_e"])
def test_many_sources(gpu_ctx, name, nsrc):
    V, src, dst = GRAPHS[name]
    w = np.random.default_rng(5).integers(1, 101, len(src)).astype(np.float32)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    sources = np.random.default_rng(nsrc).integers(0, V, nsrc).astype(np.int32)
    levels, ls = g.bfs(sources)
    dist, ds = g.sssp(sources)
    assert ls["vertices_reached"] == int((levels >= 0).sum())
    assert ds["vertices_reached"] == int((dist < api.MEDUSA_MAX).sum())
    aa = O.AAGraph(V, src, dst, None)
    for i in {0, 1, nsrc // 2, nsrc - 1, min(nsrc - 1, 127), min(nsrc - 1, 128)}:
        want, _ = O.bfs(V, aa, None, [int(sources[i])])
        np.testing.assert_array_equal(levels[i], want)
        np.testing.assert_array_equal(dist[i], O.sssp(V, src, dst, w, int(sources[i]))[0])
    g.close()


def test_superstep_cap(gpu_ctx):
    V, src, dst = GRAPHS["line"]
    g = gpu_ctx.graph_from_edges(V, src, dst, np.ones(len(src), np.float32))
    gpu_ctx.set_tunable("step_cap", 100)
    try:
        for run in (lambda: g.bfs([0]), lambda: g.sssp([0]), lambda: g.bfs([0, 1]), lambda: g.sssp([0, 1])):
            with pytest.raises(api.MedusaError) as e:
                run()
            assert e.value.code == api.MB_ERR_TIMEOUT
    finally:
        gpu_ctx.set_tunable("step_cap", -1)
    assert g.sssp([0])[0][0, -1] == V - 1
    g.close()
