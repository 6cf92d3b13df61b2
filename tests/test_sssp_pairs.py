"""SSSP from several sources in one launch: pairs whose bitmap words cross
sources, repeated sources and sources without out-edges, groups of sources
(more than one run), hub-free and skewed graphs, zero weights."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def edges(kind, V, E, seed):
    rng = np.random.default_rng(seed)
    if kind == "skewed":
        src = np.minimum((rng.random(E) ** 3 * V).astype(np.int64), V - 1)
        dst = np.minimum((rng.random(E) ** 2 * V).astype(np.int64), V - 1)
    else:
        src, dst = rng.integers(0, V - 1, E), rng.integers(0, V, E)  # V - 1 has no out-edges
    w = rng.integers(0 if kind == "zero" else 1, 101, E)
    return src.astype(np.int32), dst.astype(np.int32), w.astype(np.float32)


@pytest.mark.parametrize("kind", ["uniform", "skewed", "zero"])
@pytest.mark.parametrize("V,E,nsrc", [(2, 3, 2), (33, 100, 3), (100, 700, 32), (127, 900, 33), (128, 900, 31),
                                      (1001, 9000, 70), (70001, 400000, 7), (300000, 1200000, 5)])
def test_every_source_equals_the_oracle(gpu_ctx, kind, V, E, nsrc):
    src, dst, w = edges(kind, V, E, V + nsrc)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    rng = np.random.default_rng(nsrc)
    sources = rng.integers(0, V, nsrc).astype(np.int32)
    sources[0], sources[-1] = V - 1, sources[nsrc // 2]
    torch = pytest.importorskip("torch")
    out = torch.empty((nsrc, V), dtype=torch.float32, device="cuda")
    got, st = g.sssp(sources)
    g.sssp(sources, out=out)
    np.testing.assert_array_equal(out.cpu().numpy(), got)
    degree = np.bincount(src, minlength=V)
    reached = edges_out = 0
    want = {}
    for i, s in enumerate(sources):
        if int(s) not in want:
            want[int(s)] = O.sssp(V, src, dst, w, int(s))[0]
        np.testing.assert_array_equal(got[i].view(np.uint32), want[int(s)].view(np.uint32), err_msg="source %d" % s)
        hit = want[int(s)] < api.MEDUSA_MAX
        reached += int(hit.sum())
        edges_out += int(degree[hit].sum())
    assert st["vertices_reached"] == reached
    assert st["edges_traversed"] == edges_out
    g.close()


def test_the_lines_still_run_and_agree(gpu_ctx):
    src, dst, w = edges("skewed", 5000, 60000, 3)
    g = gpu_ctx.graph_from_edges(5000, src, dst, w)
    sources = list(range(40))
    got, _ = g.sssp(sources)
    gpu_ctx.set_tunable("mss_delta", 0)
    try:
        lines, _ = g.sssp(sources)
    finally:
        gpu_ctx.set_tunable("mss_delta", -1)
    np.testing.assert_array_equal(got, lines)
    g.close()
