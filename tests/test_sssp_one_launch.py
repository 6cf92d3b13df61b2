"""SSSP in one launch: tiles and bitmap words at their edges, buckets on and
off, the large supersteps' claim bitmap, zero, fractional and far-apart
weights, host and device outputs, and the grid barrier."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def hubs(V, E, seed, weights):
    """A graph with a hub (more than 64 out-edges), so that the kernel takes it."""
    rng = np.random.default_rng(seed)
    src = np.minimum((rng.random(E) ** 3 * V).astype(np.int64), V - 1).astype(np.int32)
    dst = np.minimum((rng.random(E) ** 2 * V).astype(np.int64), V - 1).astype(np.int32)
    src[:min(E, 100)] = 0
    w = {"int": rng.integers(1, 1001, E), "zero": rng.integers(0, 2, E) * 7,
         "fraction": rng.random(E) * 10, "apart": 10.0 ** rng.integers(0, 7, E)}[weights]
    return src, dst, w.astype(np.float32)


# buckets from 2^18 edges on, the claim bitmap in supersteps of 2^20 edges;
# bitmap words in fours (128 vertices)
SIZES = [(3, 200), (127, 1024), (128, 1025), (129, 70000), (5000, (1 << 18) - 1), (5000, 1 << 18),
         (100001, 1500000), (300000, 9000000)]


@pytest.mark.parametrize("weights", ["int", "zero", "fraction", "apart"])
@pytest.mark.parametrize("V,E", SIZES)
def test_distances_equal_the_oracle(gpu_ctx, V, E, weights):
    src, dst, w = hubs(V, E, V + E, weights)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    torch = pytest.importorskip("torch")
    out = torch.empty((1, V), dtype=torch.float32, device="cuda")
    degree = np.bincount(src, minlength=V)
    for s in {0, V - 1} if E < (1 << 20) else {0}:
        want, _ = O.sssp(V, src, dst, w, s)
        got, st = g.sssp([s])
        assert st["kernel_launches"] == 1
        np.testing.assert_array_equal(got[0].view(np.uint32), want.view(np.uint32))
        assert st["vertices_reached"] == int((want < api.MEDUSA_MAX).sum())
        assert st["edges_traversed"] == int(degree[want < api.MEDUSA_MAX].sum())
        g.sssp([s], out=out)
        np.testing.assert_array_equal(out.cpu().numpy()[0].view(np.uint32), want.view(np.uint32))
    g.close()


def test_grid_barrier_gives_up_and_recovers(gpu_ctx):
    src, dst, w = hubs(50000, 600000, 4, "int")
    g = gpu_ctx.graph_from_edges(50000, src, dst, w)
    want, _ = g.sssp([0])
    gpu_ctx.set_tunable("wait_polls", 0)
    try:
        with pytest.raises(api.MedusaError) as e:
            for _ in range(20):  # a wait of no polls ends well only if every CTA arrived before
                g.sssp([0])
        assert e.value.code == api.MB_ERR_TIMEOUT
    finally:
        gpu_ctx.set_tunable("wait_polls", -1)
    got, _ = g.sssp([0])
    np.testing.assert_array_equal(got, want)
    g.close()
