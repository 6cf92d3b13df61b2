"""One-launch SSSP about the sizes where its buckets begin (2^22 edges) and get
narrower (7 edges per vertex): distances against the oracle."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weights", ["int", "fraction", "equal"])
@pytest.mark.parametrize("V,E", [(700000, (1 << 22) - 1), (700000, 1 << 22), (600000, 4200000 - 1),
                                 (600000, 4200000)])
def test_distances_equal_the_oracle(gpu_ctx, V, E, weights):
    rng = np.random.default_rng(E)
    src = np.minimum((rng.random(E) ** 2 * V).astype(np.int64), V - 1).astype(np.int32)
    dst = rng.integers(0, V, E).astype(np.int32)
    src[:100] = 0  # a hub
    w = {"int": rng.integers(1, 1001, E), "fraction": rng.random(E) * 10, "equal": np.full(E, 3)}[weights]
    w = w.astype(np.float32)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    want, _ = O.sssp(V, src, dst, w, 0)
    got, st = g.sssp([0])
    np.testing.assert_array_equal(got[0].view(np.uint32), want.view(np.uint32))
    assert st["vertices_reached"] == int((want < api.MEDUSA_MAX).sum())
    g.close()
