"""Many sparse hub-free graphs, whose BFS goes graph by graph inside the union's
launch: sizes about a CTA's (2^16 edges and vertices), more graphs than CTAs, and
batches just past the rule, against the oracle."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def grid(k, m):
    i = np.arange(k * m).reshape(k, m)
    a = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    b = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    return k * m, np.concatenate([a, b]).astype(np.int32), np.concatenate([b, a]).astype(np.int32)


BATCHES = {
    "grids": [grid(3, 3), grid(30, 7), grid(31, 33), grid(100, 100), grid(2, 500)],
    "largest": [grid(114, 114), grid(115, 114)],  # 64524 and 65090 edges and vertices
    "past it": [grid(114, 114), grid(116, 115)],  # 66238
    "many": [grid(4 + i % 9, 3 + i % 5) for i in range(700)],
    "one dense": [grid(40, 40), (64, *(np.random.default_rng(1).integers(0, 64, 600).astype(np.int32)
                                       for _ in range(2)))],
}


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_ranks_levels_and_counts(gpu_ctx, name):
    gs = BATCHES[name]
    b = gpu_ctx.batch_upload(gs)
    sources = [(7 * i) % V for i, (V, _, _) in enumerate(gs)]
    for iters in (1, 4):
        ranks, levels, st = b.run(iters, sources)
        reached = edges = 0
        seen = {}
        for i, ((V, s, d), r, l) in enumerate(zip(gs, b.split(ranks), b.split(levels))):
            key = (V, s.tobytes(), sources[i])
            if key not in seen:
                seen[key] = (O.pagerank(V, s, d, iters, np.float32(1.0 / V), order="device"), O.bfs(V, s, d, [sources[i]])[0])
            np.testing.assert_array_equal(r, seen[key][0])
            np.testing.assert_array_equal(l, seen[key][1])
            hit = l >= 0
            reached += int(hit.sum())
            edges += int(np.bincount(s, minlength=V)[hit].sum())
        assert st["vertices_reached"] == reached
        assert st["edges_traversed"] == iters * b.total_E + edges
        assert st["kernel_launches"] == 1
    b.close()


def test_other_forms_between(gpu_ctx):
    gs = BATCHES["grids"]
    b = gpu_ctx.batch_upload(gs)
    want = b.run(2)
    gpu_ctx.set_tunable("batch_threads", 128)  # the teams, in the same buffers
    try:
        teams = b.run(2)
    finally:
        gpu_ctx.set_tunable("batch_threads", -1)
    again = b.run(2)
    for got in (teams, again):
        np.testing.assert_array_equal(got[0], want[0])
        np.testing.assert_array_equal(got[1], want[1])
    b.close()
