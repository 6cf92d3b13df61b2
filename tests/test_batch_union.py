"""The batch as one graph: graphs that share bitmap words and ELL groups, empty
and single-vertex graphs, hubs of more than one block, few supersteps (the
first two write the vertices without in-edges), and the grid barrier."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def graphs(seed):
    rng = np.random.default_rng(seed)
    out = [(1, 0), (1, 3), (2, 0), (7, 5), (31, 100), (33, 1), (500, 20000), (3000, 9000)]
    out += [(int(rng.integers(1, 40)), int(rng.integers(0, 120))) for _ in range(60)]
    gs = []
    for V, E in out:
        src = rng.integers(0, V, E).astype(np.int32)
        dst = np.minimum((rng.random(E) ** 4 * V).astype(np.int64), V - 1).astype(np.int32)
        gs.append((V, src, dst))
    n = 9000  # one vertex with 4097 in-edges (two blocks), one with 12288 (three)
    src = rng.integers(0, n, 4097 + 12288 + 5000).astype(np.int32)
    dst = np.concatenate([np.full(4097, 5), np.full(12288, 17), rng.integers(0, n, 5000)]).astype(np.int32)
    gs.append((n, src, dst))
    return gs


@pytest.mark.parametrize("iters", [1, 2, 3, 7])
def test_every_graph_equals_the_oracle(gpu_ctx, iters):
    gs = graphs(iters)
    b = gpu_ctx.batch_upload(gs)
    rng = np.random.default_rng(7)
    sources = np.array([rng.integers(0, V) for V, _, _ in gs], np.int32)
    try:
        ranks, levels, st = b.run(iters, sources)
        assert st["kernel_launches"] == 1
        for i, (V, src, dst) in enumerate(gs):
            want = O.pagerank(V, src, dst, iters, np.float32(1.0) / np.float32(V), order="device")
            np.testing.assert_array_equal(b.split(ranks)[i].view(np.uint32), want.view(np.uint32), err_msg="graph %d" % i)
            lv, _ = O.bfs(V, src, dst, [int(sources[i])])
            np.testing.assert_array_equal(b.split(levels)[i], lv, err_msg="graph %d" % i)
        again, levels2, _ = b.run(iters, sources)
        np.testing.assert_array_equal(ranks, again)
        np.testing.assert_array_equal(levels, levels2)
    finally:
        b.close()


def test_grid_barrier_gives_up_and_recovers(gpu_ctx):
    b = gpu_ctx.batch_upload(graphs(3))
    try:
        want, lv, _ = b.run(4)
        gpu_ctx.set_tunable("wait_polls", 0)
        with pytest.raises(api.MedusaError) as e:
            for _ in range(20):  # a wait of no polls ends well only if every CTA arrived before
                b.run(4)
        assert e.value.code == api.MB_ERR_TIMEOUT
        gpu_ctx.set_tunable("wait_polls", -1)
        got, lv2, _ = b.run(4)
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(lv2, lv)
    finally:
        gpu_ctx.set_tunable("wait_polls", -1)
        b.close()
