"""BFS in one launch: the one-CTA kernel (graph staged in shared memory or
not), the cooperative grid past its limits, every mix of directions, list
lengths at the pull's edges, host and device outputs, and the grid barrier."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def skewed(V, E, seed):
    rng = np.random.default_rng(seed)
    src = np.minimum((rng.random(E) ** 3 * V).astype(np.int64), V - 1).astype(np.int32)
    dst = np.minimum((rng.random(E) ** 2 * V).astype(np.int64), V - 1).astype(np.int32)
    return src, dst


# the one-CTA kernel takes V <= 10240 and E <= 65536; it stages the graph
# where 24 V + 4 E bytes fit in 220 KB
SIZES = [(1, 0), (1, 3), (2, 1), (31, 64), (33, 500), (1024, 8192), (4096, 30000), (4096, 33000),
         (10240, 65536), (10240, 65537), (10241, 60000), (40000, 500000), (200000, 1500001)]


@pytest.mark.parametrize("rule", ["default", "push", "pull", "back"])
@pytest.mark.parametrize("V,E", SIZES)
def test_levels_equal_the_oracle(gpu_ctx, V, E, rule):
    src, dst = skewed(V, E, V + E)
    g = gpu_ctx.graph_from_edges(V, src, dst)
    if rule == "push":
        gpu_ctx.set_tunable("bfs_alpha", 0)
    elif rule != "default":  # pulls from the start; "back": and pushes as soon as the frontier shrinks
        gpu_ctx.set_tunable("bfs_alpha", 1 << 20)
        gpu_ctx.set_tunable("bfs_gamma", 0)
        gpu_ctx.set_tunable("bfs_beta", (1 << 20) if rule == "pull" else 1)
    try:
        torch = pytest.importorskip("torch")
        out = torch.empty((1, V), dtype=torch.int32, device="cuda")
        aa = O.AAGraph(V, src, dst, None)
        degree = np.bincount(src, minlength=V)
        for s in {0, V // 2, V - 1}:
            want, _ = O.bfs(V, aa, None, [s])
            got, st = g.bfs([s])
            np.testing.assert_array_equal(got[0], want)
            assert st["vertices_reached"] == int((want >= 0).sum())
            assert st["edges_traversed"] == int(degree[want >= 0].sum())
            g.bfs([s], out=out)
            np.testing.assert_array_equal(out.cpu().numpy()[0], want)
    finally:
        for t in ("bfs_alpha", "bfs_gamma", "bfs_beta"):
            gpu_ctx.set_tunable(t, -1)
    g.close()


@pytest.mark.parametrize("rows,cols", [(1, 2), (1, 10240), (100, 102), (100, 103), (128, 80)])
def test_hub_free_lattices(gpu_ctx, rows, cols):
    """Both sides of the one-CTA kernel's vertex limit, long diameters."""
    V = rows * cols
    i = np.arange(V, dtype=np.int32).reshape(rows, cols)
    a = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    b = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    src, dst = np.concatenate([a, b]), np.concatenate([b, a])
    g = gpu_ctx.graph_from_edges(V, src, dst)
    s = V // 3
    want = (np.abs(i // cols - s // cols) + np.abs(i % cols - s % cols)).astype(np.int32).ravel()
    got, st = g.bfs([s])
    np.testing.assert_array_equal(got[0], want)
    assert st["vertices_reached"] == V and st["edges_traversed"] == len(src)
    g.close()


def test_pull_list_lengths(gpu_ctx):
    """In-lists whose only visited source is the last one."""
    lengths = [1, 2, 4, 5, 31, 32, 33, 34, 159, 160, 161, 1000]
    n, pad = len(lengths), 20000  # past the one-CTA kernel
    src, dst = [], []
    hub = n + max(lengths)  # the largest source id of every list: tested last
    for i, k in enumerate(lengths):
        src += list(range(n, n + k - 1)) + [hub]
        dst += [i] * k
    V = hub + 1 + pad
    src, dst = np.array(src, np.int32), np.array(dst, np.int32)
    g = gpu_ctx.graph_from_edges(V, src, dst)
    gpu_ctx.set_tunable("bfs_alpha", 1 << 20)
    gpu_ctx.set_tunable("bfs_gamma", 0)
    gpu_ctx.set_tunable("bfs_async", 0)  # the asynchronous kernel's by default: no hubs
    try:
        got, st = g.bfs([hub])
    finally:
        gpu_ctx.set_tunable("bfs_async", -1)
        gpu_ctx.set_tunable("bfs_alpha", -1)
        gpu_ctx.set_tunable("bfs_gamma", -1)
    assert st["schedule_count"][4] > 0
    want = np.full(V, -1, np.int32)
    want[:n], want[hub] = 1, 0
    np.testing.assert_array_equal(got[0], want)
    g.close()


def test_grid_barrier_gives_up_and_recovers(gpu_ctx):
    V, E = 100000, 800000
    src, dst = skewed(V, E, 9)
    g = gpu_ctx.graph_from_edges(V, src, dst)
    want, _ = g.bfs([0])
    gpu_ctx.set_tunable("wait_polls", 0)
    try:
        with pytest.raises(api.MedusaError) as e:
            for _ in range(20):  # a wait of no polls ends well only if every CTA arrived before
                g.bfs([0])
        assert e.value.code == api.MB_ERR_TIMEOUT
    finally:
        gpu_ctx.set_tunable("wait_polls", -1)
    got, _ = g.bfs([0])
    np.testing.assert_array_equal(got, want)
    g.close()
