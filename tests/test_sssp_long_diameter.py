"""SSSP on graphs with hubs and a long diameter: the one-launch kernel stops
when its steps stay small and the asynchronous kernel takes the rest, with and
without buckets (a far bitmap that holds vertices), zero, fractional and equal
weights, host and device results."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def line(n, hub):
    v = np.arange(n - 1)
    return n, np.concatenate([v, v + 1, np.full(hub, n // 2)]), np.concatenate([v + 1, v, (n // 2 + np.arange(hub)) % n])


def grid(k, hub):
    i = np.arange(k * k).reshape(k, k)
    a = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    b = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    return k * k, np.concatenate([a, b, np.full(hub, 7)]), np.concatenate([b, a, np.arange(hub)])


def core_and_lines(V, E, lines, length):
    """A skewed core (2^22 edges and more: buckets) with lines hanging off it."""
    rng = np.random.default_rng(E)
    src = (rng.random(E) ** 3 * V).astype(np.int64)
    dst = (rng.random(E) ** 2 * V).astype(np.int64)
    v = V + np.arange(lines * length)
    prev = np.where((v - V) % length == 0, rng.integers(0, V, lines * length), v - 1)
    return V + lines * length, np.concatenate([src, prev, v]), np.concatenate([dst, v, prev])


SHAPES = {"line": line(11000, 100), "grid": grid(150, 100), "core": core_and_lines(100000, 1 << 22, 40, 900)}


def distances(ctx, g, V, src, dst, w, s, core):
    if not core:
        return O.sssp(V, src, dst, w, s)[0]
    ctx.set_tunable("sssp_async", 0)  # the oracle's sweeps take too long here: the superstep loop
    try:
        return g.sssp([s])[0][0]
    finally:
        ctx.set_tunable("sssp_async", -1)


@pytest.mark.parametrize("weights", ["int", "zero", "fraction", "equal", "apart"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_distances_equal_the_oracle(gpu_ctx, name, weights):
    V, src, dst = SHAPES[name]
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    E = len(src)
    rng = np.random.default_rng(E)
    w = {"int": rng.integers(1, 101, E), "zero": rng.integers(0, 2, E) * 5, "fraction": rng.random(E) * 10,
         "equal": np.full(E, 2), "apart": 10.0 ** rng.integers(0, 4, E)}[weights].astype(np.float32)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    torch = pytest.importorskip("torch")
    out = torch.empty((1, V), dtype=torch.float32, device="cuda")
    degree = np.bincount(src, minlength=V)
    for s in (0, V - 1):
        want = distances(gpu_ctx, g, V, src, dst, w, s, name == "core")
        got, st = g.sssp([s])
        np.testing.assert_array_equal(got[0].view(np.uint32), want.view(np.uint32))
        assert st["kernel_launches"] > 1  # stopped, and taken on
        hit = want < api.MEDUSA_MAX
        assert st["vertices_reached"] == int(hit.sum())
        assert st["edges_traversed"] == int(degree[hit].sum())
        assert st["edges_scanned"] >= st["edges_traversed"]
        g.sssp([s], out=out)
        np.testing.assert_array_equal(out.cpu().numpy()[0].view(np.uint32), want.view(np.uint32))
    g.close()


def test_several_sources_one_by_one_and_other_runs_between(gpu_ctx):
    V, src, dst = SHAPES["line"]
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    w = np.random.default_rng(1).integers(1, 9, len(src)).astype(np.float32)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    sources = [0, 5500, 10999]
    gpu_ctx.set_batching(False)
    try:
        got, _ = g.sssp(sources)
    finally:
        gpu_ctx.set_batching(True)
    gpu_ctx.set_tunable("sssp_async", 0)  # the superstep loop, on the same state
    try:
        loop = [g.sssp([s])[0][0] for s in sources]
    finally:
        gpu_ctx.set_tunable("sssp_async", -1)
    for s, a, b in zip(sources, got, loop):
        want, _ = O.sssp(V, src, dst, w, s)
        np.testing.assert_array_equal(a, want)
        np.testing.assert_array_equal(b, want)
        np.testing.assert_array_equal(g.sssp([s])[0][0], want)
    g.close()


@pytest.mark.parametrize("knob,value", [("wait_polls", 0), ("step_cap", 30), ("step_cap", 200)])
def test_a_run_that_fails_leaves_the_next_one_right(gpu_ctx, knob, value):
    V, src, dst = SHAPES["line"]
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    w = np.ones(len(src), np.float32)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    want, _ = g.sssp([0])
    gpu_ctx.set_tunable(knob, value)
    try:
        with pytest.raises(api.MedusaError) as e:
            for _ in range(20):
                g.sssp([0])
        assert e.value.code == api.MB_ERR_TIMEOUT
    finally:
        gpu_ctx.set_tunable(knob, -1)
    np.testing.assert_array_equal(g.sssp([0])[0], want)
    g.close()
