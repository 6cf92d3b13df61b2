"""BFS on graphs with hubs whose frontiers stay small for long: supersteps of
one CTA around the size of a tile (1024 out-edges), entered and left again,
more of them than one call takes (1024), the superstep cap and a wait that
gives up inside, in a single BFS and in the many-graph call."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def chain(parts):
    """Layers of the given widths, each vertex joined to one or more of the
    next layer, and a hub beside the first vertex."""
    src, dst, first = [], [], 0
    for a, b in zip(parts, parts[1:]):
        i = np.arange(max(a, b))
        src.append(first + i % a)
        dst.append(first + a + i % b)
        first += a
    V = sum(parts) + 100
    hub = np.arange(V - 99, V)
    return V, np.concatenate(src + [np.full(99, V - 100), [0]]), np.concatenate(dst + [hub, [V - 100]])


def both(V, src, dst):
    return V, np.concatenate([src, dst]).astype(np.int32), np.concatenate([dst, src]).astype(np.int32)


SHAPES = {
    "line": chain([1] * 12000),
    "widths": chain([1] * 20 + [1023] * 15 + [1] * 15 + [1024] * 15 + [5] * 1100 + [1025] * 15 + [2] * 2200 + [6000]),
    "fan": chain([3] * 2000 + [9000] + [3] * 1500 + [9000] * 3 + [1] * 1030),
    "both ways": both(*chain([1] * 500 + [400] * 20 + [3] * 9000)),
}


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_levels_and_counts(gpu_ctx, name):
    V, src, dst = SHAPES[name]
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    g = gpu_ctx.graph_from_edges(V, src, dst)
    assert V > 10240 or len(src) > 65536  # past the one-CTA kernel
    for s in (0, 3, V // 2):
        want, _ = O.bfs(V, src, dst, [s])
        got, st = g.bfs([s])
        np.testing.assert_array_equal(got[0], want)
        hit = want >= 0
        assert st["vertices_reached"] == int(hit.sum())
        assert st["edges_traversed"] == int(np.bincount(src, minlength=V)[hit].sum())
        gpu_ctx.set_tunable("tail_edges", 2000)  # the superstep loop
        try:
            loop, lst = g.bfs([s])
        finally:
            gpu_ctx.set_tunable("tail_edges", -1)
        np.testing.assert_array_equal(loop, got)
        assert st["supersteps"] == lst["supersteps"]
        assert st["schedule_count"] == lst["schedule_count"]
    assert g.bfs([0])[1]["kernel_launches"] == 2  # the small frontiers by one CTA
    g.close()


def test_cap_and_wait_inside(gpu_ctx):
    V, src, dst = SHAPES["line"]
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    g = gpu_ctx.graph_from_edges(V, src, dst)
    want, _ = O.bfs(V, src, dst, [0])
    for knob, value in (("step_cap", 50), ("step_cap", 1500), ("wait_polls", 0)):
        gpu_ctx.set_tunable(knob, value)
        try:
            with pytest.raises(api.MedusaError):
                g.bfs([0])
        finally:
            gpu_ctx.set_tunable(knob, -1)
        np.testing.assert_array_equal(g.bfs([0])[0][0], want)
    g.close()


def test_many_graphs(gpu_ctx):
    gs = [(V, s.astype(np.int32), d.astype(np.int32)) for V, s, d in SHAPES.values()]
    b = gpu_ctx.batch_upload(gs)
    _, levels, _ = b.run(1, [0] * len(gs))
    for (V, s, d), got in zip(gs, b.split(levels)):
        np.testing.assert_array_equal(got, O.bfs(V, s, d, [0])[0])
    b.close()
