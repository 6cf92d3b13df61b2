"""The arrays of mb_graph_device_view are cudaMalloc's own memory (another
process can open them), keep their contents and addresses, and the graph's
runs, captured ones among them, go on after the view as before."""
import ctypes

import numpy as np
import pytest

from medusa_b200 import api

pytestmark = pytest.mark.gpu


class View(ctypes.Structure):
    ARRAYS = ("row", "col", "esrc", "rrow", "rcol", "mslot", "outdeg", "wt")
    _fields_ = [("num_vertices", ctypes.c_int32), ("num_edges", ctypes.c_int64)] + \
               [(k, ctypes.c_void_p) for k in ARRAYS]


def view(g):
    v = View()
    assert api.lib.mb_graph_device_view(g.h, ctypes.byref(v)) == api.MB_OK
    return v


def can_be_opened_elsewhere(ptr):
    from cuda.bindings import runtime as rt
    err, _ = rt.cudaIpcGetMemHandle(ptr)
    return err == rt.cudaError_t.cudaSuccess


# one CTA, the cooperative grid, the loops and the captured runs
@pytest.mark.parametrize("V,E,hub", [(900, 5000, 0), (20000, 300000, 300), (30000, 90000, 0)])
def test_view_between_runs(gpu_ctx, V, E, hub):
    rng = np.random.default_rng(V)
    src, dst = rng.integers(0, V, E).astype(np.int32), rng.integers(0, V, E).astype(np.int32)
    src[:hub] = 1
    w = rng.integers(1, 50, E).astype(np.float32)
    g = gpu_ctx.graph_from_edges(V, src, dst, w)
    sources = [1, 5, 9]

    def results():
        out = [g.bfs([1])[0], g.sssp([1])[0], g.bfs(sources)[0], g.sssp(sources)[0], g.pagerank(4)[0]]
        gpu_ctx.set_tunable("tail_edges", 1000)  # the superstep loops instead of the one-launch kernels
        try:
            out += [g.bfs([1])[0], g.sssp([1])[0]]
        finally:
            gpu_ctx.set_tunable("tail_edges", -1)
        x = g.export()
        return out + [x[k] for k in sorted(x)]

    want = results()
    v = view(g)
    for k in View.ARRAYS:
        assert can_be_opened_elsewhere(getattr(v, k)), k
    again = view(g)
    assert all(getattr(v, k) == getattr(again, k) for k in View.ARRAYS)
    for a, b in zip(want, results()):
        np.testing.assert_array_equal(a, b)
    g.close()


def test_view_amid_a_stepped_run(gpu_ctx):
    V, E = 20000, 80000
    rng = np.random.default_rng(1)
    g = gpu_ctx.graph_from_edges(V, rng.integers(0, V, E).astype(np.int32), rng.integers(0, V, E).astype(np.int32))
    want = g.bfs([2])[0][0]
    step, go = 0, True
    while go:
        go = g.superstep(api.MB_APP_BFS, step, source=2)
        if step == 1:
            view(g)
        step += 1
    np.testing.assert_array_equal(g.superstep_result(api.MB_APP_BFS)[0], want)
    g.close()
