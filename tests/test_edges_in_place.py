"""mb_graph_from_edges reads the caller's device arrays in place: arrays that
another stream rewrites during the call, ids out of range among them, give an
error or a graph whose arrays are consistent, and nothing else."""
import numpy as np
import pytest

from medusa_b200 import api

pytestmark = pytest.mark.gpu


def consistent(g):
    x = g.export()
    V, E = g.V, g.E
    for row, ids in ((x["row"], x["col"]), (x["rrow"], x["rcol"])):
        assert row[0] == 0 and row[V] == E and (np.diff(row) >= 0).all()
        assert ids.min() >= 0 and ids.max() < V
    assert (np.sort(x["mslot"]) == np.arange(E)).all()


@pytest.mark.parametrize("V", [200, 70000])
@pytest.mark.parametrize("weighted", [True, False], ids=["weighted", "unit"])
def test_arrays_that_change_during_the_build(V, weighted):
    torch = pytest.importorskip("torch")
    E = 1 << 21
    gen = torch.Generator(device="cuda").manual_seed(V)
    good = torch.randint(0, V, (E,), dtype=torch.int32, device="cuda", generator=gen)
    other = torch.randint(0, V, (E,), dtype=torch.int32, device="cuda", generator=gen)
    bad = other.clone()
    bad[::1000] = V + 7
    bad[1::1000] = -1
    src, dst = good.clone(), other.clone()
    w = torch.rand(E, device="cuda", generator=gen) if weighted else None
    ctx = api.Context(0)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    built = failed = 0
    for i in range(12):
        with torch.cuda.stream(side):
            for k in range(60):  # some milliseconds of writes
                (src if i % 2 else dst).copy_((other, good, bad)[k % (3 if i % 3 else 2)])
        try:
            g = ctx.graph_from_edges(V, src, dst, w)
            consistent(g)
            g.close()
            built += 1
        except api.MedusaError:
            failed += 1
        side.synchronize()
        src.copy_(good)
        dst.copy_(other)
        torch.cuda.synchronize()
    assert built + failed == 12
    g = ctx.graph_from_edges(V, src, dst, w)  # the context is as good as before
    consistent(g)
    g.close()
    ctx.close()


@pytest.mark.parametrize("which", ["src", "dst"])
@pytest.mark.parametrize("value", [1000, 1 << 20, -1])
def test_ids_out_of_range_are_refused(gpu_ctx, which, value):
    torch = pytest.importorskip("torch")
    V, E = 1000, 9001
    rng = np.random.default_rng(5)
    e = {"src": rng.integers(0, V, E).astype(np.int32), "dst": rng.integers(0, V, E).astype(np.int32)}
    e[which][E - 1] = value
    for args in ((e["src"], e["dst"]), [torch.from_numpy(e[k]).cuda() for k in ("src", "dst")]):
        torch.cuda.synchronize()
        with pytest.raises(api.MedusaError):
            gpu_ctx.graph_from_edges(V, *args)
