"""One graph ranked from several contexts: the captured run kept on the graph
belongs to the context that captured it (its wait limit, its tunables, its
error word), also when the contexts' tunables changed equally often and after
the first context is gone."""
import numpy as np
import pytest

from medusa_b200 import api

pytestmark = pytest.mark.gpu


def lend(ctx, g):
    """g's handle under another context; the caller gives it back."""
    other = api.Graph(ctx, g.h.value)
    return other


def give_back(*lent):
    for g in lent:
        g.h = None


def make(ctx, V, E, seed, hub=0):
    rng = np.random.default_rng(seed)
    src, dst = rng.integers(0, V, E), rng.integers(0, V, E)
    dst[:hub] = 5
    return ctx.graph_from_edges(V, src.astype(np.int32), dst.astype(np.int32))


@pytest.mark.parametrize("order", [api.MB_PR_ORDER_REFERENCE, api.MB_PR_ORDER_FIXED])
def test_a_wait_that_gives_up_is_the_running_contexts(order):
    a, b = api.Context(0), api.Context(0)
    a.set_pagerank_order(order)
    b.set_pagerank_order(order)
    a.set_tunable("batch_threads", 256)  # as many changes as b's, and none to a run
    b.set_tunable("wait_polls", 0)
    g = make(a, 4000, 60000, 1)
    want, _ = g.pagerank(7)
    gb = lend(b, g)
    with pytest.raises(api.MedusaError):
        gb.pagerank(7)
    np.testing.assert_array_equal(g.pagerank(7)[0], want)
    b.set_tunable("wait_polls", -1)
    np.testing.assert_array_equal(gb.pagerank(7)[0], want)
    give_back(gb)
    g.close()
    a.close()
    b.close()


def test_the_graph_outlives_the_context_that_captured():
    a, b = api.Context(0), api.Context(0)
    g = make(a, 4000, 60000, 2)
    want, _ = g.pagerank(7)
    gb = lend(b, g)
    a.close()
    np.testing.assert_array_equal(gb.pagerank(7)[0], want)
    give_back(g)
    gb.close()
    b.close()


def test_hub_lists_of_two_contexts_in_turn():
    a, b = api.Context(0), api.Context(0)
    a.set_tunable("pr_hub_min", 64)
    b.set_tunable("pr_hub_min", 700)
    g = make(a, 3000, 40000, 3, hub=5000)
    gb = lend(b, g)
    want, _ = g.pagerank(5)
    for _ in range(2):
        np.testing.assert_array_equal(gb.pagerank(5)[0], want)
        np.testing.assert_array_equal(g.pagerank(5)[0], want)
    give_back(gb)
    g.close()
    a.close()
    b.close()
