"""PageRank with all supersteps in one launch, and the launches per superstep
that replace it past the resident warps: group edges (32 vertices per warp),
vertices without in- or out-edges, both orders; and its bounded barrier."""
import numpy as np
import pytest

from medusa_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu

WARPS = 148 * 64  # resident warps, one group of 32 vertices each


def ring_graph(V, rng):
    """Every vertex but the last third of a tenth has 2 in-edges; some have no out-edges."""
    with_in = V if V < 40 else V - V // 30
    dst = np.repeat(rng.permutation(V)[:with_in], 2)
    senders = max(1, V - V // 10)
    src = rng.integers(0, senders, len(dst))
    return src.astype(np.int32), dst.astype(np.int32)


@pytest.mark.parametrize("order", ["reference", "device"])
@pytest.mark.parametrize("V", [1, 31, 32, 33, 1025, 32 * WARPS, 32 * WARPS + 32 * (WARPS // 20)])
def test_ranks_equal_the_oracle(gpu_ctx, V, order):
    src, dst = ring_graph(V, np.random.default_rng(V))
    g = gpu_ctx.graph_from_edges(V, src, dst)
    gpu_ctx.set_pagerank_order(api.MB_PR_ORDER_REFERENCE if order == "reference" else api.MB_PR_ORDER_FIXED)
    try:
        for iters in (1, 2, 3, 5):
            rank, _ = g.pagerank(iters)
            want = O.pagerank(V, src, dst, iters, np.float32(1.0 / V), order=order)
            np.testing.assert_array_equal(rank, want, err_msg="%d supersteps" % iters)
    finally:
        gpu_ctx.set_pagerank_order(api.MB_PR_ORDER_REFERENCE)
    g.close()


def test_barrier_gives_up_and_recovers(gpu_ctx):
    V = 20000
    src, dst = ring_graph(V, np.random.default_rng(3))
    g = gpu_ctx.graph_from_edges(V, src, dst)
    want, _ = g.pagerank(4)
    gpu_ctx.set_tunable("wait_polls", 0)
    try:
        with pytest.raises(api.MedusaError) as e:
            for _ in range(20):  # a wait of no polls ends well only if every CTA arrived before
                g.pagerank(4)
        assert e.value.code == api.MB_ERR_TIMEOUT
    finally:
        gpu_ctx.set_tunable("wait_polls", -1)
    got, _ = g.pagerank(4)
    np.testing.assert_array_equal(got, want)
    g.close()


ONE_CTA = 148 * 32  # warps of one full CTA per SM


@pytest.mark.parametrize("order", ["reference", "device"])
@pytest.mark.parametrize("groups", [ONE_CTA, ONE_CTA + 1, ONE_CTA + 147, ONE_CTA + 149, WARPS - 148, WARPS - 147])
def test_groups_spread_over_two_ctas_per_sm(gpu_ctx, groups, order):
    V = 32 * groups - 7
    rng = np.random.default_rng(groups)
    src, dst = rng.integers(0, V - V // 10, 3 * V).astype(np.int32), rng.integers(0, V - V // 50, 3 * V).astype(np.int32)
    g = gpu_ctx.graph_from_edges(V, src, dst)
    gpu_ctx.set_pagerank_order(api.MB_PR_ORDER_REFERENCE if order == "reference" else api.MB_PR_ORDER_FIXED)
    try:
        rank, _ = g.pagerank(4)
        np.testing.assert_array_equal(rank, O.pagerank(V, src, dst, 4, np.float32(1.0 / V), order=order))
    finally:
        gpu_ctx.set_pagerank_order(api.MB_PR_ORDER_REFERENCE)
    g.close()


def test_one_group_more_than_a_cta_per_sm_takes_no_leap(gpu_ctx):
    # 13.1 and 13.8 us per superstep; 23.3 where five SMs had two CTAs of 32 warps
    ms = []
    for groups in (ONE_CTA - 40, ONE_CTA + 134):
        V = 32 * groups
        rng = np.random.default_rng(7)
        g = gpu_ctx.graph_from_edges(V, rng.integers(0, V, 21 * V).astype(np.int32), rng.integers(0, V, 21 * V).astype(np.int32))
        g.pagerank(10)
        ms.append(np.median([g.pagerank(10)[1]["device_ms"] for _ in range(9)]))
        g.close()
    assert ms[1] < 1.4 * ms[0], ms
