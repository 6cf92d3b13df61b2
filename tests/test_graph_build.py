"""Graph construction against numpy's stable sorts: sort tiles (4096 elements)
and their remainders, every number of digit passes, skewed and single keys,
gaps without edges, both orders, host and device arrays."""
import numpy as np
import pytest

from medusa_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,E", [(1, 1), (1, 5000), (2, 4095), (3, 4096), (200, 4097), (256, 70000), (257, 8192),
                                 (65536, 12289), (65537, 100001), (1 << 20, 33), (1 << 24, 20000),
                                 (1 << 24 | 1, 300000)])
@pytest.mark.parametrize("reference", [True, False], ids=["reference", "input"])
@pytest.mark.parametrize("weighted", [True, False], ids=["weighted", "unit"])
def test_export_equals_numpy(gpu_ctx, V, E, reference, weighted):
    rng = np.random.default_rng(V + E)
    # squared: low ids far more often
    src = np.minimum((rng.random(E) ** 2 * V).astype(np.int64), V - 1).astype(np.int32)
    dst = rng.integers(0, V, E).astype(np.int32)
    w = rng.integers(1, 1000, E).astype(np.float32) if weighted else None
    if E % 2:
        torch = pytest.importorskip("torch")
        args = [torch.from_numpy(x).cuda() if x is not None else None for x in (src, dst, w)]
        torch.cuda.synchronize()
    else:
        args = [src, dst, w]
    g = gpu_ctx.graph_from_edges(V, *args, reference_order=reference)
    got = g.export()
    order = np.arange(E)[::-1] if reference else np.arange(E)
    order = order[np.argsort(src[order], kind="stable")]
    s, d = src[order], dst[order]
    ww = w[order] if weighted else np.ones(E, np.float32)
    np.testing.assert_array_equal(got["row"], np.concatenate([[0], np.cumsum(np.bincount(s, minlength=V))]))
    np.testing.assert_array_equal(got["col"], d)
    np.testing.assert_array_equal(got["w"], ww)
    back = np.argsort(d, kind="stable")
    np.testing.assert_array_equal(got["rrow"], np.concatenate([[0], np.cumsum(np.bincount(d, minlength=V))]))
    np.testing.assert_array_equal(got["rcol"], s[back])
    slot = np.empty(E, np.int64)
    slot[back] = np.arange(E)
    np.testing.assert_array_equal(got["mslot"], slot)
    if args[0] is not src:  # the caller's arrays are only read
        np.testing.assert_array_equal(args[0].cpu().numpy(), src)
        np.testing.assert_array_equal(args[1].cpu().numpy(), dst)
    g.close()
