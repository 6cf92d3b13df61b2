"""Device arrays at addresses that are no multiple of their elements' size (a
view into a packed buffer) go through a copy, as edges in and as results out,
for every route of BFS and SSSP, PageRank and the many-graph call."""
import numpy as np
import pytest

from medusa_b200 import api

pytestmark = pytest.mark.gpu


class Packed:
    """A 4-byte array at an odd offset of a device buffer."""

    def __init__(self, torch, shape, dtype, offset, values=None):
        self.torch, self.shape, self.dtype, self.offset = torch, shape, dtype, offset
        self.n = 4 * int(np.prod(shape))
        self.buf = torch.zeros(self.n + 16, dtype=torch.uint8, device="cuda")
        if values is not None:
            self.buf[offset:offset + self.n] = torch.from_numpy(
                np.ascontiguousarray(values, dtype).view(np.uint8).ravel().copy()).cuda()

    def data_ptr(self):
        return self.buf.data_ptr() + self.offset

    def is_contiguous(self):
        return True

    def numpy(self):
        b = self.buf.cpu().numpy()
        assert not b[:self.offset].any() and not b[self.offset + self.n:].any()
        return b[self.offset:self.offset + self.n].copy().view(self.dtype).reshape(self.shape)


# one CTA; the cooperative grid (a hub); the asynchronous kernel (hub-free)
@pytest.mark.parametrize("V,E,hub", [(500, 2500, 0), (30000, 300000, 500), (40000, 120000, 0)])
@pytest.mark.parametrize("offset", [1, 2, 7])
def test_edges_and_results_off_alignment(gpu_ctx, V, E, hub, offset):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(V + offset)
    src, dst = rng.integers(0, V, E).astype(np.int32), rng.integers(0, V, E).astype(np.int32)
    src[:hub] = 3
    w = rng.integers(1, 100, E).astype(np.float32)
    ref = gpu_ctx.graph_from_edges(V, src, dst, w)
    packed = [Packed(torch, x.shape, x.dtype, offset, x) for x in (src, dst, w)]
    torch.cuda.synchronize()
    g = gpu_ctx.graph_from_edges(V, *packed)
    a, b = ref.export(), g.export()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k])
    for sources in ([3], [3, 11, 200]):
        for f, want, dtype in ((g.bfs, ref.bfs(sources)[0], np.int32), (g.sssp, ref.sssp(sources)[0], np.float32)):
            out = Packed(torch, want.shape, dtype, offset)
            torch.cuda.synchronize()
            f(sources, out=out)
            np.testing.assert_array_equal(out.numpy(), want)
    out = Packed(torch, (V,), np.float32, offset)
    torch.cuda.synchronize()
    g.pagerank(3, out=out)
    np.testing.assert_array_equal(out.numpy(), ref.pagerank(3)[0])
    b = gpu_ctx.batch_upload([(V, src, dst), (2, np.array([0], np.int32), np.array([1], np.int32))])
    ranks, levels, _ = b.run(2, [3, 0])
    r, l = Packed(torch, ranks.shape, np.float32, offset), Packed(torch, levels.shape, np.int32, offset)
    torch.cuda.synchronize()
    b.run(2, [3, 0], r, l)
    np.testing.assert_array_equal(r.numpy(), ranks)
    np.testing.assert_array_equal(l.numpy(), levels)
    b.close()
    ref.close()
    g.close()
