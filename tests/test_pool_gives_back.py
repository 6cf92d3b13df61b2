"""Device memory that the library holds after its graphs are gone: 3 GB at most
while a context lives, none after the last one."""
import gc

import pytest

from medusa_b200 import api

pytestmark = pytest.mark.gpu


def test_memory_of_destroyed_graphs_goes_back():
    torch = pytest.importorskip("torch")
    gc.collect()
    ctx = api.Context(0)
    E = 1 << 24
    src = torch.randint(0, 1 << 20, (E,), dtype=torch.int32, device="cuda")
    dst = torch.randint(0, 1 << 20, (E,), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.graph_from_edges(1000, src[:100] % 1000, dst[:100] % 1000).close()
    free0 = torch.cuda.mem_get_info()[0]
    graphs = [ctx.graph_from_edges(1 << 20, src, dst) for _ in range(12)]
    held = free0 - torch.cuda.mem_get_info()[0]
    assert held > 4 << 30  # twelve CSR pairs: 5 GB and more
    for g in graphs:
        g.close()
    left = free0 - torch.cuda.mem_get_info()[0]
    assert left <= (3 << 30) + (64 << 20)
    ctx.close()
