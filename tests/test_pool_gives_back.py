"""Device memory that the library holds after its graphs are gone: 3 GB at most
while a context lives, none after the last one.  In a process of its own, where
nothing else has filled the pool."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

BODY = """
import sys
sys.path.insert(0, %r)
import torch
from medusa_b200 import api


def free():
    return torch.cuda.mem_get_info()[0]


E = 1 << 24
src = torch.randint(0, 1 << 20, (E,), dtype=torch.int32, device="cuda")
dst = torch.randint(0, 1 << 20, (E,), dtype=torch.int32, device="cuda")
small = src[:100] %% 1000
torch.cuda.synchronize()
ctx = api.Context(0)
ctx.graph_from_edges(1000, small, small).close()
at_first = free()
graphs = [ctx.graph_from_edges(1 << 20, src, dst) for _ in range(12)]
assert at_first - free() > 4 << 30, "twelve CSR pairs: 5 GB and more"
for g in graphs:
    g.close()
assert at_first - free() <= (3 << 30) + (64 << 20)
ctx.close()
assert at_first - free() <= 64 << 20
print("RIGHT")
""" % ROOT


def test_memory_of_destroyed_graphs_goes_back():
    r = subprocess.run([sys.executable, "-c", BODY], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "RIGHT" in r.stdout, r.stderr[-2000:]
