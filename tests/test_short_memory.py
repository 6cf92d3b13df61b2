"""Calls that have a form with less device memory take it when the other one
does not fit: the batched BFS without kept frontiers, SSSP with fewer sources
at a time, many graphs by teams.  Each runs in a process of its own, whose
other memory is taken away first."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HEAD = """
import sys
sys.path.insert(0, %r)
import numpy as np
import torch
from medusa_b200 import api


def take_all_but(mb):
    torch.cuda.synchronize()
    return torch.empty(torch.cuda.mem_get_info()[0] - (mb << 20), dtype=torch.uint8, device="cuda")


def edges(V, E, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(0, V, E).astype(np.int32), rng.integers(0, V, E).astype(np.int32)


ctx = api.Context(0)
""" % ROOT

CASES = {
    "batched bfs": """
V, E, n = 1 << 22, 1 << 20, 8
src, dst = edges(V, E, 1)
src[:400000] = 7  # dense supersteps
g = ctx.graph_from_edges(V, src, dst)
sources = [7, 1, 2, int(src[-1]), 3, 4, 5, 6]
want = [g.bfs([s])[0][0] for s in sources]
g.close()
g = ctx.graph_from_edges(V, src, dst)
hold = take_all_but(480)  # 218 MB of state and 134 of results; 268 more for the kept frontiers
got, _ = g.bfs(sources)
for a, b in zip(got, want):
    np.testing.assert_array_equal(a, b)
""",
    "sssp pairs": """
V, E, n = 1 << 20, 1 << 21, 32
src, dst = edges(V, E, 2)
w = np.random.default_rng(2).integers(1, 100, E).astype(np.float32)
g = ctx.graph_from_edges(V, src, dst, w)
sources = list(range(100, 100 + n))
want, _ = g.sssp(sources)
g.close()
g = ctx.graph_from_edges(V, src, dst, w)
out = np.empty((n, V), np.float32)
hold = take_all_but(300)  # 906 MB for 32 sources
got, _ = g.sssp(sources, out=out)
np.testing.assert_array_equal(got, want)
""",
    "many graphs": """
gs = [(1 << 18,) + edges(1 << 18, 1 << 22, s) for s in range(4)]
sources = [int(s[0]) for _, s, _ in gs]
b = ctx.batch_upload(gs)
want = b.run(3, sources)
b.close()
b = ctx.batch_upload(gs)
hold = take_all_but(60)  # 270 MB for the union
for _ in range(2):
    got = b.run(3, sources)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
""",
}
# the pool's memory of the first run is given back before the second
TRIM = "ctx.close()\nctx = api.Context(0)\n"


@pytest.mark.parametrize("case", sorted(CASES))
def test_the_smaller_form_gives_the_same(case):
    body = CASES[case].replace("g.close()\n", "g.close()\n" + TRIM).replace("b.close()\n", "b.close()\n" + TRIM)
    r = subprocess.run([sys.executable, "-c", HEAD + body + "print('RIGHT')\n"], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "RIGHT" in r.stdout, r.stderr[-3000:]
