"""Sources per run of the one-launch SSSP (medusa_b200/csrc/pairs_limit.h on the
host): every edge number of a run's largest queue, rounded up to whole tiles,
stays inside signed 32 bits."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

TILE = 1024  # edges of a tile of the kernel, or more


@pytest.fixture(scope="module")
def sources(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs_limit")
    src, lib = str(d / "p.cpp"), str(d / "p.so")
    with open(src, "w") as f:
        f.write('#include "pairs_limit.h"\nextern "C" int sources(int V, long long E) '
                "{ return mb::pairs_sources(V, E); }\n")
    subprocess.check_call(["g++", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "medusa_b200", "csrc"), src,
                           "-o", lib])
    so = ctypes.CDLL(lib)
    so.sources.argtypes = [ctypes.c_int, ctypes.c_longlong]
    return so.sources


@pytest.mark.parametrize("V", [1, 1000, 1 << 20, (1 << 20) + 1, 1 << 24, 1 << 25, (1 << 31) - 1])
@pytest.mark.parametrize("E", [0, 1, 1 << 24, (1 << 26) - 1, 1 << 26, (1 << 27) - 1, 1 << 27, 1 << 30, (1 << 31) - 1])
def test_edge_numbers_stay_in_range(sources, V, E):
    n = sources(V, E)
    assert 1 <= n <= 32
    last = n * E - 1
    assert last < 1 << 31
    if n > 1:
        assert n * V <= 1 << 25
    assert n * E + TILE - 1 < 1 << 32  # the unsigned rounding up


@pytest.mark.parametrize("V,E,n", [(1 << 20, 1 << 24, 32), (1 << 22, 1 << 26, 8), (1 << 20, 1 << 26, 31),
                                   (1 << 20, (1 << 27) - 1, 16), (1 << 26, 1 << 28, 1)])
def test_ordinary_graphs_keep_their_sources(sources, V, E, n):
    assert sources(V, E) == n
