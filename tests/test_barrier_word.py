"""The grid barrier's word over long runs, on the CPU: the decisions of
medusa_b200/csrc/barrier_word.h compiled for the host, driven past the arrival
counts that a BFS or SSSP along a chain of millions of vertices reaches."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

SRC = r"""
#include "barrier_word.h"
using namespace mb;
// Barriers [first, first + n) of a run on `grid` CTAs, after each arrival a poll
// of a CTA that waits at this barrier and of one that waits at the next.  0:
// every wait ended at its own last arrival; 1: one ended early; 2: one did not end.
extern "C" int run(long long first, long long n, int grid) {
    for (long long k = first; k < first + n; k++) {
        uint32_t word = (uint32_t)((unsigned long long)k * grid);
        const uint32_t here = bar_target((uint32_t)(k + 1), grid), next = bar_target((uint32_t)(k + 2), grid);
        for (int c = 0; c < grid; c++) {
            word += 1;
            if (c + 1 < grid && bar_passed(word, here)) return 1;
            if (c + 1 == grid && !bar_passed(word, here)) return 2;
            if (bar_passed(word, next)) return 1;
        }
        // CTAs that run ahead to the next barrier keep this one passed
        for (int c = 0; c + 1 < grid; c++)
            if (!bar_passed(word += 1, here)) return 2;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def word(tmp_path_factory):
    d = tmp_path_factory.mktemp("barrier_word")
    src, lib = str(d / "w.cpp"), str(d / "w.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.check_call(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "medusa_b200", "csrc"), src,
                           "-o", lib])
    so = ctypes.CDLL(lib)
    so.run.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
    return so


@pytest.mark.parametrize("grid", [1, 16, 444, 592, 2368])
@pytest.mark.parametrize("arrivals", [0, 1 << 31, 1 << 32, 1 << 45])
def test_every_barrier_ends_with_its_own_last_arrival(word, grid, arrivals):
    first = max(arrivals // grid - 50, 0)
    assert word.run(first, 100, grid) == 0
