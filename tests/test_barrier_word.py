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
// Barriers [first, first + n) of a run on `grid` CTAs, each arrival followed by
// a poll of every CTA that waits (one of them stands for all).  0: every wait
// ended at its own last arrival; 1: one ended early; 2: one did not end;
// 3: one gave up.
extern "C" int run(long long first, long long n, int grid) {
    for (long long k = first; k < first + n; k++) {
        BarWord word = (BarWord)k * grid;
        const BarWord target = (BarWord)(k + 1) * grid;
        for (int c = 0; c < grid; c++) {
            word += 1;
            const BarWait w = bar_poll(word, target);
            if (w == BAR_GIVEN_UP) return 3;
            if (c + 1 < grid && w == BAR_PASSED) return 1;
            if (c + 1 == grid && w != BAR_PASSED) return 2;
        }
    }
    return 0;
}
// A wait that gives up: every later poll says so, whatever arrives.
extern "C" int gives_up(long long arrivals, int grid) {
    BarWord word = (BarWord)arrivals;
    word |= kBarGivenUp;
    for (int c = 0; c < grid; c++, word += 1)
        if (bar_poll(word, word & ~kBarGivenUp) != BAR_GIVEN_UP) return 0;
    return 1;
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
    so.gives_up.argtypes = [ctypes.c_longlong, ctypes.c_int]
    return so


@pytest.mark.parametrize("grid", [1, 16, 444, 592, 2368])
@pytest.mark.parametrize("arrivals", [0, 1 << 31, 1 << 32, 1 << 45])
def test_every_barrier_ends_with_its_own_last_arrival(word, grid, arrivals):
    first = max(arrivals // grid - 50, 0)
    assert word.run(first, 100, grid) == 0


@pytest.mark.parametrize("arrivals", [0, 591, 1 << 31, 1 << 45])
def test_a_barrier_given_up_ends_every_wait(word, arrivals):
    assert word.gives_up(arrivals, 592) == 1
