"""The draw of a triangle or varying record (rz_draws.h, which the kernels include) on the CPU:
the right draw for lists of any draws, without more loads than a binary search would take."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

HARNESS = r"""
#include "rz_draws.h"
// base[n], items 0 .. items - 1: the draw of each item and the loads of the list it took
extern "C" void lookup(const uint32_t* base, uint32_t n, uint32_t items, uint32_t* draw, uint32_t* loads) {
    std::vector<uint32_t> table{7u};  // tables follow one another
    rz::add_draw_table(table, n, items, [&](uint32_t d) { return base[d]; });
    for (uint32_t i = 0; i < items; ++i) {
        uint32_t count = 0;
        draw[i] = rz::draw_in_table(i, [&](uint32_t g) { return table.at(1 + g); },
                                    [&](uint32_t d) { ++count; return base[d]; });
        loads[i] = count;
    }
}
"""


@pytest.fixture(scope="module")
def lookup(tmp_path_factory):
    d = tmp_path_factory.mktemp("draws")
    (d / "h.cpp").write_text(HARNESS)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rosy_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", csrc, "-o", str(d / "h.so"), str(d / "h.cpp")],
                   check=True)
    fn = C.CDLL(str(d / "h.so")).lookup

    def call(lengths):
        base = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32)
        n, items = len(lengths), int(base[-1])
        draw, loads = np.zeros(items, np.uint32), np.zeros(items, np.uint32)
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        fn(p(base), n, items, p(draw), p(loads))
        return base[:-1], draw, loads

    return call


@pytest.mark.parametrize("lengths", [
    [1], [255], [256], [257], [1] * 1000, [2] * 700, [12] * 100, [4096] * 20, [0] * 300 + [256], [256] + [0] * 5000 + [3],
    [255, 1, 0, 0, 256, 0, 257], [0, 0, 1, 0]] + [list(np.random.default_rng(k).integers(0, 1 << k, 400)) for k in range(1, 11)])
def test_draw_of_every_item(lookup, lengths):
    base, draw, loads = lookup(lengths)
    items = np.arange(len(draw))
    assert np.array_equal(draw, np.searchsorted(base, items, side="right") - 1)
    # the draws that an item's 256 can belong to: those that start in them, and the one before
    first = items // 256 * 256
    candidates = np.searchsorted(base, first + 256, side="right") - np.searchsorted(base, first, side="right") + 1
    assert (loads <= np.ceil(np.log2(candidates))).all()
    assert loads.max() <= math.ceil(math.log2(max(len(lengths), 2)))
