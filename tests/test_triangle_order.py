"""The host-side triangle order of the tiled assembly, compiled by itself: every triangle once, regular meshes
ordered as without the bound on a dof's open triangles, and an apex shared by 20 000 triangles in linear time."""
from __future__ import annotations

import ctypes
import subprocess
import time

import numpy as np
import pytest

from conftest import REPO, golden_buffers

SOURCE = r"""
#include "triangle_order.h"
extern "C" int scan_bound() { return hbem::kOrderScan; }
extern "C" void order(const int *l2g, int T, int n_dof, int scan, int *out) {
    std::vector<int> seed(T), result;
    for (int t = 0; t < T; ++t) seed[t] = t;
    hbem::cluster_order(std::vector<int>(l2g, l2g + 3 * T), n_dof, seed, 8, 32, scan, result);
    std::copy(result.begin(), result.end(), out);
}
"""


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "order.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O3", "-std=c++17", "-shared", "-fPIC", "-I", str(REPO / "hornlab_metal_bem_b200" / "csrc"),
                    str(d / "order.cpp"), "-o", str(d / "order.so")], check=True)
    lib = ctypes.CDLL(str(d / "order.so"))

    def call(l2g, scan=None):
        l2g = np.ascontiguousarray(l2g, np.int32)
        out = np.empty(len(l2g), np.int32)
        lib.order(ctypes.c_void_p(l2g.ctypes.data), len(l2g), int(l2g.max()) + 1,
                  lib.scan_bound() if scan is None else scan, ctypes.c_void_p(out.ctypes.data))
        return out

    return call


@pytest.mark.parametrize("name", ["tiny", "ico2", "horn_quarter", "horn_full"])
def test_regular_meshes_keep_their_order(order, name):
    l2g = np.asarray(golden_buffers(name).p1_local2global_i32).reshape(-1, 3)
    got = order(l2g)
    assert np.array_equal(np.sort(got), np.arange(len(l2g)))
    assert np.array_equal(got, order(l2g, scan=1 << 30))


def test_apex_of_many_triangles(order):
    n = 20000
    i = np.arange(n)
    l2g = np.stack([i, (i + 1) % n, np.full(n, n)], 1)
    t0 = time.perf_counter()
    got = order(l2g)
    assert time.perf_counter() - t0 < 1.0   # 0.05 s; 4 s where each step looked at all of them
    assert np.array_equal(np.sort(got), i)
