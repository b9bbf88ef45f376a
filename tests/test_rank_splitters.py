"""The splitters of the basin tree's ranking (rank_splitter in csrc/fsb_routing.cu), on the
CPU: one entry of every group, inside the list, and no list in a regular order
goes far without meeting one -- a walk between two of them is one thread's
serial chain of loads.  With one of 16 entries a splitter, n/16 walks of random
length have their longest at about 16 ln(n/16); the bound is twice that.  (The
entries' successors in the basin tree's tour are regular: along a chain of basins
in the order of their heights every second entry, forwards or backwards.)"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "fastscapelib-fortran_b200", "csrc", "fsb_routing.cu")


@pytest.fixture(scope="module")
def splitters(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    text = open(SRC).read()
    i = text.index("template <int STRIDE, bool DRAWN>\n__host__ __device__ inline size_t rank_splitter")
    code = text[i:text.index("\n}\n", i) + 3].replace("__host__ __device__ ", "")
    d = tmp_path_factory.mktemp("splitters")
    cpp, so = d / "s.cpp", d / "s.so"
    cpp.write_text("#include <cstddef>\n" + code + 'extern "C" size_t splitter(int stride, unsigned t, size_t n) '
                   "{ return stride == 16 ? rank_splitter<16, true>(t, n) : rank_splitter<4, true>(t, n); }\n")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(cpp)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.splitter.argtypes = [ctypes.c_int, ctypes.c_uint, ctypes.c_size_t]
    lib.splitter.restype = ctypes.c_size_t
    return lib.splitter


@pytest.mark.parametrize("stride,n", [(4, 8193), (4, 32001), (16, 33000), (16, 65535), (16, 400007)])
def test_regular_lists_meet_splitters(splitters, stride, n):
    groups = (n + stride - 1) // stride
    at = np.array([splitters(stride, t, n) for t in range(groups)])
    assert np.all(at // stride == np.arange(groups)) and at.max() < n
    is_split = np.zeros(n, bool)
    is_split[at] = True
    bound = 2 * stride * np.log(groups)
    for step in (1, 2, 3, 4, 8, 16, 32, 48):  # successors this far apart
        for first in range(min(step, 6)):
            order = np.arange(first, n, step)
            for o in (order, order[::-1]):
                hits = np.flatnonzero(is_split[o])
                gaps = np.diff(np.concatenate(([0], hits, [o.size])))
                assert gaps.max() <= bound, (step, first, gaps.max())
