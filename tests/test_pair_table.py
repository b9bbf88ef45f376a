"""The table of basin pairs (ht_insert / ht_find in csrc/fsb_locmin.cu) where
many basins in a row own more pairs than the eight slots each has: a strip three
nodes wide between two open sides.  Every pair must find a place whatever the
neighbouring basins' slots hold.  On the CPU the functions are compiled for the
host; on the GPU one step of such grids is compared with the oracle, receivers
and sorted passes bit for bit."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from fastscapelib_fortran import workloads as W
from test_nr_level_emulation import SRC, _between

DRIVER = r"""
#include <cstddef>
#include <cstdlib>
#define __device__
#define __forceinline__ inline
#define __restrict__
struct ulonglong2 { unsigned long long x, y; };
static unsigned long long atomicCAS(unsigned long long* p, unsigned long long c, unsigned long long v) {
  const unsigned long long o = *p;
  if (o == c) *p = v;
  return o;
}
@code@
// inserts every pair twice and finds it again; returns the pairs that went wrong
extern "C" int fill(size_t cap, int n, const int* b, const int* nb) {
  unsigned long long* keys = static_cast<unsigned long long*>(std::aligned_alloc(64, cap * 8));
  for (size_t s = 0; s < cap; ++s) keys[s] = ~0ull;
  int bad = 0;
  for (int pass = 0; pass < 2; ++pass)
    for (int e = 0; e < n; ++e) {
      const unsigned long long key = (unsigned long long)b[e] << 32 | (unsigned)nb[e];
      const unsigned s = ht_insert(keys, cap, key);
      bad += s == 0xffffffffu || keys[s] != key || ht_find(keys, cap, key) != s;
    }
  bad += ht_find(keys, cap, 0x12345ull << 40) != 0xffffffffu;  // a pair that is not there
  std::free(keys);
  return bad;
}
"""


@pytest.fixture(scope="module")
def table(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    text = open(SRC).read()
    code = _between(text, "__device__ inline unsigned long long mix64", "// ---- basins", False)
    code += _between(text, "constexpr int kPairSlots", "// pass 0: insert pairs", False)
    d = tmp_path_factory.mktemp("pairs")
    cpp, so = d / "pairs.cpp", d / "pairs.so"
    cpp.write_text(DRIVER.replace("@code@", code))
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-w", "-o", str(so), str(cpp)], check=True)
    lib = ctypes.CDLL(str(so))
    pi = ctypes.POINTER(ctypes.c_int)
    lib.fill.argtypes = [ctypes.c_size_t, ctypes.c_int, pi, pi]
    return lib


@pytest.mark.parametrize("first,rows,pairs", [(1, 400, 12), (5000, 2000, 12), (60000, 6667, 10), (1, 30000, 6)])
def test_runs_of_basins_with_many_pairs(table, first, rows, pairs):
    b = np.repeat(np.arange(first, first + rows, dtype=np.int32), pairs)
    nb = (b + first + rows + np.tile(np.arange(pairs), rows) * 7).astype(np.int32)
    nroots, cap = max(int(b.max()), rows * pairs // 6), 1024
    while cap < 8 * (nroots + 1):
        cap *= 2
    ptr = lambda a: np.ascontiguousarray(a).ctypes.data_as(ctypes.POINTER(ctypes.c_int))  # noqa: E731
    assert table.fill(cap, b.size, ptr(b), ptr(nb)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(60000, 3), (3, 60000), (9001, 4)])
def test_strip_matches_oracle(nx, ny):
    import fastscapelib_fortran as fs
    wl = W.mfd(nx, ny, seed=7, p=-2.0)  # single flow
    wl.apply(O)
    O.fastscape_execute_step()
    g = fs.FastScape(0)
    g.set_nx_ny(nx, ny)
    g.setup()
    g.set_xl_yl(wl.xl, wl.yl)
    g.set_dt(wl.dt)
    g.init_h(wl.h0.copy())
    g.set_erosional_parameters(wl.kf, wl.kfsed, wl.m, wl.n, wl.kd, wl.kdsed, wl.g1, wl.g2, wl.p)
    g.set_u(wl.u)
    g.set_bc(wl.bc)
    g.set_capture(True)
    g.execute_step()
    dg, do = g.locmin_debug(), O.locmin_debug()
    for k in ("w", "sort_id", "tree"):
        assert np.array_equal(dg[k], do[k]), k
    assert np.array_equal(g.copy_int("rec"), O.copy_int("rec"))
    assert np.array_equal(g.copy_int("stack"), O.copy_int("stack"))
    g.destroy()
