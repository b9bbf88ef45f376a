"""The index sort's block kernel on the CPU, with weights that hold NaN.

`k_nr_block` in csrc/fsb_locmin.cu (partitions by a block and by a warp, the
queues between them, the placement of the last few elements) is compiled for
the host with g++.  A thread of the block is a coroutine that runs up to the
next barrier, ballot or shuffle of its group, so one CPU thread runs the
kernel as it stands.  The chunk sizes are replaced by small ones: listings end,
are reloaded and cross inside a few hundred elements.

What it must give is the sequential sort (`nr_sort_local`: the reference's
quicksort, LocalMinima.f90:947-1046, its insertion held inside a segment), ties,
infinities and NaN included: the Hoare scans stop where a weight is not below
(above) the pivot, so a NaN stops both, and a NaN pivot stops them everywhere.
Without NaN that is the oracle's permutation.  The grid-wide levels are checked
on the same arrays through the driver of test_nr_level_emulation.py.
"""
import ctypes
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from test_nr_level_emulation import SRC, _between, _function, emulate  # noqa: F401

SHIM = r"""
#include <climits>
#include <cstdint>
#include <cstring>
#include <ucontext.h>
#include <vector>
static int min(int a, int b) { return a < b ? a : b; }
static int max(int a, int b) { return a < b ? b : a; }
#define __device__
#define __global__
#define __forceinline__ inline
#define __align__(x) alignas(x)
#define __launch_bounds__(...)
#define __shared__
struct Fiber { ucontext_t ctx; bool done; };
static ucontext_t g_main;
static std::vector<Fiber> g_fibers;
static int g_me;
struct Dim { int x; };
#define threadIdx (Dim{g_me})
static void yield() { const int me = g_me; swapcontext(&g_fibers[me].ctx, &g_main); }
struct Group {
  int n = 0, arrived = 0;
  unsigned gen = 0;
  std::vector<long long> in, out;
  void init(int size) { n = size; arrived = 0; gen = 0; in.assign(size, 0); out.assign(size, 0); }
  const std::vector<long long>& meet(int at, long long v) {
    in[at] = v;
    if (++arrived == n) { out = in; arrived = 0; ++gen; }
    else for (const unsigned g = gen; g == gen;) yield();
    return out;
  }
};
static Group g_block, g_warp[64];
static const std::vector<long long>& warp_meet(long long v) { return g_warp[g_me / 32].meet(g_me % 32, v); }
static void __syncthreads() { g_block.meet(g_me, 0); }
static void __syncwarp() { warp_meet(0); }
static int __syncthreads_count(bool p) {
  int n = 0;
  for (long long v : g_block.meet(g_me, p)) n += (int)v;
  return n;
}
static unsigned __ballot_sync(unsigned, bool p) {
  const std::vector<long long>& v = warp_meet(p);
  unsigned m = 0;
  for (int l = 0; l < 32; ++l) m |= (unsigned)v[l] << l;
  return m;
}
template <class T>
static T lane_value(long long b) { T v; std::memcpy(&v, &b, sizeof v); return v; }
template <class T>
static T __shfl_sync(unsigned, T v, int src, int width = 32) {
  long long b = 0;
  std::memcpy(&b, &v, sizeof v);
  const int lane = g_me % 32;
  return lane_value<T>(warp_meet(b)[lane / width * width + src % width]);
}
template <class T>
static T __shfl_up_sync(unsigned, T v, int d) {
  long long b = 0;
  std::memcpy(&b, &v, sizeof v);
  const int lane = g_me % 32;
  return lane_value<T>(warp_meet(b)[lane >= d ? lane - d : lane]);
}
static int __popc(unsigned v) { return __builtin_popcount(v); }
template <class T> static T __ldcg(const T* p) { return *p; }
static void __threadfence() {}
static void __threadfence_block() {}
static void __nanosleep(int) { yield(); }
static int atomicAdd(int* p, int v) { const int o = *p; *p += v; return o; }
static int atomicSub(int* p, int v) { const int o = *p; *p -= v; return o; }
static int atomicExch(int* p, int v) { const int o = *p; *p = v; return o; }
static int atomicCAS(int* p, int c, int v) { const int o = *p; if (o == c) *p = v; return o; }
constexpr int kSpinLimit = 1 << 21;
// far larger than the kernel's part, so that a stray index fails the comparison
alignas(16) static unsigned char nr_smem[1 << 20];
@enum@
@code@
namespace sequential {
constexpr int kNrMedium = 1 << 24;
@sort_local@
}
extern "C" int sort_sequential(double* key, int* id, int n) { return sequential::nr_sort_local(key, id, n) ? 0 : 1; }

struct Call { unsigned long long* med; int cap; double* key; int* idx; int* cnt; };
static Call g_call;
static void fiber_main() {
  k_nr_block(g_call.med, g_call.cap, g_call.key, g_call.idx, g_call.cnt);
  const int me = g_me;
  g_fibers[me].done = true;
  swapcontext(&g_fibers[me].ctx, &g_main);
}
// sorts w[0..n-1] as nr_indexx does for n in one block's range; 0 or what went wrong
extern "C" int block_sort(int n, const double* w, int* perm) {
  std::vector<int> idx(n + 2), cnt(32, 0);
  std::vector<double> key(n + 2);
  const int cap = n / 8 + 8;
  std::vector<unsigned long long> med(cap, 0ull);
  for (int q = 1; q <= n; ++q) { idx[q] = q; key[q] = w[q - 1]; }
  med[0] = (unsigned long long)n << 32 | 1u;
  cnt[C_NMED] = 1;
  cnt[C_NROPEN] = 1;
  g_call = Call{med.data(), cap, key.data(), idx.data(), cnt.data()};
  std::vector<std::vector<char>> stacks(kNrThreads, std::vector<char>(64 * 1024));
  g_fibers.assign(kNrThreads, Fiber{});
  g_block.init(kNrThreads);
  for (int v = 0; v < kNrWarps; ++v) g_warp[v].init(32);
  for (int t = 0; t < kNrThreads; ++t) {
    getcontext(&g_fibers[t].ctx);
    g_fibers[t].ctx.uc_stack.ss_sp = stacks[t].data();
    g_fibers[t].ctx.uc_stack.ss_size = stacks[t].size();
    g_fibers[t].ctx.uc_link = nullptr;
    makecontext(&g_fibers[t].ctx, fiber_main, 0);
  }
  for (long long turn = 0, live = kNrThreads; live > 0; ++turn) {
    if (turn > 20000000) return -1;
    live = 0;
    for (int t = 0; t < kNrThreads; ++t)
      if (!g_fibers[t].done) { ++live; g_me = t; swapcontext(&g_main, &g_fibers[t].ctx); }
  }
  for (int q = 1; q <= n; ++q) perm[q - 1] = idx[q] - 1;
  return cnt[C_OVERFLOW];
}
"""

SIZES = {"kNrBlock": 128, "kNrThreads": 64, "kNrRuns": 1, "kNrEach": 2}


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    text = open(SRC).read()
    enum = _between(text, "enum {\n  C_NBASINS", "};")
    sort_local = _function(text, "__device__ bool nr_sort_local(").replace("__device__ ", "")
    code = "\n".join(l for l in text.splitlines() if re.match(r"constexpr int kNr(Medium|Block|Split) = ", l))
    code += "\n" + sort_local
    code += _between(text, "constexpr int kNrThreads", "static_assert(sizeof(NrBlockShared)", False)
    code += _between(text, "// Partitions positions l..ir", "__global__ void k_rank_from_perm", False)
    code = code.replace("extern __shared__ __align__(16) unsigned char nr_smem[];", "")
    for name, value in SIZES.items():
        code, hits = re.subn(r"\b%s = \d+" % name, "%s = %d" % (name, value), code)
        assert hits == 1, name
    d = tmp_path_factory.mktemp("nrblock")
    cpp, so = d / "nrblock.cpp", d / "nrblock.so"
    cpp.write_text(SHIM.replace("@enum@", enum).replace("@code@", code)
                   .replace("@sort_local@", sort_local.replace("stk[32]", "stk[64]").replace("2 > 32", "2 > 64")))
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-w", "-o", str(so), str(cpp)],
                   check=True)
    lib = ctypes.CDLL(str(so))
    pd, pi = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
    lib.block_sort.argtypes = [ctypes.c_int, pd, pi]
    lib.sort_sequential.argtypes = [pd, pi, ctypes.c_int]
    return lib


def _array(n, kind):
    rng = np.random.default_rng(n + len(kind))
    if kind == "ties":
        return rng.integers(0, 5, n).astype(np.float64)
    a = rng.random(n)
    if kind == "ordered":
        return np.sort(a) + rng.random(n) * 0.01
    if kind == "nan":  # all of them
        a[:] = np.nan
    elif kind in ("some nan", "many nan"):
        a[rng.random(n) < (0.05 if kind == "some nan" else 0.8)] = np.nan
        a[rng.random(n) < 0.1] = np.inf
        a[rng.random(n) < 0.1] = -np.inf
    elif kind == "nan pivot":  # the first median of three
        a[[0, 1, n - 1, (n - 1) // 2]] = np.nan
    return a


def _ptr(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double if a.dtype == np.float64 else ctypes.c_int))


def sequential(lib, w):
    key, ids = w.copy(), np.arange(w.size, dtype=np.int32)
    assert lib.sort_sequential(_ptr(key), _ptr(ids), w.size) == 0
    return ids


KINDS = ["random", "ties", "ordered", "nan", "some nan", "many nan", "nan pivot"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [8, 9, 40, 127, 128, 129, 130, 257, 700, 1500])
def test_block_sort(host, n, kind):
    w = _array(n, kind)
    perm = np.full(n, -1, dtype=np.int32)
    assert host.block_sort(n, _ptr(w), _ptr(perm)) == 0
    expected = sequential(host, w)
    np.testing.assert_array_equal(perm, expected)
    if not np.isnan(w).any():
        np.testing.assert_array_equal(perm, O.indexx(w))


@pytest.mark.parametrize("kind", [k for k in KINDS if "nan" in k])
@pytest.mark.parametrize("n", [600, 3000])
def test_levels(host, emulate, n, kind):  # noqa: F811
    w = _array(n, kind)
    perm, levels = np.full(n, -1, dtype=np.int32), ctypes.c_int()
    assert emulate.nr_emulate(n, _ptr(w), _ptr(perm), ctypes.byref(levels)) == 0
    np.testing.assert_array_equal(perm, sequential(host, w))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,px,py", [(60, 40, 12, 10), (90, 80, 60, 50), (330, 320, 300, 300)])
def test_surface_with_a_nan_patch(host, nx, ny, px, py):
    """Every node of the patch is a pit whose passes weigh NaN: parts of one
    block's shared memory, of its partitions, and grid-wide levels."""
    import fastscapelib_fortran as fs
    from fastscapelib_fortran import workloads as W
    wl = W.plain_d8(nx, ny, seed=nx)
    h = wl.h0.reshape(ny, nx).copy()
    h[10:10 + py, 8:8 + px] = np.nan
    g = fs.FastScape(0)
    g.set_nx_ny(nx, ny)
    g.setup()
    g.set_xl_yl(wl.xl, wl.yl)
    g.set_dt(wl.dt)
    g.init_h(h.ravel())
    g.set_erosional_parameters(wl.kf, wl.kfsed, wl.m, wl.n, np.zeros(wl.nn), -1.0, wl.g1, wl.g2, wl.p)
    g.set_bc(wl.bc)
    g.set_capture(True)
    g.execute_step()
    d = g.locmin_debug()
    w = np.ascontiguousarray(d["w"])
    assert np.isnan(w).sum() > 3 * px * py
    np.testing.assert_array_equal(d["sort_id"], sequential(host, w))
    assert d["tree_size"] == d["nbasins"] - 1
    g.destroy()
