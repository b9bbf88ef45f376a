"""The Euler tour's tiles on narrow grids (TourTiles in csrc/fsb_kernels.cuh), whose
sides follow the grid's shorter one.  On the CPU: no tile has more ways out than
list elements, and strips list fewer elements than the tour's 2 nn entries.  On
the GPU: the stack of strips around the tiles' sides, bit for bit."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from fastscapelib_fortran import workloads as W
from test_advect import make_gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "fastscapelib-fortran_b200", "csrc", "fsb_kernels.cuh")


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    text = open(SRC).read()
    i = text.index("constexpr int kTourNodes")
    code = text[i:text.index("\n};\n", i) + 4]
    d = tmp_path_factory.mktemp("tour")
    cpp, so = d / "t.cpp", d / "t.so"
    cpp.write_text("#include <cstddef>\n" + code + 'extern "C" void tiles(int nx, int ny, int* o) { TourTiles t(nx, ny); '
                   "o[0] = t.lx; o[1] = t.ly; o[2] = t.tiles_x; o[3] = t.tiles_y; o[4] = t.slots; }\n")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(cpp)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.tiles.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]

    def get(nx, ny):
        o = (ctypes.c_int * 5)()
        lib.tiles(nx, ny, o)
        return tuple(o)
    return get


def _ring(n, lt, count):
    """Per tile along a side: nodes, and those within two of a neighbouring tile (cyclic sides included)."""
    for t in range(count):
        size = min(1 << lt, n - (t << lt))
        yield size, min(size, 4) if count > 1 else 0


def test_every_way_out_has_an_element(tiles):
    sides = list(range(3, 70)) + [96, 127, 128, 129, 255, 256, 257, 511, 512, 513, 700, 2049]
    for nx in sides:
        for ny in sides:
            lx, ly, cx, cy, slots = tiles(nx, ny)
            assert lx + ly == 11 and cx << lx >= nx and cy << ly >= ny
            assert (cx - 1) << lx < nx and (cy - 1) << ly < ny
            for w, ex in set(_ring(nx, lx, cx)):
                for h, ey in set(_ring(ny, ly, cy)):
                    out = w * h - (w - ex) * (h - ey)  # nodes near a side that the grid continues beyond
                    assert 2 * out + h <= slots, (nx, ny)


@pytest.mark.parametrize("nx,ny", [(3, 60000), (60000, 3), (5, 60000), (8, 40000), (11, 30000), (24, 15000), (15000, 17)])
def test_strips_list_less_than_the_tour(tiles, nx, ny):
    _, _, cx, cy, slots = tiles(nx, ny)
    assert cx * cy * slots < 2 * nx * ny


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(3, 1030), (4, 512), (5, 600), (8, 257), (9, 700), (16, 130), (17, 129), (32, 65), (33, 70),
                                   (1030, 3), (513, 4), (600, 5), (257, 8), (700, 9), (129, 16), (130, 17)])
@pytest.mark.parametrize("bc", [1111, 1010, 101])
@pytest.mark.parametrize("surface", ["random", "pits", "ramp"])
def test_stack_of_strips(nx, ny, bc, surface):
    wl = W.plain_d8(nx, ny, seed=nx + bc)
    wl.bc = bc
    j, i = np.divmod(np.arange(wl.nn), nx)
    if surface == "pits":
        wl.h0 = np.where((i % 2 == 0) & (j % 2 == 0), 0.0, 10.0) + wl.h0
    elif surface == "ramp":
        wl.h0 = wl.h0 + 0.7 * (i if nx > ny else j)
    wl.apply(O)
    g = make_gpu(wl)
    O.fastscape_execute_step()
    g.execute_step()
    assert np.array_equal(g.copy_int("rec"), O.copy_int("rec"))
    assert np.array_equal(g.copy_int("stack"), O.copy_int("stack"))
    g.destroy()
