"""The stack from the Euler tour ranked in tiles (k_tour_tiles in
csrc/fsb_routing.cu) on grids that end before, at and after a tile's 64 x 32
nodes, with cyclic sides (neighbours in other tiles), and on surfaces made of
roots only or of many pits (paths that end with the next root of a row).  The
stack and the receivers are bit-exact."""
import numpy as np
import pytest

import oracle as O
from fastscapelib_fortran import workloads as W
from test_advect import make_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(5, 4), (63, 31), (64, 32), (65, 33), (130, 5), (4, 70), (129, 97)])
@pytest.mark.parametrize("bc", [1111, 1010, 101, 1000])
@pytest.mark.parametrize("surface", ["random", "pits", "steps"])
def test_stack(nx, ny, bc, surface):
    wl = W.plain_d8(nx, ny, seed=nx + bc)
    wl.bc = bc
    k = np.arange(wl.nn)
    if surface == "pits":
        wl.h0 = np.where((k % nx % 2 == 0) & (k // nx % 2 == 0), 0.0, 10.0) + wl.h0
    elif surface == "steps":
        wl.h0 = np.floor(wl.h0 * 3)  # many nodes without a lower neighbour
    wl.apply(O)
    g = make_gpu(wl)
    O.fastscape_execute_step()
    g.execute_step()
    assert np.array_equal(g.copy_int("rec"), O.copy_int("rec"))
    assert np.array_equal(g.copy_int("stack"), O.copy_int("stack"))
    g.destroy()
