"""The index sort of the basin-graph edges as the GPU runs it (k_nr_levels and
k_nr_block in csrc/fsb_locmin.cu): segments that one block finishes, alone
(fewer than 8192 edges) and after grid-wide levels (more), with few and with
very many equal weights, whose order the reference's quicksort fixes.  The
permutation, the spanning tree and the corrected receivers are bit-exact."""
import numpy as np
import pytest

import oracle as O
from fastscapelib_fortran import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [5, 9, 24, 60, 140, 170, 260])
@pytest.mark.parametrize("levels", [0, 400, 40])  # distinct heights (0: all of them)
def test_sort_permutation(side, levels):
    import fastscapelib_fortran as fs
    wl = W.plain_d8(side, side + 3, seed=side)
    if levels:
        wl.h0 = np.floor(wl.h0 * levels) / levels
    wl.apply(O)
    O.fastscape_execute_step()
    g = fs.FastScape(0)
    g.set_nx_ny(wl.nx, wl.ny)
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
    for k in ("nconn", "tree_size"):
        assert dg[k] == do[k], k
    for k in ("w", "sort_id", "tree", "ob1", "ob2"):
        assert np.array_equal(dg[k], do[k]), k
    assert np.array_equal(g.copy_int("rec"), O.copy_int("rec"))
    g.destroy()


@pytest.mark.parametrize("side", [200, 560, 900])  # edges: below and above one block's partition
@pytest.mark.parametrize("levels", [0, 40])
def test_sort_permutation_of_block_partitions(side, levels):
    test_sort_permutation(side, levels)
