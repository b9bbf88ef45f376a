"""The tridiagonal line solver at the edges of its chunks and warps.

`k_thomas` in csrc/fsb_flow.cu moves the equations of 32 systems through
chunks of 8 in the elimination and of 16 (one right-hand side) or 12 (three)
in the back substitution, different warps working on successive chunks.  The
sizes below put the last equation and the last system on either side of those
edges.  Diffusion alone has one right-hand side, advection alone three.
"""
import numpy as np
import pytest

import oracle as O
from fastscapelib_fortran import workloads as W
from test_advect import field, make_gpu
from test_oracle import velocity_field

pytestmark = pytest.mark.gpu

SIZES = [(4, 5), (8, 9), (7, 34), (9, 35), (16, 17), (17, 33), (25, 31), (41, 66)]


def still(nx, ny, seed):
    wl = W.plain_d8(nx, ny, seed=seed)
    wl.kf = np.zeros(wl.nn)
    wl.u = np.zeros(wl.nn)
    return wl


@pytest.mark.parametrize("nx,ny", SIZES)
def test_three_right_hand_sides(nx, ny):
    wl = still(nx, ny, nx)
    wl.kd = np.zeros(wl.nn)
    vx, vy = velocity_field(nx, ny, 5)
    wl.apply(O)
    O.fastscape_set_v(vx, vy)
    g = make_gpu(wl)
    g.set_v(vx, vy)
    for _ in range(2):
        O.fastscape_execute_step()
        g.execute_step()
    for f in ("h", "basement", "total_erosion"):
        assert np.array_equal(field(g, f), O.copy_double(f)), f
    g.destroy()


@pytest.mark.parametrize("nx,ny", SIZES)
def test_one_right_hand_side(nx, ny):
    wl = still(nx, ny, ny)
    wl.apply(O)
    g = make_gpu(wl)
    O.fastscape_execute_step()
    g.execute_step()
    for f in ("h", "basement", "total_erosion"):
        a, b = field(g, f), O.copy_double(f)
        assert np.max(np.abs(a - b) / np.maximum(np.abs(b), 1.0)) <= 1e-12, f
    g.destroy()
