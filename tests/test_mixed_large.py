"""The mixed form's sweeps run in FP32 up to 296 blocks of 256 x 128 nodes and in
FP64 beyond (fp32_sweeps in csrc/fsb_region.cu): every area of an FP32 sweep is a
float, those of an FP64 sweep are not.  And one step of a large grid stays within
1e-6 of the FP64 form's elevations, the bound of test_mixed.py."""
import numpy as np
import pytest

from fastscapelib_fortran import workloads as W
from test_region_engine import _field

pytestmark = pytest.mark.gpu


def _step(wl, precision):
    import fastscapelib_fortran as fs
    g = fs.FastScape(0)
    g.set_nx_ny(wl.nx, wl.ny)
    g.setup()
    g.set_xl_yl(wl.xl, wl.yl)
    g.set_dt(wl.dt)
    g.init_h(wl.h0.copy())
    g.set_erosional_parameters(wl.kf, wl.kfsed, wl.m, wl.n, wl.kd, wl.kdsed, wl.g1, wl.g2, wl.p)
    g.set_u(wl.u)
    g.set_bc(wl.bc)
    g.set_precision(precision)
    g.execute_step()
    a, h = _field(g, "drainage_area", wl.nn), _field(g, "h", wl.nn)
    g.destroy()
    return a, h


@pytest.mark.parametrize("nx,ny,fp32", [(4, 37888, True), (4, 37889, False), (70000, 5, True), (75777, 5, False)])
def test_width_of_the_sweeps(nx, ny, fp32):
    a, _ = _step(W.mfd(nx, ny, seed=nx), "mixed")
    assert np.array_equal(a, a.astype(np.float32).astype(np.float64)) == fp32


def test_large_grid_stays_close():
    wl = W.mfd(4097, seed=3)
    (a, h), (am, hm) = _step(wl, "fp64"), _step(wl, "mixed")
    assert np.max(np.abs(hm - h) / np.maximum(np.abs(h), 1.0)) <= 1e-6
    assert np.max(np.abs(am - a) / a) <= 2e-5  # the FP32 weights alone: 9e-6
