"""The region-owned multiple-flow sweeps (csrc/fsb_region.cu) where their tiles
begin and end: one step of grids around the tile sides of 32 and 64 nodes, of
partial and single tiles, wrapped in x, in y or not at all, with each form of
the stream-power solve, against the oracle.  Routing is bit-exact; the floats
agree to 1e-9 relative (the area sums its donors in another valid order; see
test_gpu_parity.py)."""
import numpy as np
import pytest

import oracle as O
from fastscapelib_fortran import workloads as W

pytestmark = pytest.mark.gpu

GRIDS = [(3, 3), (5, 33), (31, 32), (32, 32), (33, 64), (64, 31), (65, 65), (63, 129), (97, 34), (130, 96),
         (600, 520)]  # the last: more than 2^18 nodes, the area's larger tiles
FORMS = [(1010, 1.5), (101, 1.0), (1111, 1.27), (1000, 1.5), (10, 1.0)]


def _step(wl, precision="fp64"):
    import fastscapelib_fortran as fs
    g = fs.FastScape(0)
    wl.apply(O)
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
    O.fastscape_execute_step()
    return g


def _rel(a, b):
    return np.max(np.abs(a - b) / np.maximum(np.abs(b), 1.0))


@pytest.mark.parametrize("nx,ny", GRIDS)
@pytest.mark.parametrize("bc,n", FORMS)
def test_step_matches_oracle(nx, ny, bc, n):
    wl = W.mfd(nx, ny, seed=nx * 1000 + ny, n=n, bc=bc)
    g = _step(wl)
    assert np.array_equal(g.copy_int("rec"), O.copy_int("rec"))
    for f in ("drainage_area", "h", "total_erosion"):
        out = np.empty(wl.nn)
        g.copy(f, out)
        assert _rel(out, O.copy_double(f)) <= 1e-9, f
    g.destroy()


@pytest.mark.parametrize("nx,ny,n", [(33, 64, 1.5), (97, 34, 1.0), (65, 65, 1.27), (600, 520, 1.5)])
def test_mixed_step_matches_oracle(nx, ny, n):
    wl = W.mfd(nx, ny, seed=nx + ny, n=n)
    g = _step(wl, "mixed")
    out = np.empty(wl.nn)
    g.copy("h", out)
    assert np.array_equal(g.copy_int("rec"), O.copy_int("rec"))
    assert _rel(out, O.copy_double("h")) <= 1e-6  # FP32 increments, as test_mixed.py
    g.destroy()
