"""The region sweeps (csrc/fsb_region.cu) on strips: cyclic sides that one tile
spans, whose nodes release each other without the mailbox, and the borders of
the rule that gives strips the larger tiles.  The sweeps' timers count launches,
so that a step that fell back to the queue engine of fsb_flow.cu would show.
Against the oracle as in test_region_sweeps.py.

Both engines do a node's arithmetic in the same order: with g > 0 below the
smallest normal number the step takes one Gauss-Seidel iteration, which is the
g = 0 solve on the queue engine (and no deposition), and must give its bits."""
import numpy as np
import pytest

import oracle as O
from fastscapelib_fortran import workloads as W
from test_region_sweeps import _rel

pytestmark = pytest.mark.gpu


def _gpu(wl, g=0.0):
    import fastscapelib_fortran as fs
    x = fs.FastScape(0)
    x.set_nx_ny(wl.nx, wl.ny)
    x.setup()
    x.set_xl_yl(wl.xl, wl.yl)
    x.set_dt(wl.dt)
    x.init_h(wl.h0.copy())
    x.set_erosional_parameters(wl.kf, wl.kfsed, wl.m, wl.n, wl.kd, wl.kdsed, g, g, wl.p)
    x.set_u(wl.u)
    x.set_bc(wl.bc)
    x.set_profile(True)
    x.execute_step()
    return x


def _field(x, name, nn):
    out = np.empty(nn)
    x.copy(name, out)
    return out


def _tilted(wl):
    j, i = np.divmod(np.arange(wl.nn), wl.nx)
    wl.h0 = wl.h0 + 0.3 * (j if wl.ny > wl.nx else i)  # flow along the strip
    return wl


STRIPS = [(3, 700, 1010), (700, 4, 101), (20, 300, 1000), (300, 31, 1), (32, 300, 1010), (33, 256, 1010), (33, 255, 1111),
          (256, 64, 101), (64, 300, 1111), (65, 300, 1010), (300, 64, 1)]


@pytest.mark.parametrize("nx,ny,bc", STRIPS)
@pytest.mark.parametrize("n", [1.0, 1.5, 1.27])
def test_strips_match_oracle(nx, ny, bc, n):
    wl = _tilted(W.mfd(nx, ny, seed=nx * 1000 + ny, n=n, bc=bc))
    wl.apply(O)
    O.fastscape_execute_step()
    x = _gpu(wl)
    st = x.stage_times()
    assert st["k_area_sweep"][1] == 1 and st["k_spl_sweep"][1] == 1
    assert np.array_equal(x.copy_int("rec"), O.copy_int("rec"))
    for f in ("drainage_area", "h", "total_erosion"):
        assert _rel(_field(x, f, wl.nn), O.copy_double(f)) <= 1e-9, f
    x.destroy()


@pytest.mark.parametrize("nx,ny,bc", [(3, 3, 1010), (33, 64, 1010), (130, 96, 101), (64, 300, 1111), (20, 300, 1000),
                                      (600, 520, 10)])
@pytest.mark.parametrize("n", [1.0, 1.5, 1.27])
def test_engines_give_the_same_bits(nx, ny, bc, n):
    wl = W.mfd(nx, ny, seed=nx + ny, n=n, bc=bc)
    a, b = _gpu(wl), _gpu(wl, g=1.0e-310)
    assert a.stage_times()["k_spl_sweep"][1] == 1 and b.stage_times()["k_spl_sweep"][1] == 0
    for f in ("h", "total_erosion", "erosion_rate"):
        assert np.array_equal(_field(a, f, wl.nn).view(np.int64), _field(b, f, wl.nn).view(np.int64)), f
    a.destroy()
    b.destroy()
