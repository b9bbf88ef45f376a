"""The heavy-path chain sweeps (csrc/fsb_chains.cu) where a chain changes
worker: strips whose flow paths are one node, just below and at the length that
gets a warp of its own (16), and around its chunks of 32 nodes; and comb-shaped
relief with many short chains on long ones.  One single-flow step per grid from
the oracle's state, with a precipitation that rules out the area's closed form:
routing bit-exact, floats within 1e-12 relative (CUDA's pow and glibc's may
differ in the last ulp; sums and the fill run in the reference's order)."""
import numpy as np
import pytest

import oracle as O
from fastscapelib_fortran import workloads as W

pytestmark = pytest.mark.gpu

LENGTHS = [3, 15, 16, 17, 18, 32, 33, 34, 65, 97, 300]


def _run(wl, bc, n, h0, precip):
    import fastscapelib_fortran as fs
    wl.n, wl.bc, wl.h0 = n, bc, h0
    wl.apply(O)
    O.fastscape_set_precip(precip)
    g = fs.FastScape(0)
    g.set_nx_ny(wl.nx, wl.ny)
    g.setup()
    g.set_xl_yl(wl.xl, wl.yl)
    g.set_dt(wl.dt)
    g.init_h(h0.copy())
    g.set_erosional_parameters(wl.kf, wl.kfsed, wl.m, wl.n, wl.kd, wl.kdsed, wl.g1, wl.g2, wl.p)
    g.set_u(wl.u)
    g.set_precip(precip)
    g.set_bc(bc)
    g.execute_step()
    O.fastscape_execute_step()
    assert np.array_equal(g.copy_int("rec"), O.copy_int("rec"))
    assert np.array_equal(g.copy_int("stack"), O.copy_int("stack"))
    for f in ("drainage_area", "lake_depth", "h", "total_erosion"):
        a, b = np.empty(wl.nn), O.copy_double(f)
        g.copy(f, a)
        assert np.max(np.abs(a - b) / np.maximum(np.abs(b), 1.0)) <= 1e-12, f
    chi, want = np.empty(wl.nn), np.empty(wl.nn)
    g.copy_chi(chi)
    O.fastscape_copy_chi(want)
    assert np.max(np.abs(chi - want) / np.maximum(np.abs(want), 1.0)) <= 1e-12
    assert np.allclose(g.get_fluxes(), O.fastscape_get_fluxes(), rtol=1e-12, atol=0)
    g.destroy()


@pytest.mark.parametrize("length", LENGTHS)
@pytest.mark.parametrize("n", [1.0, 1.5, 1.37])
def test_strip(length, n):
    """One path per column down a strip that drains over its lower edge only."""
    wl = W.plain_d8(3, length, seed=length)
    rng = np.random.default_rng(length)
    h0 = np.repeat(np.arange(length, dtype=np.float64), 3) * 5.0 + rng.random(wl.nn)
    _run(wl, 1000, n, h0, 0.5 + rng.random(wl.nn))


@pytest.mark.parametrize("nx,ny", [(33, 70), (64, 40), (101, 23)])
def test_comb(nx, ny):
    """Side slopes of every length into valleys that run down the grid; some pits."""
    wl = W.plain_d8(nx, ny, seed=nx)
    rng = np.random.default_rng(ny)
    x, y = np.tile(np.arange(nx), ny), np.repeat(np.arange(ny), nx)
    h0 = 2.0 * y + 3.0 * np.abs(x % 16 - 8) + rng.random(wl.nn) * 4.0
    _run(wl, 1010, 1.37, h0, 0.5 + rng.random(wl.nn))
