"""List ranking through several levels of splitters.

`rank_list` in csrc/fsb_routing.cu keeps a few slots per level for list heads.
The basin tree's tour begins at an arbitrary entry (its arcs are stored in the
order of atomics), so whether its head is itself a splitter differs from run
to run; the slots no head takes must stay out of the next level's heads.  A
closed basin of this size has a tour of half a million arcs, two levels of
splitters above the block that ends the recursion.
"""
import numpy as np
import pytest

from fastscapelib_fortran import workloads as W
from test_advect import make_gpu

pytestmark = pytest.mark.gpu


def test_tour_heads_anywhere():
    wl = W.closed_basin(1501, nsteps=1)
    stacks = []
    for _ in range(6):
        g = make_gpu(wl)
        g.execute_step()
        stacks.append(g.copy_int("stack"))
        g.destroy()
    for s in stacks:
        assert np.array_equal(np.sort(s), np.arange(wl.nn) + s.min())
        assert np.array_equal(s, stacks[0])
