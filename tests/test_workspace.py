"""fsb_workspace_bytes on the CPU: a strip needs no more device memory than a
square grid of as many nodes (its tiles hold fewer nodes than their area)."""
import ctypes
import math

import pytest

import fastscapelib_fortran as fs


def _bytes(nx, ny):
    lib = fs._lib
    h, b = ctypes.c_void_p(), ctypes.c_size_t()
    assert lib.fsb_create(ctypes.byref(h)) == 0
    assert lib.fsb_set_nx_ny(h, nx, ny) == 0
    assert lib.fsb_workspace_bytes(h, ctypes.byref(b)) == 0
    lib.fsb_destroy(h)
    return b.value / (nx * ny)


@pytest.mark.parametrize("nx,ny", [(3, 100000), (100000, 3), (5, 60000), (8, 100000), (40, 30000)])
def test_strips_need_no_more_than_squares(nx, ny):
    side = int(math.sqrt(nx * ny))
    # the table of basin pairs is a power of two: compare at the same fill
    table = lambda n: 24.0 * 2 ** math.ceil(math.log2(8 * n)) / n  # noqa: E731
    assert _bytes(nx, ny) - table(nx * ny) <= 1.01 * (_bytes(side, side) - table(side * side))
