"""Numbers of planes that the line transforms take: limited by the blocks of a launch, not by the grid's elements.

The sizes are checked before the pointers, so calls with null pointers and no GPU tell one refusal from the other.
"""

import numpy as np
import pytest

import pygrog_b200

INVALID, RANGE = 1, 5


def _shapes(*s):
    a = np.array(s, dtype=np.int64)
    return a, a.ctypes.data


@pytest.mark.parametrize("B,C,grid,status", [
    (328, 16, (640, 640), INVALID),  # 17 GB of grids: the null pointer is what is wrong
    (5000, 16, (320, 320), INVALID),
    (1, 1 << 20, (64, 64), INVALID),
    (64, 32, (96, 192, 192), INVALID),
    (1 << 20, 1 << 12, (64, 64), RANGE),
    (1 << 14, 1 << 14, (64, 640), RANGE),
    (1 << 12, 1 << 12, (64, 960, 960), RANGE),
])
def test_planes_of_the_line_transforms(B, C, grid, status):
    lib = pygrog_b200.load_library()
    n, npt = _shapes(*grid)
    tw = np.full(len(grid), 64, dtype=np.uint64)  # not read: nothing is launched
    st = lib.pgb_line_to_grid(None, None, None, None, None, B, C, len(grid), npt, npt, tw.ctypes.data, None)
    assert st == status, lib.pgb_last_error()
    st = lib.pgb_line_to_image(None, None, None, None, None, B, C, len(grid), npt, npt, tw.ctypes.data, 1.0, None, 0.0, None)
    assert st == status, lib.pgb_last_error()
