"""Alignment of the operator table in the ordered expansion: what its loads need, no more."""

import numpy as np
import pytest
import torch

import pygrog_b200
from pygrog_b200.calib import GrogInterpolator
from pygrog_b200.workloads import radial2d

INVALID, UNSUPPORTED = 1, 4


@pytest.mark.parametrize("C,table,status", [
    (3, 8, UNSUPPORTED), (3, 4, INVALID), (6, 16, UNSUPPORTED), (6, 8, INVALID), (8, 32, UNSUPPORTED), (8, 16, INVALID),
])
def test_alignment_by_coils(C, table, status):
    """Checked before the sizes: nothing is launched (3000 cells a sample are refused)."""
    lib = pygrog_b200.load_library()
    assert lib.pgb_grog_expand_sorted(8, 1, None, 0, 3000, 8, 8, table, 1, C, 1, 8, None) == status, lib.pgb_last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("C", [6, 8])
def test_tables_that_are_views(cuda, C):
    rng = np.random.default_rng(C)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    g = GrogInterpolator(shape=(48, 48), coords=radial2d(30, 300, 24.0), oversamp=1.0, kernel_width=3,
                         kernel_shape="square", device=cuda)
    g.calc_interp_table(cplx(C, 12, 12), lamda=0.1, precision=1)
    x = torch.from_numpy(cplx(C, 30, 300)).to(cuda)
    g.gridder_mode = "ordered"
    want = g.interpolate(x), g.grid(x)
    t = torch.empty(g._table_d.numel() + 2, dtype=torch.complex64, device=cuda)[2:].view(g._table_d.shape)
    t.copy_(g._table_d)
    assert t.data_ptr() % 32 == 16
    g._table_d, g._interp_kernel, g._brick_plans = t, t, None
    assert torch.equal(g.interpolate(x), want[0]) and torch.equal(g.grid(x), want[1])
