"""Indices of ``pgb_cell_sum`` outside its operands."""

import numpy as np
import pytest
import torch

import pygrog_b200
from pygrog_b200._fftops import CellLists, FFTStage


def test_a_basis_has_encodings():
    g = np.array([8, 8], dtype=np.int64)
    lib = pygrog_b200.load_library()
    st = lib.pgb_cell_sum(None, None, None, None, None, 8, 0, None, 0, 1, 2, 0, 2, g.ctypes.data, None, 0, None, 0, None,
                          None)
    assert st == 1  # T = 0


@pytest.mark.gpu
def test_encodings_and_samples_out_of_range_add_nothing(cuda):
    """Against the lists of the replicas in range alone: the same sums in the same order."""
    grid, R, T, C, K = (21, 40), 6000, 7, 3, 4
    g = torch.Generator(device=cuda).manual_seed(2)
    cell = torch.randint(0, 840, (R,), device=cuda, generator=g)
    cell[:3000] = 400  # a long list
    t = torch.randint(-2, T + 2, (R,), device=cuda, generator=g)
    w = torch.rand(R, device=cuda, generator=g) + 0.1
    y = torch.randn(1, C, R, dtype=torch.complex64, device=cuda, generator=g)
    phi = torch.randn(K, T, dtype=torch.complex64, device=cuda, generator=g)
    st = FFTStage(grid, grid)
    lists = CellLists(grid, cell.int(), w)
    out = []
    ok = (t >= 0) & (t < T)
    n = R - 100  # fewer samples than listed
    for tt, ww in ((t, w), (t.clamp(0, T - 1), torch.where(ok, w, 0.0))):
        u = torch.empty(1, K, C, *grid, dtype=torch.complex64, device=cuda)
        yy = y[..., :n].contiguous()
        out.append(st.cell_sum(yy, lists, ww[lists.rep].contiguous(), u, 1, C, n, tt[lists.rep].int().contiguous(), phi))
    assert torch.equal(*out)
