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


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [(4, 4, 16), (5, 9, 33), (16, 16, 48), (31, 7, 100)])
@pytest.mark.parametrize("R", [1, 300, 2000])
def test_sparse_and_dense_grids_of_3d(cuda, grid, R):
    """Odd and even numbers of bricks, fewer and more replicas than cells: M terms a cell (a long list among
    them), M eps of their magnitudes, eps = 6e-8."""
    g = torch.Generator(device=cuda).manual_seed(R)
    G, C = int(np.prod(grid)), 5
    cell = torch.randint(0, G, (R,), device=cuda, generator=g)
    cell[:20] = G // 2
    w = torch.rand(R, device=cuda, generator=g) + 0.1
    y = torch.randn(2, C, R, dtype=torch.complex64, device=cuda, generator=g)
    st, lists = FFTStage(grid, grid), CellLists(grid, cell.int(), w)
    u = torch.full((2, C, *grid), float("nan"), dtype=torch.complex64, device=cuda)
    st.cell_sum(y, lists, w[lists.rep].contiguous(), u, 2, C, R)
    terms = y.to(torch.complex128) * w.double()
    ref = torch.zeros(2, C, G, dtype=torch.complex128, device=cuda).index_add_(2, cell, terms)
    size = torch.zeros(2, C, G, dtype=torch.float64, device=cuda).index_add_(2, cell, terms.abs())
    most = int(torch.bincount(cell).max())
    assert bool(((u.reshape(2, C, G) - ref).abs() <= (most + 3) * 6e-8 * size).all())
