"""The C entries that add weighted samples to a grid (``pgb_sparse_scatter``, ``pgb_subspace_scatter``)."""

import pytest
import torch

import pygrog_b200
from pygrog_b200 import _lib


def test_the_entries_are_there_and_check_their_sizes():
    lib = pygrog_b200.load_library()
    assert lib.pgb_sparse_scatter(None, None, None, None, 1, -1, 4, None) == 1
    assert lib.pgb_sparse_scatter(None, None, None, None, 1, 1, 4, None) == 1
    assert lib.pgb_sparse_scatter(None, None, None, None, 1, 0, 4, None) == 0
    assert lib.pgb_subspace_scatter(None, None, None, None, None, None, 1, 1, 33, 2, 1, 4, None) == 1
    assert lib.pgb_subspace_scatter(None, None, None, None, None, None, 1, 1, 2, 0, 1, 4, None) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("BC,R,G", [(1, 1, 7), (3, 4097, 50), (12, 900, 2000)])
def test_scatter_matches_fp64(cuda, BC, R, G):
    """Entries without a cell or a weight add nothing; M terms a cell: M eps of their magnitudes (eps = 6e-8)."""
    g = torch.Generator(device=cuda).manual_seed(R)
    y = torch.randn(BC, R, dtype=torch.complex64, device=cuda, generator=g)
    cell = torch.randint(-2, G + 2, (R,), device=cuda, generator=g)
    w = torch.rand(R, device=cuda, generator=g) * (torch.rand(R, device=cuda, generator=g) > 0.2)
    u0 = torch.randn(BC, G, dtype=torch.complex64, device=cuda, generator=g)
    u, cell32 = u0.clone(), cell.int()
    _lib.call("pgb_sparse_scatter", y.data_ptr(), cell32.data_ptr(), w.data_ptr(), u.data_ptr(), BC, R, G,
              _lib.stream_ptr(cuda))
    ok = (cell >= 0) & (cell < G) & (w != 0)
    t = y[:, ok].to(torch.complex128) * w[ok].double()
    ref = u0.to(torch.complex128).index_add_(1, cell[ok], t)
    size = u0.abs().double().index_add_(1, cell[ok], t.abs())
    most = int(torch.bincount(cell[ok], minlength=1).max()) if bool(ok.any()) else 0
    assert bool(((u - ref).abs() <= (most + 3) * 6e-8 * size).all())


@pytest.mark.gpu
def test_subspace_scatter_matches_fp64(cuda):
    B, C, K, T, R, G = 2, 3, 4, 5, 3000, 60
    g = torch.Generator(device=cuda).manual_seed(1)
    y = torch.randn(B, C, R, dtype=torch.complex64, device=cuda, generator=g)
    phi = torch.randn(K, T, dtype=torch.complex64, device=cuda, generator=g)
    cell = torch.randint(-2, G + 2, (R,), device=cuda, generator=g)
    ti = torch.randint(-1, T + 1, (R,), device=cuda, generator=g)
    w = torch.rand(R, device=cuda, generator=g)
    u = torch.zeros(B, K, C, G, dtype=torch.complex64, device=cuda)
    cell32, ti32 = cell.int(), ti.int()
    _lib.call("pgb_subspace_scatter", y.data_ptr(), cell32.data_ptr(), w.data_ptr(), ti32.data_ptr(), phi.data_ptr(),
              u.data_ptr(), B, C, K, T, R, G, _lib.stream_ptr(cuda))
    ok = (cell >= 0) & (cell < G) & (ti >= 0) & (ti < T)
    t = (y[:, None, :, ok].to(torch.complex128) * (phi[:, ti[ok]].to(torch.complex128) * w[ok].double())[None, :, None])
    ref = torch.zeros(u.shape, dtype=torch.complex128, device=cuda).index_add_(3, cell[ok], t)
    size = torch.zeros(u.shape, dtype=torch.float64, device=cuda).index_add_(3, cell[ok], t.abs())
    most = int(torch.bincount(cell[ok]).max())
    assert bool(((u - ref).abs() <= 2 * (most + 3) * 6e-8 * size).all())  # a complex product doubles a term's error
