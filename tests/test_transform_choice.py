"""Which transforms the 2-D normal operators take, and that both routes agree.

Tolerance: two FP32 transforms of about 2 log2(N) = 16 roundings a value each, eps = 6e-8, sqrt-wise 6 eps, and the
PSF and maps: 1e-6 of the image's norm is twice that.
"""

import math

import pytest
import torch

from pygrog_b200._toep import circulant_length, line_components, line_images
from pygrog_b200.operator import SparseFFT, with_subspace


@pytest.mark.parametrize("N,cuffts_over_lines", [(500, 0.78), (368, 0.78), (361, 0.83), (289, 0.88), (196, 0.89),
                                                 (300, 1.01), (297, 1.06), (319, 1.66), (277, 3.0), (247, 1.41)])
def test_scalar_operator_follows_the_measurements(N, cuffts_over_lines):
    g = (N, N)
    assert (line_images(g, g) < math.inf) == (cuffts_over_lines < 0.97)
    assert line_images(g, (N // 2, N // 2)) == math.inf  # oversampled
    assert line_images((N, 256), (N, 256)) == math.inf  # only one axis is moved
    assert line_images((64, N, N), (64, N, N)) == math.inf  # 3-D: its own lengths


@pytest.mark.parametrize("N,K,lines", [(500, 2, False), (500, 5, False), (361, 3, False), (209, 2, True), (209, 3, False),
                                       (209, 4, True), (209, 5, False), (279, 5, True), (203, 5, True), (182, 5, False),
                                       (182, 3, True), (277, 5, True), (192, 5, True)])
def test_components_follow_the_measurements(N, K, lines):
    assert line_components((N, N), (N, N), K) == lines
    assert line_components((N, N), (N // 2, N // 2), K)


def _reference(psf, smaps, x, n, N):
    """Centred transforms in FP64: psf (N, N) or (N, N, K, K), x (.., n, n) or (K, n, n)."""
    o = (N - n) // 2
    u = torch.zeros(*x.shape[:-2], smaps.shape[0], N, N, dtype=torch.complex128, device=x.device)
    u[..., o:o + n, o:o + n] = x[..., None, :, :].to(torch.complex128) * smaps.to(torch.complex128)
    ax = (-2, -1)
    k = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(u, dim=ax), dim=ax), dim=ax)
    if psf.ndim == 2:
        k = k * psf.double()
    else:
        k = torch.einsum("yxab,bcyx->acyx", psf.to(torch.complex128), k)
    v = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(k, dim=ax), dim=ax), dim=ax)
    return (v[..., o:o + n, o:o + n] * smaps.to(torch.complex128).conj()).sum(-3)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [196, 289])
@pytest.mark.parametrize("C,frames", [(15, 1), (16, 1), (5, 3), (5, 4)])
def test_scalar_operator_on_both_routes(cuda, N, C, frames):
    g = torch.Generator(device=cuda).manual_seed(N + C)
    rnd = lambda *s: torch.randn(s, dtype=torch.complex64, device=cuda, generator=g)  # noqa: E731
    smaps, x = rnd(C, N, N), rnd(frames, N, N)
    op = SparseFFT(grid_shape=(N, N), image_shape=(N, N), indices=torch.randint(0, N * N, (4000,)),
                   weights=torch.rand(4000), smaps=smaps, toeplitz=True, device=cuda)
    y = op.normal(x)
    t = op._toep_op
    assert t._line_images == 15 and circulant_length(N, N) > 1.9 * N and (t._lines is None) == (C > 15)
    ref = _reference(t.psf, smaps, x, N, N)
    assert float((y - ref).norm() / ref.norm()) < 1e-6
    one = op.normal(x[0])  # fewer coil images: the other route where the frames made it
    assert float((one - ref[0]).norm() / ref[0].norm()) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(196, 2), (209, 2), (209, 3)])
def test_components_on_both_routes(cuda, N, K):
    g = torch.Generator(device=cuda).manual_seed(N + K)
    rnd = lambda *s: torch.randn(s, dtype=torch.complex64, device=cuda, generator=g)  # noqa: E731
    T, C = 6, 4
    smaps, x = rnd(C, N, N), rnd(K, N, N)
    base = SparseFFT(grid_shape=(N, N), image_shape=(N, N), indices=torch.randint(0, N * N, (T * 700,)),
                     weights=torch.rand(T * 700), smaps=smaps, toeplitz=True, device=cuda)
    base.natural_shape = (T, 700)
    op = with_subspace(base, rnd(K, T), encoding_axis=-2)
    y = op.normal(x)
    assert (op._toep_op._lines is not None) == line_components((N, N), (N, N), K)
    ref = _reference(op._toep_op.psf, smaps, x, N, N)
    assert float((y - ref).norm() / ref.norm()) < 1e-6
