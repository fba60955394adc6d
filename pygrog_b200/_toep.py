"""GROG Toeplitz normal operator on the GPU.

Mirrors ``_toep/_grog_toep.py`` (``GrogToeplitzOp``, 30-209) of
FiRMLAB-Pisa/pygrog: the PSF is the per-cell sum of squared sqrt-weights,
``PSF[j] = sum_i w_i delta(j == idx_i)`` built once with
``psf_scatter_scalar`` (or the ``density`` grid of a MaskedFFT), and
``A^H A x = sum_c conj(S_c) crop(IFFT(PSF * FFT(pad(S_c x))))``.

Here, 2-D: three kernels with the library's own line FFTs (``csrc/toep_fft.cu``),
on a circulant length of their choice (:func:`circulant_length`); 3-D: five on
the grid's own lengths (``csrc/line_fft.cu``).  Lengths that are not built: one
coil-expansion kernel, one batched cuFFT, one PSF multiply (PSF stored in FFT
order with the two ortho scales folded in), one batched inverse cuFFT and one
crop + coil-sum kernel per call.  All coils at once in both.
"""

from __future__ import annotations

__all__ = ["GrogToeplitzOp"]

import math

import numpy as np
import torch

from . import _ext, _lib
from ._fftops import FFTStage, as_c64, compute_device, line_lengths, made_now


def circulant_length(N: int, n: int) -> int | None:
    """Line FFT length for the convolution of ``n`` image points behind a PSF on ``N`` grid points.

    The cropped convolution needs the kernel lags ``|l| < n`` only, so any
    length ``L >= 2 n - 1`` gives it; ``N`` itself always does.  The shortest
    of those that is built (``None``: there is none): a grid that is not
    oversampled keeps its own length where that is smooth, and moves to about
    twice its width where it is not (cuFFT's Bluestein transform pads as far).
    Measured, application on cuFFT / on lines, us: 16 coils, 640 (image 320)
    147 / 57; 14 coils, 277 105 / 37; 8 coils, 300 34 / 32, 64 16 / 9, 900
    151 / 119; a full image of 1024 loses (183 / 188) and keeps cuFFT.  Grids whose
    own length cuFFT transforms well are exceptions: below.
    """
    fit = [L for L in line_lengths() if L >= 2 * n or (L == N and L < 1024)]
    return min(fit) if fit else None


# Where an image is as wide as its grid, the circulant length is about twice the grid's and the planes of the lines
# have four times its cells.  That still beats cuFFT on lengths with a prime factor above 31, but not on every
# other one: which, depends on the kernels that cuFFT has for the length.  Measured on square grids of every length
# from 150 to 512 without line FFTs and with factors up to 31 (time on cuFFT / on lines):
#  - the scalar operator from 16 coil images on (20 to 32 coils): below 0.97 (500: 0.78, 361: 0.87, 196: 0.90); below
#    16 coils 0.9 to 1.7, on the others 0.97 to 2.7;
#  - with 2 to 5 components (6 and 16 coils), the matrix of every frequency on top: below 0.9 on average over the
#    components (500: 0.61, 361: 0.67), 0.9 to 1.1, 1.1 to 1.2.  3 and 5 components, whose packed matrix is not
#    whole float4s, are at 0.93 and 0.88 of that average, 2 and 4 at 1.06 and 1.15.
_GRID_LENGTHS = frozenset((
    196, 289, 324, 325, 343, 352, 361, 364, 368, 390, 392, 399, 414, 416, 425, 455, 462, 464, 484, 490, 495,
    496, 500, 504, 510,
))
_GRID_LENGTHS_SUB = frozenset((
    196, 200, 243, 248, 250, 252, 255, 260, 264, 270, 272, 273, 285, 289, 297, 300, 304, 306, 308, 315, 323,
    324, 325, 330, 336, 338, 340, 342, 343, 345, 350, 351, 352, 357, 361, 363, 364, 368, 375, 378, 385, 390,
    391, 392, 396, 399, 405, 408, 414, 416, 420, 425, 429, 437, 440, 441, 448, 450, 455, 459, 462, 464, 468,
    483, 484, 486, 490, 495, 496, 500, 504, 507, 510,
))
_GRID_LENGTHS_SUB35 = frozenset((
    150, 152, 156, 162, 165, 168, 169, 175, 176, 184, 190, 195, 198, 204, 208, 209, 210, 220, 221, 224, 225,
    230, 231, 232, 234, 242, 245, 247, 253, 275, 276, 280, 299, 322, 341, 348, 372, 380, 435, 460, 475, 476, 494,
))
_GRID_LENGTHS_SUB5 = frozenset((
    132, 136, 153, 170, 182, 189, 228, 261, 294, 312, 319, 403, 406, 456, 493,
))


def _twice(grid, image, lengths) -> bool:
    """Both axes of a 2-D grid are among ``lengths`` and their circulant lengths about twice that."""
    return len(grid) == 2 and all(
        N in lengths and (circulant_length(N, n) or 0) >= 1.9 * N for N, n in zip(grid, image))


def line_images(grid, image) -> float:
    """Coil images up to which the scalar operator is faster on lines than on cuFFT transforms of the grid."""
    return 15 if _twice(grid, image, _GRID_LENGTHS) else math.inf


def line_components(grid, image, K: int) -> bool:
    """Whether the operator of ``K`` components is faster on lines than on cuFFT transforms of the grid."""
    lengths = _GRID_LENGTHS_SUB
    if K in (3, 5):
        lengths = lengths | _GRID_LENGTHS_SUB35
    if K == 5:
        lengths = lengths | _GRID_LENGTHS_SUB5
    return not _twice(grid, image, lengths)


def line_plan(psf: torch.Tensor, grid, image):
    """``(L0, L1, psf in slot order, twiddles of L0, of L1)`` of the line-FFT normal operator for a centred
    float32 PSF ``(S, *grid)`` or ``(S, *grid, M)``; ``None`` if its lengths are not built."""
    if len(grid) != 2 or max(grid) >= 2**20:
        return None
    L0, L1 = (circulant_length(N, n) for N, n in zip(grid, image))
    if L0 is None or L1 is None:
        return None
    S, M = int(psf.shape[0]), int(psf.shape[3]) if psf.ndim == 4 else 1
    (N0, N1), dev = grid, psf.device
    lib = _lib.lib()
    tw = [torch.empty(lib.pgb_fft_twiddles(L), dtype=torch.complex64, device=dev) for L in (L0, L1)]
    work = torch.empty(N0 * L0 + N1 * L1 + N0 * L1 * M, dtype=torch.float64, device=dev)
    out = torch.empty(S, L0, L1, M, dtype=torch.float32, device=dev)
    _lib.call("pgb_toep2d_plan", psf.contiguous().data_ptr(), S, M, N0, N1, *image, L0, L1, work.data_ptr(),
              out.data_ptr(), tw[0].data_ptr(), tw[1].data_ptr(), _lib.stream_ptr(dev))
    return L0, L1, out, tw[0], tw[1]


def line_normal(plan, s: int, x, smaps, out, B: int, C: int, K: int, image, damp: float) -> None:
    """``out = A^H A x + damp x`` for ``B`` frames of ``C`` coils (of ``K`` components, ``K > 0``) with stack
    element ``s`` of a :func:`line_plan`."""
    L0, L1, psf, tw0, tw1 = plan
    work = torch.empty(B * max(K, 1) * C * image[0] * L1, dtype=torch.complex64, device=x.device)
    _lib.call("pgb_toep2d", x.data_ptr(), smaps.data_ptr() if smaps is not None else None, psf[s].data_ptr(),
              work.data_ptr(), out.data_ptr(), B, C, K, *image, L0, L1, tw0.data_ptr(), tw1.data_ptr(),
              x.data_ptr() if damp else None, float(damp), _lib.stream_ptr(x.device))


class GrogToeplitzOp:
    """Self-adjoint ``A^H A`` of a :class:`SparseFFT` or :class:`MaskedFFT`."""

    def __init__(self, sparse_fft, device=None):
        self.sparse_fft = sparse_fft
        self.device = compute_device(device if device is not None else getattr(sparse_fft, "device", None))
        self.grid_shape = tuple(sparse_fft.grid_shape)
        self.image_shape = tuple(sparse_fft.image_shape)
        self.fft_axes = sparse_fft.fft_axes
        self._pad_slices = sparse_fft._pad_slices
        self.stack_shape = tuple(getattr(sparse_fft, "stack_shape", ()) or ())
        self._stage = FFTStage(self.grid_shape, self.image_shape)
        S = int(np.prod(self.stack_shape)) if self.stack_shape else 1
        G = self._stage.G
        dens = getattr(sparse_fft, "density", None)
        if dens is not None:
            psf = torch.as_tensor(dens).to(self.device, torch.float32).reshape(S, *self.grid_shape).clone()
        else:
            idx = sparse_fft.indices.reshape(S, -1).to(self.device)
            sw = sparse_fft.sqrt_weights.reshape(S, -1).to(self.device, torch.float32)
            psf = torch.zeros(S, G, dtype=torch.float32, device=self.device)
            for s in range(S):
                _ext.psf_scatter_scalar(psf[s], idx[s].contiguous(), (sw[s] * sw[s]).contiguous())
            psf = psf.reshape(S, *self.grid_shape)
        # reference attribute: PSF on the centred grid
        self.psf = psf.reshape(*self.stack_shape, *self.grid_shape) if self.stack_shape else psf[0]
        self._line_images = line_images(self.grid_shape, self.image_shape)
        smaps = sparse_fft.smaps
        self._lines = None
        if smaps is None or int(smaps.shape[0]) <= self._line_images:
            self._lines = line_plan(psf, self.grid_shape, self.image_shape)
        self._psf3 = None  # 3-D: PSF (S, G) of pgb_toep3d
        if len(self.grid_shape) == 3 and self._stage._lines(self.device) is not None:
            self._psf3 = torch.empty(S, G, dtype=torch.float32, device=self.device)
            for s in range(S):
                p = self._stage.to_fft_order(psf[s]).to(torch.float64).contiguous()
                _lib.call("pgb_toep_slots", p.data_ptr(), self.grid_shape[0], G // self.grid_shape[0], 1.0 / G,
                          self._psf3[s].data_ptr(), _lib.stream_ptr(p.device))
        self._psf_fft = None  # PSF (S, G) of the cuFFT transforms
        if self._psf3 is None and self._lines is None:
            self._psf_fft = self._grid_psf()

    def _grid_psf(self) -> torch.Tensor:
        psf = self.psf.reshape(-1, *self.grid_shape)
        return (self._stage.to_fft_order(psf) * (1.0 / self._stage.G)).reshape(-1, self._stage.G).contiguous()

    def __setstate__(self, state):
        # saved before: cuFFT alone, or lines wherever they were made
        self.__dict__.update({"_line_images": math.inf, "_lines": None, "_psf3": None, "_psf_fft": None, **state})

    def _n_coils(self, x):
        sm = self.sparse_fft.smaps
        return int(sm.shape[0]) if sm is not None else int(x.shape[1])

    def _apply_frames(self, x: torch.Tensor, s: int, out: torch.Tensor, damp: float = 0.0) -> torch.Tensor:
        """x (B, *img) [smaps] or (B, C, *img) on device -> out (same shape)."""
        st = self._stage
        smaps = getattr(self.sparse_fft, "_smaps_d", None)
        B = int(x.shape[0])
        C = self._n_coils(x)
        if self._psf3 is not None:
            g, n = st.grid_shape, st.image_shape
            v = torch.empty(B * C * n[0] * g[1] * g[2], dtype=torch.complex64, device=x.device)
            u = v if n[1] == g[1] else torch.empty(B * C * n[0] * n[1] * g[2], dtype=torch.complex64, device=x.device)
            b, c = (B, C) if smaps is not None else (B * C, 1)
            tw = st._lines(x.device)
            _lib.call("pgb_toep3d", x.data_ptr(), smaps.data_ptr() if smaps is not None else None,
                      self._psf3[s].data_ptr(), u.data_ptr(), v.data_ptr(), out.data_ptr(), b, c, st._n.ctypes.data,
                      st._g.ctypes.data, tw[1].ctypes.data, x.data_ptr() if damp else None, float(damp),
                      _lib.stream_ptr(x.device))
            return out
        if self._lines is not None and B * C <= self._line_images:
            b, c = (B, C) if smaps is not None else (B * C, 1)
            line_normal(self._lines, s, x, smaps, out, b, c, 0, st.image_shape, damp)
            return out
        u = torch.empty(B, C, *st.grid_shape, dtype=torch.complex64, device=x.device)
        st.expand(x, smaps, u, B, C, 1.0, x_has_coils=smaps is None)
        U = st.fft(u)
        psf = self._psf_fft
        if psf is None:  # more coil images than lines are worth, for the first time
            psf = self._grid_psf()
            if made_now(self.device):
                self._psf_fft = psf
        st.psf_apply(U, psf[s], B * C, st.G)
        V = st.ifft(U)
        st.combine(V, smaps, out, B, C, 1.0, add=x if damp else None, add_scale=damp)
        return out

    def _apply_into(self, x: torch.Tensor, out: torch.Tensor, damp: float = 0.0) -> torch.Tensor:
        """One frame, stack element 0: ``out = A^H A x + damp * x``."""
        return self._apply_frames(x.reshape(1, *x.shape), 0, out.reshape(1, *out.shape), damp)

    def __call__(self, image):
        x = torch.as_tensor(image)
        src_dev = x.device
        sf = self.sparse_fft
        s_shape = self.stack_shape
        single_ndim = len(self.image_shape) + (0 if sf.smaps is not None else 1)
        prefix = tuple(int(s) for s in x.shape[: x.ndim - single_ndim])
        if s_shape:
            if len(prefix) < len(s_shape) or tuple(prefix[-len(s_shape):]) != s_shape:
                raise ValueError(f"image prefix {prefix} must end with stack_shape {s_shape}")
            B_shape = prefix[: len(prefix) - len(s_shape)]
        else:
            B_shape = prefix
        single = tuple(int(s) for s in x.shape[x.ndim - single_ndim:])
        S = int(np.prod(s_shape)) if s_shape else 1
        Bt = int(np.prod(B_shape)) if B_shape else 1
        xd = as_c64(x, self.device).reshape(Bt, S, *single)
        out = torch.empty_like(xd)
        for s in range(S):
            xs = xd[:, s].contiguous()
            os_ = torch.empty_like(xs) if S > 1 else out.view(xs.shape)
            self._apply_frames(xs, s, os_)
            if S > 1:
                out[:, s] = os_
        return out.reshape(x.shape).to(src_dev)
