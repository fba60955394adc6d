"""Shared GPU stages of the Cartesian operators: cuFFT plus the pointwise
kernels of ``csrc/fft_stage.cu``.

Buffers passed to cuFFT are kept in FFT order (centred index p stored at
m = (p - g//2) mod g), so the centred ortho transforms of the reference
(``_base/_fftc.py:114-139``: ifftshift -> fftn -> fftshift, ortho) become
one unscaled transform with the index maps and the ortho scale folded into
its ends: the library's own line FFTs where the grid's lengths are built
(``csrc/line_fft.cu``), cuFFT between two index-remapping kernels elsewhere.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from . import _lib


def with_torch(fn):
    """numpy arrays in -> torch tensors inside -> numpy arrays out (container only)."""

    @functools.wraps(fn)
    def wrapper(*args, **kwargs):
        was_numpy = any(isinstance(a, np.ndarray) for a in args) or any(
            isinstance(v, np.ndarray) for v in kwargs.values()
        )
        args = tuple(torch.as_tensor(a) if isinstance(a, np.ndarray) else a for a in args)
        kwargs = {k: (torch.as_tensor(v) if isinstance(v, np.ndarray) else v) for k, v in kwargs.items()}
        out = fn(*args, **kwargs)
        if was_numpy and isinstance(out, torch.Tensor):
            return out.detach().cpu().numpy()
        return out

    return wrapper


def compute_device(device) -> torch.device:
    """The CUDA device that runs the kernels (the reference's ``device`` argument
    may name the CPU; computation here is always on a GPU)."""
    if device is not None:
        d = torch.device(device)
        if d.type == "cuda":
            return d
    return torch.device("cuda", torch.cuda.current_device() if torch.cuda.is_available() else 0)


def made_now(device) -> bool:
    """Whether device state just made on the current stream may be kept for later calls, which may come from any
    stream: it is complete on return.

    In a stream capture it is only recorded: it exists while that graph runs, so the caller uses it and
    keeps nothing."""
    if torch.cuda.is_current_stream_capturing():
        return False
    torch.cuda.current_stream(device).synchronize()
    return True


class FFTStage:
    """Shapes and launchers for one (grid_shape, image_shape) pair."""

    def __init__(self, grid_shape, image_shape):
        self.grid_shape = tuple(int(s) for s in grid_shape)
        self.image_shape = tuple(int(s) for s in image_shape)
        self.ndim = len(self.grid_shape)
        if self.ndim not in (2, 3):
            raise ValueError(f"only 2-D and 3-D grids are supported, got {self.ndim}-D")
        if len(self.image_shape) != self.ndim:
            raise ValueError("image_shape and grid_shape must have the same length")
        self.G = int(np.prod(self.grid_shape))
        self.I = int(np.prod(self.image_shape))
        self.axes = tuple(range(-self.ndim, 0))
        self._g = np.ascontiguousarray(self.grid_shape, dtype=np.int64)
        self._n = np.ascontiguousarray(self.image_shape, dtype=np.int64)
        self.ortho = 1.0 / math.sqrt(self.G)
        self.__setstate__({})

    def __getstate__(self):
        # the twiddles and the shape go with their addresses: a copy makes its own
        return {**self.__dict__, "_tw": {}}

    def __setstate__(self, state):
        self.__dict__.update(state, _tw={})
        self._g_ptr = self._g.ctypes.data

    # -- transforms with the coil maps ----------------------------------------
    def _lines(self, device):
        """Twiddles of the grid's own line lengths, ``(tensors, their addresses)``; ``None`` where a length is
        not built.

        Measured (coils x grid, image; to the grid / to the image, us, cuFFT with its expansion or combine
        pass against lines): 8 x 128^2 38 / 34 against 23 / 20 (launches), 16 x 640^2, 320^2 83 / 79 against
        44 / 50, 24 x 768^2, 384^2 196 / 186 against 92 / 107, 8 x 900^2, 600^2 72 / 68 against 61 / 62; at
        1024^2 the columns' 32 x 32 stages lose: 16 coils, 512^2 147 / 139 against 127 / 146, 8 coils, 1024^2
        98 / 107 against 138 / 123.
        """
        key = device.index if device.index is not None else torch.cuda.current_device()
        if key not in self._tw:
            tw = None
            if all(g in line_lengths() and g < 1024 for g in self.grid_shape):
                lib, st = _lib.lib(), _lib.stream_ptr(device)
                tw = [torch.empty(lib.pgb_fft_twiddles(g), dtype=torch.complex64, device=device) for g in self.grid_shape]
                for d, g in enumerate(self.grid_shape[:-2]):
                    _lib.call("pgb_fft_twiddle_tables", g, 0, tw[d].data_ptr(), None, st)
                _lib.call("pgb_fft_twiddle_tables", *self.grid_shape[-2:], tw[-2].data_ptr(), tw[-1].data_ptr(), st)
                tw = (tw, np.array([t.data_ptr() for t in tw], dtype=np.uint64))
                if not made_now(device):
                    return tw
            self._tw[key] = tw
        return self._tw[key]

    def _line_work(self, grid: torch.Tensor, B: int, C: int) -> tuple:
        """Buffers of the passes between an image and its grid: ``(after the rows, before z)``; the grid itself
        along axes without padding."""
        g, n = self.grid_shape, self.image_shape
        z = grid if self.ndim == 2 or n[0] == g[0] else torch.empty(
            B * C * n[0] * g[1] * g[2], dtype=grid.dtype, device=grid.device)
        y = z if n[-2] == g[-2] else torch.empty(
            B * C * (n[0] if self.ndim == 3 else 1) * n[-2] * g[-1], dtype=grid.dtype, device=grid.device)
        return y, z

    def to_grid(self, x, smaps, B: int, C: int) -> torch.Tensor:
        """FFT-order grids ``(B, C, *grid)`` of images ``x`` (``(B, *image)`` with ``smaps``, else
        ``(B, C, *image)``): maps, zero padding and the unscaled forward transform."""
        u = torch.empty(B, C, *self.grid_shape, dtype=torch.complex64, device=x.device)
        tw = self._lines(x.device)
        if tw is None:
            self.expand(x, smaps, u, B, C, 1.0, x_has_coils=smaps is None)
            return self.fft(u)
        y, z = self._line_work(u, B, C)
        b, c = (B, C) if smaps is not None else (B * C, 1)
        _lib.call("pgb_line_to_grid", x.data_ptr(), smaps.data_ptr() if smaps is not None else None, y.data_ptr(),
                  z.data_ptr(), u.data_ptr(), b, c, self.ndim, self._n.ctypes.data, self._g.ctypes.data,
                  tw[1].ctypes.data, _lib.stream_ptr(x.device))
        return u

    def to_image(self, u, smaps, out, B: int, C: int, scale: float, add=None, add_scale: float = 0.0):
        """``out`` from grids ``u (B, C, *grid)`` in FFT order (overwritten): unscaled inverse transform, crop
        and coil sum (``(B, *image)`` with ``smaps``, else ``(B, C, *image)``), times ``scale``, plus
        ``add_scale * add``."""
        tw = self._lines(u.device)
        if tw is None:
            return self.combine(self.ifft(u), smaps, out, B, C, scale, add, add_scale)
        y, z = self._line_work(u, B, C)
        b, c = (B, C) if smaps is not None else (B * C, 1)
        _lib.call("pgb_line_to_image", u.data_ptr(), smaps.data_ptr() if smaps is not None else None, y.data_ptr(),
                  z.data_ptr(), out.data_ptr(), b, c, self.ndim, self._n.ctypes.data, self._g.ctypes.data,
                  tw[1].ctypes.data, float(scale), add.data_ptr() if add is not None else None, float(add_scale),
                  _lib.stream_ptr(u.device))
        return out

    # -- index maps ---------------------------------------------------------
    def fft_order_index(self, centred_flat: torch.Tensor) -> torch.Tensor:
        """FFT-order flat index of centred flat grid indices."""
        idx = centred_flat.to(torch.int64)
        out = torch.zeros_like(idx)
        rem = idx
        mult = 1
        for d in reversed(range(self.ndim)):
            g = self.grid_shape[d]
            p = rem % g
            rem = rem // g
            m = (p - g // 2) % g
            out = out + m * mult
            mult *= g
        return out

    def to_fft_order(self, grid_centred: torch.Tensor) -> torch.Tensor:
        """Real or complex array (..., *grid) centred -> FFT order (ifftshift)."""
        return torch.fft.ifftshift(grid_centred, dim=self.axes)

    # -- launchers --------------------------------------------------------------
    def expand(self, x, smaps, u, B, C, scale, x_has_coils):
        _lib.call(
            "pgb_fft_expand", x.data_ptr(), smaps.data_ptr() if smaps is not None else None, u.data_ptr(),
            B, C, self.ndim, self._g.ctypes.data, self._n.ctypes.data, float(scale), int(x_has_coils),
            _lib.stream_ptr(u.device),
        )
        return u

    def combine(self, v, smaps, out, B, C, scale, add=None, add_scale=0.0):
        _lib.call(
            "pgb_fft_combine", v.data_ptr(), smaps.data_ptr() if smaps is not None else None, out.data_ptr(),
            B, C, self.ndim, self._g.ctypes.data, self._n.ctypes.data, float(scale),
            add.data_ptr() if add is not None else None, float(add_scale), _lib.stream_ptr(v.device),
        )
        return out

    def shift(self, src, mask, dst, BC, scale, to_centred):
        _lib.call(
            "pgb_fft_shift", src.data_ptr(), mask.data_ptr() if mask is not None else None, dst.data_ptr(),
            BC, self.ndim, self._g.ctypes.data, float(scale), int(to_centred), _lib.stream_ptr(src.device),
        )
        return dst

    def fft(self, u):
        """Unscaled forward DFT over the grid axes of an FFT-order buffer."""
        return torch.fft.fftn(u, dim=self.axes, norm="backward")

    def ifft(self, U):
        """Unscaled inverse DFT over the grid axes."""
        return torch.fft.ifftn(U, dim=self.axes, norm="forward")

    def cell_sum(self, data, lists, w, u, B, C, R, tix=None, basis=None):
        """Grid ``u (B, [K,] C, *grid)`` in FFT order from samples ``data (B, C, R)``; every cell is written.
        ``w`` (and ``tix``): the weights (and basis columns) of the listed replicas."""
        K, T = basis.shape if basis is not None else (1, 0)
        n_seg, n_cells = lists.seg.shape[0], lists.cells.shape[0]
        part = torch.empty(B * K * C * n_seg, dtype=torch.complex64, device=u.device) if n_cells else None
        _lib.call("pgb_cell_sum", data.data_ptr(), lists.start.data_ptr(), lists.src.data_ptr(), w.data_ptr(),
                  tix.data_ptr() if tix is not None else None, basis.data_ptr() if basis is not None else None, T,
                  u.data_ptr(), B, C, K, R, self.ndim, self._g_ptr, lists.seg.data_ptr(), n_seg,
                  lists.cells.data_ptr(), n_cells, part.data_ptr() if n_cells else None, _lib.stream_ptr(u.device))
        return u

    @staticmethod
    def gather(U, cellpos, w, out, BC, R, G):
        _lib.call("pgb_sparse_gather", U.data_ptr(), cellpos.data_ptr(), w.data_ptr(), out.data_ptr(),
                  BC, R, G, _lib.stream_ptr(U.device))

    @staticmethod
    def psf_apply(U, psf, BC, G):
        _lib.call("pgb_psf_apply", U.data_ptr(), psf.data_ptr(), BC, G, _lib.stream_ptr(U.device))


class CellLists:
    """The replicas that have a weight and a cell, listed by cell for ``csrc/cell_sum.cu``.

    ``rep``: their numbers by cell (in a cell ascending), ``src`` the same as int32, ``start``: each cell
    slot's range in them; ``seg`` / ``cells``: the cuts of the long lists and the cells with more than one.
    Built on the device from ``cellpos`` (FFT-order cell, int32) and ``w``; outside a stream capture the
    array lengths are read back, inside one they are upper bounds and the rest stays empty.
    """

    def __init__(self, grid_shape, cellpos: torch.Tensor, w: torch.Tensor):
        dev, nd = cellpos.device, len(grid_shape)
        capturing = torch.cuda.is_current_stream_capturing()
        g = np.ascontiguousarray(grid_shape, dtype=np.int64)
        slots = _lib.lib().pgb_cell_slots(nd, g.ctypes.data)
        R = int(cellpos.numel())
        st = _lib.stream_ptr(dev)
        key = torch.empty(R, dtype=torch.int32, device=dev)
        _lib.call("pgb_cell_keys", cellpos.data_ptr(), w.data_ptr(), R, nd, g.ctypes.data, key.data_ptr(), st)
        small = R <= 2**22  # a small sort costs less than telling the others apart first
        if capturing or small:  # the replicas without a cell stay in the list, past its end
            key, self.rep = torch.sort(key, stable=True)
        else:
            r = torch.nonzero(key < slots).squeeze(1)
            key, perm = torch.sort(key[r], stable=True)
            self.rep = r[perm]
        self.src = self.rep.to(torch.int32)
        self.start = torch.searchsorted(key, torch.arange(slots + 1, dtype=torch.int32, device=dev), out_int32=True)
        most = np.zeros(2, dtype=np.int64)
        _lib.lib().pgb_cell_bounds(int(key.numel()), most.ctypes.data)
        rows = torch.zeros(int(most.sum()) + 1, 4, dtype=torch.int32, device=dev)
        count, self.seg, self.cells = rows[0], rows[1 : 1 + int(most[0])], rows[1 + int(most[0]) :]
        _lib.call("pgb_cell_segments", self.start.data_ptr(), nd, g.ctypes.data, self.seg.data_ptr(),
                  self.cells.data_ptr(), count.data_ptr(), st)
        if not capturing:
            n_seg, n_cells = count[:2].tolist()
            self.seg, self.cells = self.seg[:n_seg], self.cells[:n_cells]
            if not small:  # do not keep the upper bounds
                self.seg, self.cells = self.seg.clone(), self.cells.clone()


@functools.lru_cache(maxsize=1)
def line_lengths() -> tuple:
    """Lengths of the library's own line FFTs, ascending (``csrc/fft_core.cuh``)."""
    out = []
    while n := _lib.lib().pgb_fft_length(len(out)):
        out.append(n)
    return tuple(out)


def as_c64(t: torch.Tensor, device) -> torch.Tensor:
    """complex64, contiguous, on ``device`` (the kernels compute in complex64)."""
    t = torch.as_tensor(t)
    if t.dtype != torch.complex64:
        if t.is_complex() or t.is_floating_point():
            t = t.to(torch.complex64)
        else:
            raise TypeError(f"expected a complex tensor, got {t.dtype}")
    return t.to(device).contiguous()
