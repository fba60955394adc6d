"""Coil counts above the kernels' limit are refused with a message, whatever the mode."""

import numpy as np
import pytest
import torch

from pygrog_b200.calib import GrogInterpolator
from pygrog_b200.calib._grog import GrogGridder
from pygrog_b200.workloads import radial2d


def test_ordered_mode_above_32_coils():
    tgt, idx, w = torch.zeros(4, dtype=torch.int64), torch.zeros(4, dtype=torch.int64), torch.ones(4)
    with pytest.raises(ValueError, match="C <= 32"):
        GrogGridder(tgt, idx, w, 1, (8, 8), torch.zeros(9, 33, 33, dtype=torch.complex64), None, 3, mode="ordered")


@pytest.mark.gpu
def test_default_above_32_coils(cuda):
    rng = np.random.default_rng(0)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    g = GrogInterpolator(shape=(24, 24), coords=radial2d(8, 48, 12.0), oversamp=1.0, kernel_width=2, device=cuda)
    g.calc_interp_table(cplx(33, 10, 10), lamda=0.1, precision=1)
    with pytest.raises(RuntimeError, match="32"):
        g.grid(torch.from_numpy(cplx(33, 8, 48)).to(cuda))
