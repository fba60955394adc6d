"""Which expansion ``interpolate`` takes for few coils, and that the result does not depend on it."""

import numpy as np
import pytest
import torch

from pygrog_b200 import _lib
from pygrog_b200.calib import GrogInterpolator
from pygrog_b200.calib._grog import expand_order
from pygrog_b200.workloads import radial2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,precision,ordered", [(1, 1, False), (2, 1, False), (4, 1, False), (6, 1, False), (8, 1, True),
                                                 (2, 2, True), (4, 2, True), (5, 2, True), (6, 2, True)])
def test_few_coils(cuda, C, precision, ordered):
    """Measured, sample order / ordered: 121 operators of 1 / 2 / 4 / 6 coils 0.8 / 0.98 / 1 / 0.95, of 8 1.35;
    10,201 of 2 / 4 / 5 / 6 on a small plan 1.73 / 1.84 / 1.47 / 1.64."""
    rng = np.random.default_rng(C)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    n, spokes, readout = 64, 12, 300
    g = GrogInterpolator(shape=(n, n), coords=radial2d(spokes, readout, n / 2.0), oversamp=1.0,
                         kernel_width=5 if precision == 2 else 3, kernel_shape="square", device=cuda)
    g.calc_interp_table(cplx(C, 12, 12), lamda=0.1, precision=precision)
    x = torch.from_numpy(cplx(C, spokes, readout)).to(cuda)
    idx = g._interp_idx.reshape(-1)
    K, kw = int(g._table_d.shape[0]), int(g.plan.target_idx.shape[-1])
    shared = expand_order(idx, K, C, kw) is not None  # runs long enough, as far as those go
    got = g.interpolate(x)
    assert (g._orders.get((0, C)) is not None) == (ordered and shared)
    assert shared or not ordered or precision == 2
    a = torch.empty(1, C, idx.numel(), dtype=torch.complex64, device=cuda)
    _lib.call("pgb_grog_expand", x.data_ptr(), spokes * readout, kw, idx.data_ptr(), g._table_d.data_ptr(), K, C, 1,
              a.data_ptr(), _lib.stream_ptr(cuda))
    assert torch.equal(got.reshape(a.shape), a)


def test_large_plans_of_5_and_6_coils_keep_the_sample_order(cuda):
    rng = np.random.default_rng(0)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    for C in (5, 6):
        g = GrogInterpolator(shape=(128, 128), coords=radial2d(100, 300, 64.0), oversamp=1.0, kernel_width=5,
                             kernel_shape="square", device=cuda)
        g.calc_interp_table(cplx(C, 12, 12), lamda=0.1, precision=2)
        g.interpolate(torch.from_numpy(cplx(C, 100, 300)).to(cuda))
        assert g.plan.target_idx.numel() > 600_000 and g._orders == {(0, C): None}
