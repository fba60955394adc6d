"""The autotuner beside what an interpolator takes untuned."""

import numpy as np
import pytest
import torch

from pygrog_b200.calib import GrogInterpolator, autotune_gridder
from pygrog_b200.calib._autotune import clear_cache
from pygrog_b200.workloads import radial2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [8, 20])
def test_the_default_stays_where_it_is_the_fastest(cuda, C):
    rng = np.random.default_rng(C)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    g = GrogInterpolator(shape=(96, 96), coords=radial2d(60, 192, 48.0), oversamp=1.0, kernel_width=2, device=cuda)
    g.calc_interp_table(cplx(C, 12, 12), lamda=0.1, precision=1)
    assert g._brick(0).mode == "ordered"
    x = torch.from_numpy(cplx(C, 60, 192)).to(cuda)
    want = g.grid(x)
    clear_cache()
    for cached in (False, True):
        res = autotune_gridder(g, tolerance=1e-6, reps=5)
        assert res["cached"] == cached and res["default_ms"] > 0
        stays = res["default_ms"] <= res["ms"]
        assert (res["installed"] is None) == stays
        assert (g.gridder_mode, g.gridder_brick) == ((None, None) if stays else (res["mode"], res["brick"]))
        assert g._brick(0).mode == ("ordered" if stays else res["mode"])
        assert float((g.grid(x) - want).norm() / want.norm()) < 2e-5
    clear_cache()
    res = autotune_gridder(g, tolerance=1e-6, reps=1, families=["global"])  # asked for: nothing else
    assert res["default_ms"] is None and g.gridder_mode == "global"
    clear_cache()
