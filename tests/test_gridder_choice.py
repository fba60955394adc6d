"""Which kernels the default gridder takes, by plan and by batch, and that they agree."""

import math

import numpy as np
import pytest
import torch

from pygrog_b200.calib import GrogInterpolator
from pygrog_b200.calib._grog import GrogGridder
from pygrog_b200.workloads import kooshball, radial2d


def _limit(C, other, run):
    g = GrogGridder.__new__(GrogGridder)
    g.C = C
    return g._order_limit(other, run)


# replicas (frames times the plan's), coils, family, run: time of the other family over the ordered kernels' time
@pytest.mark.parametrize("work,C,other,run,gain", [
    (80e3, 12, ("v8", (4, 8, 8)), 1.13, 1.55), (144e3, 4, ("v8", (8, 8, 8)), 1.23, 1.14),
    (250e3, 12, ("v8", (4, 8, 8)), 1.19, 0.86), (420e3, 11, ("v8", (4, 8, 8)), 1.33, 0.80),
    (600e3, 13, ("v8", (2, 4, 8)), 1.2, 1.5), (43e6, 13, ("v8", (2, 4, 8)), 1.29, 1.05),
    (33e3, 8, ("v8", (1, 16, 32)), 1.01, 2.09), (524e3, 8, ("v8", (1, 16, 32)), 1.01, 0.87),
    (179e3, 11, ("v8", (1, 16, 32)), 1.04, 0.80), (197e3, 8, ("v8", (1, 16, 32)), 12.1, 1.51),
    (246e3, 8, ("v8", (1, 16, 32)), 8.4, 1.25), (394e3, 9, ("v8", (1, 16, 32)), 12.1, 1.36),
    (358e3, 13, ("v8", (1, 16, 32)), 5.2, 0.87), (538e3, 16, ("v8", (1, 16, 32)), 5.6, 0.93),
    (1.2e6, 16, ("global", None), 1.27, 1.42), (3e6, 32, ("global", None), 1.15, 1.35),
    (288e3, 31, ("global", None), 1.11, 1.90), (420e3, 31, ("global", None), 1.16, 0.81),
    (800e3, 15, ("global", None), 1.25, 0.65), (420e3, 20, ("global", None), 1.21, 1.41),
    (1.2e6, 17, ("global", None), 1.23, 0.54), (2.9e6, 31, ("global", None), 2.88, 1.3),
])
def test_rule_follows_the_measurements(work, C, other, run, gain):
    assert (work <= _limit(C, other, run)) == (gain > 1)
    assert _limit(C, other, math.inf) >= _limit(C, other, run)  # the bound before the runs are known


# replicas of the plan, frames, coils, replicas a cell
@pytest.mark.parametrize("V,frames,C,density,gain", [
    (137e3, 16, 8, 0.07, 1.53), (432e3, 4, 12, 0.11, 1.27), (388e3, 1, 8, 0.13, 1.17), (344e3, 1, 12, 0.16, 1.17),
    (516e3, 1, 8, 0.25, 0.86), (344e3, 2, 4, 0.16, 0.91), (388e3, 1, 4, 0.13, 1.25), (388e3, 4, 4, 0.13, 0.96), (188e3, 1, 6, 0.13, 1.17), (188e3, 2, 6, 0.13, 0.92),
    (1080e3, 1, 12, 0.26, 0.83),
])
def test_rule_for_sparse_3d_plans(V, frames, C, density, gain):
    g = GrogGridder.__new__(GrogGridder)
    g.C = C
    limit = g._order_limit(("v8", (8, 8, 8)), 1.1, density, V)
    assert (V * frames <= limit) == (gain > 1)
    assert g._order_limit(("v8", (8, 8, 8)), math.inf, density, V) >= limit


def _gridder(dev, ndim, n, spokes, readout, C, **kw):
    rng = np.random.default_rng(n)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    coords = (radial2d if ndim == 2 else kooshball)(spokes, readout, n / 2.0)
    g = GrogInterpolator(shape=(n,) * ndim, coords=coords, oversamp=1.0, kernel_width=2,
                         kernel_shape="circle" if ndim == 2 else "sphere", device=dev)
    g.calc_interp_table(cplx(C, *(10,) * ndim), lamda=0.1, precision=1)
    return g, lambda B: torch.from_numpy(cplx(B, C, spokes, readout)).to(dev)


@pytest.mark.gpu
@pytest.mark.parametrize("C", [6, 11])
def test_large_3d_plans_keep_the_brick_kernels(cuda, C):
    g, _ = _gridder(cuda, 3, 64, 3000, 128, C)
    V = int((g.plan.target_idx >= 0).sum())
    assert V > 256e3 and g._brick(0).mode == "v8"


@pytest.mark.gpu
@pytest.mark.parametrize("ndim,n,spokes,readout,C", [(3, 32, 300, 48, 5), (2, 64, 40, 128, 12), (2, 48, 30, 96, 20)])
def test_batches_take_the_faster_family_and_agree(cuda, ndim, n, spokes, readout, C):
    """Frames one by one (ordered) against a batch above the limit (the other family): both within the bound of
    the brick kernels' own tests, 1e-5 of the FP64 result, so 2e-5 of each other."""
    g, make = _gridder(cuda, ndim, n, spokes, readout, C)
    bp = g._brick(0)
    assert bp.mode == "ordered"
    bp.max_batch = 2  # (a limit that a test can pass)
    x = make(3)
    k = g.grid(x)
    s = g.degrid(k)
    other = bp._other
    assert other is not None and other.mode == ("global" if C > 16 else "v8")
    for i in range(3):
        ki = g.grid(x[i])
        assert float((ki - k[i]).norm() / ki.norm()) < 2e-5
        si = g.degrid(k[i])
        assert float((si - s[i]).norm() / si.norm()) < 2e-5
    assert g._brick(0)._other is other


@pytest.mark.gpu
def test_a_capture_takes_what_exists(cuda):
    g, make = _gridder(cuda, 2, 64, 40, 128, 6)
    g._brick(0).max_batch = 1
    x = make(2)
    want = torch.stack([g.grid(x[0]), g.grid(x[1])])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        k = g.grid(x)
    graph.replay()
    torch.cuda.synchronize()
    assert g._brick(0)._other is None and torch.equal(k, want)


@pytest.mark.gpu
def test_slices_of_a_batch(cuda, monkeypatch):
    """A batch whose shifted replicas exceed the workspace is taken in slices, with the same bits."""
    from pygrog_b200.calib import _grog

    g, make = _gridder(cuda, 2, 64, 40, 128, 6)
    x = make(5)
    k = g.grid(x)
    s = g.degrid(k)
    bp = g._brick(0)
    monkeypatch.setattr(_grog, "_ORDERED_BYTES", 2 * (8 * 6 * bp.plan.n_valid + 1))
    taken, whole = [], GrogGridder._ordered

    def seen(self, x, *a):
        taken.append(x.shape[0])
        return whole(self, x, *a)

    monkeypatch.setattr(GrogGridder, "_ordered", seen)
    assert torch.equal(g.grid(x), k) and torch.equal(g.degrid(k), s)
    assert taken[1:4] == taken[5:] and sum(taken[1:4]) == 5


@pytest.mark.gpu
def test_hot_cell_on_the_brick_kernels(cuda):
    """20,000 samples in one cell: the brick kernels split the brick and add its parts."""
    n, C = 32, 4
    rng = np.random.default_rng(0)
    coords = np.zeros((1, 20000, 2), dtype=np.float32)
    coords[0, :, 0] = np.linspace(-1e-3, 1e-3, 20000)
    coords[0, 0, :] = [n / 2 - 1, n / 2 - 1]  # sets the coordinate scale of both axes
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    g = GrogInterpolator(shape=(n, n), coords=coords, oversamp=1.0, kernel_width=1, device=cuda)
    g.calc_interp_table(cplx(C, 8, 8), precision=1)
    x = torch.from_numpy(cplx(C, 1, 20000)).to(cuda)
    want = g.grid(x)
    back = g.degrid(want)
    g.gridder_mode, g._brick_plans = "v8", None
    k = g.grid(x)
    bp = g._brick(0)
    assert bp.mode == "v8"
    assert float((k - want).norm() / want.norm()) < 2e-5 and float((g.grid(x) - k).norm() / k.norm()) < 1e-6
    assert float((g.degrid(want) - back).norm() / back.norm()) < 2e-5
