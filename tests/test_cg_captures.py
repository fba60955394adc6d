"""How many graphs the solves of one right-hand side shape capture, and that they do not change the result."""

import numpy as np
import pytest
import torch

from pygrog_b200._solve import DeviceCG
from pygrog_b200.calib import GrogInterpolator
from pygrog_b200.operator import SparseFFT
from pygrog_b200.workloads import radial2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iters,captures", [(3, (0, 1, 0)), (5, (1, 0, 0)), (10, (1, 0, 0)), (13, (1, 1, 0))])
def test_the_first_solve_captures_once(cuda, monkeypatch, iters, captures):
    """As many as a single graph of one iteration would need, or none."""
    n, C = 64, 4
    g = GrogInterpolator(shape=(n, n), coords=radial2d(24, 96, n / 2.0), oversamp=1.0, kernel_width=2, device=cuda)
    rng = np.random.default_rng(iters)
    cplx = lambda *s: torch.from_numpy(  # noqa: E731
        (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).to(cuda)
    op = SparseFFT(plan=g.plan, smaps=cplx(C, n, n), toeplitz=True, device=cuda)
    y = [cplx(C, *op.natural_shape) for _ in range(3)]
    op.normal(cplx(n, n))  # the PSF, from here on the same
    made, whole = [], DeviceCG.capture

    def capture(self, iters=1):
        made.append(iters)
        return whole(self, iters)

    monkeypatch.setattr(DeviceCG, "capture", capture)
    for b, want in zip(y, captures):
        before = len(made)
        x = op.solve(b, method="cg", damp=1e-3, max_iter=iters, tol=0.0)
        assert len(made) - before == want
        eager = DeviceCG(op, op.adjoint(b), 1e-3, 0.0).run(iters, None, use_graph=False)
        assert torch.equal(x, eager)
