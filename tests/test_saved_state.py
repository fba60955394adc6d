"""Objects saved by earlier versions, whose states lack what came later, load and work."""

import math
import pickle

import numpy as np
import pytest
import torch

from pygrog_b200.calib import GrogInterpolator
from pygrog_b200.calib._grog import GrogGridder
from pygrog_b200.operator import SparseFFT
from pygrog_b200.workloads import radial2d


def test_ordered_gridder_with_a_table():
    t = torch.zeros(5, 3, 3, dtype=torch.complex64)
    g = GrogGridder.__new__(GrogGridder)
    g.__setstate__({"mode": "ordered", "C": 3, "table": t, "table_h": t.mT})
    assert g.ops[0] is t and g.ops[1] is None and g.K == 5 and g.n_outer == 1 and g.max_batch == math.inf
    other = GrogGridder.__new__(GrogGridder)
    other.__setstate__({"mode": "v8", "C": 3})
    assert "ops" not in other.__dict__


def test_arrays_of_the_first_call_are_made_again():
    op = SparseFFT.__new__(SparseFFT)
    op.__setstate__({"_arrays": [object()], "ndim": 2})
    assert op._arrays is None and op.ndim == 2


def _old(state, new, **old):
    return {**{k: v for k, v in state.items() if k not in new}, **old}


@pytest.mark.gpu
def test_saved_objects_work(cuda):
    rng = np.random.default_rng(0)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    n, C = 64, 4
    g = GrogInterpolator(shape=(n, n), coords=radial2d(24, 96, n / 2.0), oversamp=1.0, kernel_width=2, device=cuda)
    g.calc_interp_table(cplx(C, 12, 12), lamda=0.1, precision=1)
    x = torch.from_numpy(cplx(C, 24, 96)).to(cuda)
    k, s = g.grid(x), g.degrid(g.grid(x))
    again = pickle.loads(pickle.dumps(g))  # as it is now
    assert torch.equal(again.grid(x), k) and torch.equal(again.degrid(k), s)
    bp = g._brick(0)
    assert bp.mode == "ordered" and bp.ops[1] is None
    old = GrogGridder.__new__(GrogGridder)
    old.__setstate__(_old(bp.__dict__, ("ops", "ops_h", "K", "n_outer", "max_batch", "_other", "_make_other"),
                          table=bp.ops[0], table_h=bp.ops_h[0]))
    g._brick_plans = {0: old}
    assert torch.equal(g.grid(x), k) and torch.equal(g.degrid(k), s)

    op = SparseFFT(plan=g.plan, smaps=torch.from_numpy(cplx(C, n, n)).to(cuda), toeplitz=True, device=cuda)
    y, img = torch.from_numpy(cplx(C, *op.natural_shape)).to(cuda), torch.from_numpy(cplx(n, n)).to(cuda)
    a, m = op.adjoint(y), op.normal(img)
    copy = pickle.loads(pickle.dumps(op))
    assert torch.equal(copy.adjoint(y), a) and torch.equal(copy.normal(img), m)
    toep = op._toep_op
    state = _old(toep.__dict__, ("_line_images",))
    toep.__dict__.clear()
    toep.__setstate__(state)
    assert torch.equal(op.normal(img), m)
