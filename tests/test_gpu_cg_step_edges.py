"""The one-launch CG vector step beside the three kernels that it stands in for: exact scalars, and values that
are not finite.

Both add FP32 products in FP64: n terms, relative to the sum of their magnitudes n 2^-53 < 2e-11 at n = 160,000, in
any order; the terms of |r|^2 are positive and those of <p, Ap> made so.
"""

import pytest
import torch

from pygrog_b200 import _lib

pytestmark = pytest.mark.gpu


def _run(dev, x, r, p, Ap, scal, fused):
    frames, n = x.shape
    words = (int(_lib.lib().pgb_reduce_scratch_bytes()) + 7) // 8
    scratch = torch.zeros(frames * words, dtype=torch.float64, device=dev)
    x, r, p, scal = (t.clone() for t in (x, r, p, scal))
    a = [t.data_ptr() for t in (x, r, p, Ap)]
    st = _lib.stream_ptr(dev)
    if fused:
        _lib.call("pgb_cg_step_batched", *a, n, frames, scal.data_ptr(), scratch.data_ptr(), st)
    else:
        _lib.call("pgb_dot_f64_batched", a[2], a[3], n, frames, scratch.data_ptr(), scal.data_ptr(), 1, 0, st)
        _lib.call("pgb_cg_update_xr_rr_batched", *a, n, frames, scal.data_ptr(), scratch.data_ptr(), st)
        _lib.call("pgb_cg_update_p_batched", a[2], a[1], n, frames, scal.data_ptr(), scratch.data_ptr(), st)
    return x, r, p, scal


def _state(dev, n, frames=3):
    g = torch.Generator(device=dev).manual_seed(n)
    x, r, p = (torch.randn(frames, n, dtype=torch.complex64, device=dev, generator=g) for _ in range(3))
    Ap = p * (torch.rand(frames, n, device=dev, generator=g) + 0.5)  # <p, Ap> of positive terms
    scal = torch.zeros(frames, 8, dtype=torch.float64, device=dev)
    scal[:, 0] = r.abs().double().square().sum(1)
    scal[:, 3] = scal[:, 0].sqrt()
    scal[:, 6] = 1e-9
    return x, r, p, Ap, scal


@pytest.mark.parametrize("n", [1, 511, 4096 * 4, 4096 * 8 - 1, 65536, 65537, 160000])
def test_scalars_are_summed_in_fp64(cuda, n):
    s = _state(cuda, n)
    x, r, p, scal = _run(cuda, *s, True)
    pap = (s[2].to(torch.complex128).conj() * s[3].to(torch.complex128)).real.sum(1)
    assert bool(((scal[:, 1] - pap).abs() <= 1e-10 * pap).all())
    rr = r.to(torch.complex128).abs().square().sum(1)  # of the residual that it stored
    assert bool(((scal[:, 2] - rr).abs() <= 1e-10 * rr).all())
    assert bool(((scal[:, 4] - rr.sqrt() / s[4][:, 3]).abs() <= 1e-10 * scal[:, 4]).all())


@pytest.mark.parametrize("n", [700, 40000, 160000])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["r", "p", "Ap"])
def test_values_that_are_not_finite(cuda, n, bad, where):
    """One frame of three: the same elements stop being finite, the flags agree, the others are untouched by it."""
    s = list(_state(cuda, n))
    clean = _run(cuda, *s, True)
    i = ("x", "r", "p", "Ap").index(where)
    s[i] = s[i].clone()
    s[i][1, n // 2] = complex(bad, 0.0)
    one, three = _run(cuda, *s, True), _run(cuda, *s, False)
    for a, b in zip(one[:3], three[:3]):
        assert torch.equal(torch.view_as_real(a).isnan(), torch.view_as_real(b).isnan())
        assert torch.equal(torch.view_as_real(a).isinf(), torch.view_as_real(b).isinf())
    assert torch.equal(one[3].isnan(), three[3].isnan()) and torch.equal(one[3][:, 5], three[3][:, 5])
    for a, b in zip(one, clean):
        assert torch.equal(a[[0, 2]], b[[0, 2]])
