"""Device state that an operator makes at its first call and keeps: replica lists, twiddles, PSF operators."""

import numpy as np
import pytest
import torch

from pygrog_b200 import _lib
from pygrog_b200._fftops import FFTStage
from pygrog_b200.calib import GrogInterpolator
from pygrog_b200.operator import SparseFFT, with_subspace
from pygrog_b200.operator._sparse_fft import _StackArrays
from pygrog_b200.workloads import kooshball, radial2d


@pytest.fixture
def recorded(monkeypatch):
    """CPU tensors and launches that do nothing, as inside a stream capture."""
    monkeypatch.setattr(_lib, "call", lambda *a: None)
    monkeypatch.setattr(_lib, "stream_ptr", lambda *a: 0)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)


def test_state_recorded_in_a_capture_is_not_kept(recorded):
    st = FFTStage((64, 80), (32, 40))
    assert st._lines(torch.device("cpu")) is not None
    assert st._tw == {}
    a = _StackArrays(st, torch.arange(50), torch.ones(50))
    a.to_grid(torch.zeros(1, 2, 50, dtype=torch.complex64), 1, 2)
    assert a._lists is None


def test_state_is_complete_before_it_is_kept(recorded, monkeypatch):
    st = FFTStage((64, 80), (32, 40))
    waits = []

    class Stream:
        def synchronize(self):
            waits.append(dict(st._tw))

    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream())
    st._lines(torch.device("cpu"))
    assert waits == [{}] and len(st._tw) == 1
    st._lines(torch.device("cpu"))
    assert len(waits) == 1


def _operators(ndim, dev):
    n, C = (24, 3) if ndim == 3 else (64, 4)
    coords = kooshball(60, 32, n / 2.0) if ndim == 3 else radial2d(24, 96, n / 2.0)
    g = GrogInterpolator(shape=(n,) * ndim, coords=coords, oversamp=64 / n if ndim == 3 else 1.0, kernel_width=2,
                         kernel_shape="sphere" if ndim == 3 else "circle", device=dev)
    rng = np.random.default_rng(ndim)
    cplx = lambda *s: torch.from_numpy(  # noqa: E731
        (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).to(dev)
    smaps, x = cplx(C, *(n,) * ndim), cplx(*(n,) * ndim)

    def make(toeplitz):
        return SparseFFT(plan=g.plan, smaps=smaps, toeplitz=toeplitz, device=dev)

    nat = make(False).natural_shape
    y, basis = cplx(C, *nat), cplx(3, nat[0])
    out = {"forward": (lambda: make(False), "forward", x), "adjoint": (lambda: make(False), "adjoint", y),
           "normal": (lambda: make(True), "normal", x)}
    if ndim == 2:
        sub = lambda t: with_subspace(make(t), basis, encoding_axis=-3)  # noqa: E731
        out["subspace adjoint"] = (lambda: sub(False), "adjoint", y)
        out["subspace forward"] = (lambda: sub(False), "forward", cplx(3, n, n))
        out["subspace normal"] = (lambda: sub(True), "normal", cplx(3, n, n))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("ndim", [2, 3])
def test_calls_between_a_first_capture_and_its_replay(cuda, ndim):
    """An operator captured at its very first call works outside the graph before the graph has run, and the
    graph afterwards: the same kernels in the same order, the same bits.  The normal operators' PSF is made by
    atomic sums, whose order varies: M <= 2304 terms a cell, sqrt-wise 48 eps = 3e-6 (eps = 6e-8)."""
    for name, (make, call, arg) in _operators(ndim, cuda).items():
        want = getattr(make(), call)(arg)
        op = make()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            inside = getattr(op, call)(arg)
        eager = getattr(op, call)(arg)
        graph.replay()
        torch.cuda.synchronize()
        for got in (eager, inside, getattr(op, call)(arg)):
            if "normal" in name:
                assert float((got - want).norm() / want.norm()) < 3e-6, name
            else:
                assert torch.equal(got, want), name


@pytest.mark.gpu
@pytest.mark.parametrize("ndim", [2, 3])
def test_first_call_on_one_stream_second_on_another(cuda, ndim):
    """What the first call makes behind queued work is complete for a call on another stream."""
    for name, (make, call, arg) in _operators(ndim, cuda).items():
        want = getattr(make(), call)(arg)
        op = make()
        torch.cuda.synchronize()
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        with torch.cuda.stream(a):
            torch.cuda._sleep(10_000_000)  # some milliseconds
            first = getattr(op, call)(arg)
        with torch.cuda.stream(b):
            second = getattr(op, call)(arg)
        torch.cuda.synchronize()
        for got in (first, second):
            if "normal" in name:  # atomic sums in the PSF, as above
                assert float((got - want).norm() / want.norm()) < 3e-6, name
            else:
                assert torch.equal(got, want), name


@pytest.mark.gpu
def test_gridder_made_on_one_stream_used_on_another(cuda):
    rng = np.random.default_rng(0)
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    g = GrogInterpolator(shape=(48, 48), coords=radial2d(30, 96, 24.0), oversamp=1.0, kernel_width=2, device=cuda)
    g.calc_interp_table(cplx(6, 12, 12), lamda=0.1, precision=1)
    x = torch.from_numpy(cplx(6, 30, 96)).to(cuda)
    want = g.grid(x)
    back = g.degrid(want)
    g._brick_plans = None
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(10_000_000)
        first = g.grid(x)
    with torch.cuda.stream(b):
        second, samples = g.grid(x), g.degrid(want)
    torch.cuda.synchronize()
    assert torch.equal(first, want) and torch.equal(second, want) and torch.equal(samples, back)
