"""Right-hand sides that a CG solver's buffers take, as ``Tensor.copy_`` takes them."""

import pytest
import torch

from pygrog_b200 import _lib
from pygrog_b200._solve import BatchedDeviceCG, DeviceCG


@pytest.fixture
def seen(monkeypatch):
    """CPU tensors; the launches' first tensors, read back as the kernel would."""
    got = []

    def call(name, *args):
        if name == "pgb_cg_start_batched":
            import ctypes

            n, frames = args[4], args[5]
            buf = (ctypes.c_float * (2 * n * frames)).from_address(args[0])
            got.append(torch.view_as_complex(torch.tensor(list(buf)).reshape(frames, n, 2)))

    monkeypatch.setattr(_lib, "call", call)
    monkeypatch.setattr(_lib, "stream_ptr", lambda *a: 0)
    return got


def _forms(b):
    yield b
    yield b.to(torch.complex128)
    yield b.mT.contiguous().mT  # another stride order
    yield b.conj().resolve_conj().conj()  # a lazy conjugate
    yield b.real.clone()
    yield b[..., :1].clone()  # broadcast


def test_batched_start_reads_what_copy_would_write(seen):
    cg = BatchedDeviceCG(None, 3, (5, 6), "cpu")
    for b in _forms(torch.randn(2, 5, 6, dtype=torch.complex64)):
        want = torch.empty(2, 5, 6, dtype=torch.complex64).copy_(b)
        cg.load(b)
        assert torch.equal(seen[-1].reshape(2, 5, 6), want)
    n = len(seen)
    for shape in ((2, 5, 5), (2, 4, 6), (2, 30), (1, 5, 12)):
        with pytest.raises(RuntimeError):
            cg.load(torch.zeros(shape, dtype=torch.complex64))
    assert len(seen) == n


def test_reset_reads_what_copy_would_write(seen):
    cg = DeviceCG(None, torch.zeros(5, 6, dtype=torch.complex64), 0.0, 0.0)
    for b in _forms(torch.randn(5, 6, dtype=torch.complex64)):
        want = torch.empty(5, 6, dtype=torch.complex64).copy_(b)
        cg.reset(b)
        assert torch.equal(seen[-1].reshape(5, 6), want)
    n = len(seen)
    for shape in ((5, 5), (7, 6), (30,)):
        with pytest.raises(RuntimeError):
            cg.reset(torch.zeros(shape, dtype=torch.complex64))
    assert len(seen) == n
