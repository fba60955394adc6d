"""``stream_ptr`` takes every form of a device that ``torch.cuda.current_stream`` takes."""

from types import SimpleNamespace

import pytest
import torch

from pygrog_b200 import _lib


@pytest.mark.parametrize("device", [None, 0, "cuda", "cuda:0", torch.device("cuda"), torch.device("cuda", 0)])
def test_forms_of_a_device(monkeypatch, device):
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: 40 + i, raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: SimpleNamespace(cuda_stream=40))
    assert _lib.stream_ptr(device) == 40


def test_a_cpu_device_is_not_the_gpu_of_its_number(monkeypatch):
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: 40 + i, raising=False)

    def current(d=None):
        raise ValueError(f"Expected a cuda device, but got: {d}")

    monkeypatch.setattr(torch.cuda, "current_stream", current)
    with pytest.raises(ValueError):
        _lib.stream_ptr(torch.device("cpu", 0))
