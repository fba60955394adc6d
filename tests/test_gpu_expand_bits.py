"""The ordered expansion against the sample-ordered one, whether ordering pays or not: the same bits."""

import pytest
import torch

from pygrog_b200 import _lib
from pygrog_b200.calib._grog import expand_order

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 2, 3, 4, 6, 7, 8, 12, 13, 16, 20, 31, 32])
@pytest.mark.parametrize("N,kw,K,B", [(1, 3, 5, 1), (33, 1, 4000, 2), (700, 4, 121, 1), (5000, 25, 10201, 1)])
def test_same_bits(cuda, C, N, kw, K, B):
    g = torch.Generator(device=cuda).manual_seed(N + C)
    idx = torch.randint(-1, K + 1, (N * kw,), device=cuda, generator=g)  # two of them outside the table
    table = torch.randn(K, C, C, dtype=torch.complex64, device=cuda, generator=g)
    x = torch.randn(B, C, N, dtype=torch.complex64, device=cuda, generator=g)
    order = expand_order(idx, K, C, kw, always=True)
    if order is None:
        assert _lib.lib().pgb_grog_expand_chunk(N, C, kw) == 0 or _lib.lib().pgb_grog_expand_chunk(N, C, kw) * kw > 16384
        return
    order, entry, runs = order
    assert 1 <= int(runs) <= N * kw
    a, b = (torch.full((B, C, N * kw), float("nan"), dtype=torch.complex64, device=cuda) for _ in range(2))
    st = _lib.stream_ptr(cuda)
    _lib.call("pgb_grog_expand", x.data_ptr(), N, kw, idx.data_ptr(), table.data_ptr(), K, C, B, a.data_ptr(), st)
    _lib.call("pgb_grog_expand_sorted", x.data_ptr(), N, None, 0, kw, order.data_ptr(), entry.data_ptr(), table.data_ptr(),
              K, C, B, b.data_ptr(), st)
    assert torch.equal(a, b)
