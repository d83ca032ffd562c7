"""Which strides the appends and the value gate hand to the library (0 means packed there)."""
import pytest
import torch

from nanochat_b200 import ops

wide = torch.zeros(6, 5, 40, 128, dtype=torch.bfloat16)
one = torch.zeros(1, 1, 3, 128, dtype=torch.bfloat16)


@pytest.mark.parametrize("t,want", [(wide, 5120), (wide[:, :1], 25600), (wide[:, :, 2:9], 5120), (wide[:, :, ::2], None), (wide[:, ::2], None),
                                    (one.expand(4, 1, 3, 128), None), (one.expand(4, 7, 3, 128), None), (one.expand(1, 7, 3, 128), None),
                                    (wide[:1, :1], 25600), (wide[..., 1:], None)])
def test_token_stride(t, want):
    assert ops._token_stride(t) == want


@pytest.mark.parametrize("t,want", [(wide, 0), (wide[:, :1], 25600), (wide[:, :, 2:9], 5120), (wide[:, :, ::2], None), (wide[:, ::2], None),
                                    (one.expand(4, 1, 3, 128), None), (one.expand(4, 7, 3, 128), None)])
def test_row_stride(t, want):
    assert ops._row_stride(t) == want
