"""Soft-capped logits of many rows in one launch, at the edges of its tiles (256 rows by 256 words, 64 channels a step)."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo
from nanochat_b200 import ops

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("rows,words,channels", [(256, 4, 8), (256, 256, 64), (257, 257, 72), (300, 1003, 200), (384, 255, 136), (511, 2305, 64),
                                                 (2048, 320, 1536), (5000, 4100, 328)])
def test_capped_product(rows, words, channels):
    gen = torch.Generator(device="cuda").manual_seed(rows + words)
    a = torch.randn(rows, channels, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(words, channels, generator=gen, device="cuda") * 20 * channels ** -0.5).bfloat16()
    cap = 30.0
    got = mo.capped_product(a, w, cap)
    assert ops.read_status("cuda") == 0 and got.shape == (rows, words) and got.dtype == torch.float32
    want = cap * torch.tanh(a.double() @ w.double().t() / cap)
    # fp32 sums of K exact products err by at most (K + 1) eps times the sum of their sizes; the cap does not widen that
    # (its slope is at most one) and adds a few roundings of the result
    bound = (channels + 1) * EPS * (a.double().abs() @ w.double().abs().t()) + 8 * EPS * want.abs()
    assert ((got.double() - want).abs() <= bound).all()


def test_special_values_and_the_general_path():
    a, w = torch.zeros(256, 8, device="cuda").bfloat16(), torch.zeros(3, 8, device="cuda").bfloat16()
    a[0, 0], a[1, 0], a[2, 0], a[255, 0], w[:, 0] = float("inf"), float("-inf"), float("nan"), 3e38, 1.0
    got = mo.capped_product(a, w, 15.0)
    assert (got[0] == 15).all() and (got[1] == -15).all() and got[2].isnan().all() and (got[255] == 15).all() and (got[3:255] == 0).all()
    wide = torch.randn(300, 24, device="cuda").bfloat16()
    for x, v in ((wide[:, :16], w.new_ones(5, 16)), (wide[:255], w.new_ones(5, 24)), (wide[:, :20].contiguous(), w.new_ones(5, 20)),
                 (wide.float(), w.new_ones(5, 24).float())):  # strided, few rows, ragged channels, fp32
        want = 15 * torch.tanh(x.double() @ v.double().t() / 15)
        torch.testing.assert_close(mo.capped_product(x, v, 15.0).double(), want, rtol=1e-4, atol=1e-4)
    with pytest.raises(RuntimeError):
        mo.capped_product(wide, w.new_ones(5, 24), 0.0)
