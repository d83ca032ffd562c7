"""The product with the cap inside at the edges of its tiles, and which sizes take it: the bits of the product with the cap behind it."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo
from nanochat_b200 import ops

pytestmark = pytest.mark.gpu


def operands(rows, words, channels):
    gen = torch.Generator(device="cuda").manual_seed(rows + words)
    a = torch.randn(rows, channels, generator=gen, device="cuda").bfloat16()
    return a, (torch.randn(words, channels, generator=gen, device="cuda") * 20 * channels ** -0.5).bfloat16()


@pytest.mark.parametrize("rows,words,channels", [(1, 1, 8), (31, 5, 64), (33, 256, 64), (127, 300, 72), (128, 256, 64), (129, 257, 72), (256, 4, 8),
                                                 (257, 257, 72), (300, 1003, 200), (384, 255, 136), (511, 2305, 64), (2048, 320, 1536), (5000, 4100, 328)])
def test_edges(rows, words, channels):
    a, w = operands(rows, words, channels)
    cap = 30.0
    got = mo.linear_cap(a, w, cap)
    want = cap * torch.tanh(a.double() @ w.double().t() / cap)
    # fp32 sums of K exact products err by at most (K + 1) eps times the sum of their sizes, the cap adds a few roundings
    bound = (channels + 1) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()) + 8 * 2.0 ** -24 * want.abs()
    assert ops.read_status("cuda") == 0 and ((got.double() - want).abs() <= bound).all()


def test_special_values():
    a, w = torch.zeros(300, 8, device="cuda").bfloat16(), torch.zeros(3, 8, device="cuda").bfloat16()
    a[0, 0], a[1, 0], a[2, 0], a[299, 0], w[:, 0] = float("inf"), float("-inf"), float("nan"), 3e38, 1.0
    got = mo.linear_cap(a, w, 15.0)
    assert (got[0] == 15).all() and (got[1] == -15).all() and got[2].isnan().all() and (got[299] == 15).all() and (got[3:299] == 0).all()


# both sides of the rule
@pytest.mark.parametrize("rows,words,channels,inside", [(2048, 4096, 1024, True), (2048, 4096, 1016, False), (1000, 32768, 1536, True),
                                                        (257, 32768, 1536, False), (256, 16384, 2048, False), (300, 1000, 2048, False)])
def test_rule(monkeypatch, rows, words, channels, inside):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        assert mo.cap_in_product(rows, words, channels, sms) == inside
    taken, own = [], mo.linear_cap
    monkeypatch.setattr(mo, "linear_cap", lambda *a: (taken.append(1), own(*a))[1])
    a, w = operands(rows, words, channels)
    with mo.full_precision_sums():
        got, want = mo.capped_product(a, w, 30.0), mo.softcap(mo.product(a, w, f32_out=True), 30.0)
    assert bool(taken) == mo.cap_in_product(rows, words, channels, sms)
    torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-4)
