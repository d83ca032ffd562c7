"""The backward kernels where a CTA works on several blocks one after the other (more blocks than SMs)."""
import pytest
import torch

from nanochat_b200.flash_attention import flash_attn
from tests.test_train_attn_gpu import test_flash_attn_func_forward_and_backward as at_sizes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,Hq,Hkv,window", [
    (150, 64, 1, 1, -1),   # a CTA or two with two blocks of a single step each
    (40, 70, 12, 12, -1),
    (30, 129, 16, 4, 7),   # blocks of very different lengths, four q heads per kv head
    (16, 300, 12, 12, -1),
    (13, 520, 12, 6, 100),
    (4, 1100, 12, 12, -1),
])
def test_more_blocks_than_sms(B, T, Hq, Hkv, window):
    at_sizes(B, T, Hq, Hkv, window)


def test_a_row_sum_for_itself_and_four_at_a_time():
    """Each text's gradients, in a batch whose row sums are taken four at a time and alone: the same bits."""
    B, T, H = 21, 171, 12  # 43092 rows, the last four of a half-warp not all there
    gen = torch.Generator(device="cuda").manual_seed(4)
    q, k, v, g = (torch.randn(B, T, H, 128, generator=gen, device="cuda").bfloat16() for _ in range(4))

    def grads(part):
        ts = [t[part].clone().requires_grad_() for t in (q, k, v)]
        return torch.autograd.grad(flash_attn.flash_attn_func(*ts, causal=True, window_size=(-1, 0)), ts, g[part])

    whole = grads(slice(None))
    for b in range(0, B, 4):
        for got, want in zip(grads(slice(b, b + 1)), whole):
            assert torch.equal(got[0], want[b])
