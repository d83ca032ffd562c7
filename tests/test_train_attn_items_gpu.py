"""The backward kernels where a CTA works on several blocks one after the other (more blocks than SMs)."""
import pytest

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
