"""The bits of the delta rule in chunks, pinned.  The router behind it chooses among scores that nearly tie: with sums in another order, 2e-6 of an
output, 17 to 49 of a prompt's 6007 tokens took other experts in each of the layers that follow, and logits moved by 1 to 3 percent."""
import hashlib

import pytest
import torch

from nanochat_b200 import mixer_ops as mo
from nanochat_b200 import ops

pytestmark = pytest.mark.gpu


def spread(seed, *shape):
    """Values in [-1, 1) that every machine makes alike."""
    i = torch.arange(torch.Size(shape).numel(), dtype=torch.int64) + seed * 1000003
    i = (i * 2654435761 + 12345) % (1 << 32)
    i = ((i ^ (i >> 15)) * 2246822519) % (1 << 32)
    return (((i ^ (i >> 13)) % (1 << 20)).float() * 2.0 ** -19 - 1).view(shape).cuda()


# heads that share columns among warps and heads that do not, all paddings of the channels, ragged chunks and columns
@pytest.mark.parametrize("B,T,H,G,Dk,Dv,digest", [
    (1, 250, 12, 12, 128, 128, "07ad2bcc4ebfcf3c"),
    (3, 129, 4, 2, 128, 100, "95ff437e6214f13c"),
    (2, 97, 3, 3, 64, 40, "8e9fbd05ba0717da"),
    (8, 161, 12, 12, 128, 128, "7892252457c53b8f"),
    (40, 113, 12, 12, 64, 64, "9ab77d6fddf7b478"),
    (30, 97, 10, 2, 32, 33, "1679663e18146e59"),
])
def test_the_bits_that_prompts_have_had(monkeypatch, B, T, H, G, Dk, Dv, digest):
    q, k, v, b = (spread(i, B * T, n).bfloat16() for i, n in enumerate((G * Dk, G * Dk, H * Dv, H)))
    x, x0, state, rate = 3 * spread(4, B * T, H * Dk) - 2, spread(5, H * Dk) * 0.5, spread(6, B, H, Dk, Dv), 0.25 + 2 * spread(7, H).abs()
    monkeypatch.setattr(mo, "gated_norm", lambda o, *a, **kw: o)  # the rule alone, fp32
    out = mo.delta_rule(q, k, v, x, x0, rate, b, state, B, T, H, G, Dk, Dv, torch.zeros(B * T, H * Dv, dtype=torch.bfloat16, device="cuda"),
                        torch.ones(Dv, device="cuda"), 1e-6)
    assert ops.read_status("cuda") == 0
    assert hashlib.sha256(out.cpu().numpy().tobytes() + state.cpu().numpy().tobytes()).hexdigest()[:16] == digest
