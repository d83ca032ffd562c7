"""The append's rotation in two-wide bf16 arithmetic: the bits of the eager operations for numbers of every size, and for what is no number."""
import pytest
import torch
import torch.nn.functional as F

from nanochat_b200 import ops

pytestmark = pytest.mark.gpu


def eager(x, cos, sin):
    a, b = x[..., :64], x[..., 64:]
    y = torch.cat([a * cos + b * sin, a * (-sin) + b * cos], -1)
    return F.rms_norm(y, (128,)) * 1.2


@pytest.mark.parametrize("kind", ["every bit pattern", "small", "apart"])
def test_the_bits_of_the_eager_operations(kind):
    gen = torch.Generator(device="cuda").manual_seed(5)
    B, T, H = 3, 211, 4
    bits = lambda *s: torch.randint(0, 1 << 16, s, generator=gen, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    cos, sin = rand(1, T, 1, 64).bfloat16(), rand(1, T, 1, 64).bfloat16()
    if kind == "every bit pattern":
        q, k = bits(B, T, H, 128), bits(B, T, H, 128)
        cos, sin = bits(1, T, 1, 64), bits(1, T, 1, 64)
    elif kind == "small":  # products that leave the normal numbers
        q, k = ((rand(B, T, H, 128) * 2.0 ** -66).bfloat16() for _ in range(2))
        cos, sin = (cos * 2.0 ** -66).bfloat16(), (sin * 2.0 ** -66).bfloat16()
    else:  # terms of very different size
        q, k = ((rand(B, T, H, 128) * torch.exp2(torch.randint(-20, 20, (B, T, H, 128), generator=gen, device="cuda").float())).bfloat16()
                for _ in range(2))
    v = rand(B, T, H, 128).bfloat16()
    kc, vc = (torch.zeros(B, T, H, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    got = ops.append_rope_norm(q, k, v, kc, vc, torch.zeros(B, dtype=torch.int32, device="cuda"), cos, sin)
    for have, x in ((got, q), (kc, k)):
        want = eager(x, cos, sin)
        assert torch.equal(have.isnan(), want.isnan())
        assert torch.equal(have.nan_to_num(0.0).view(torch.int16), want.nan_to_num(0.0).view(torch.int16))
    assert torch.equal(vc, v) and ops.read_status("cuda") == 0
