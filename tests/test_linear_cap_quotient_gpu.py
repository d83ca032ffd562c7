"""The cap inside the product divides as the pass behind it does: the same bits where the sums are exact."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [30.0, 15.0, 29.999998, 0.1, 1e4, 2.0 ** -60, 2.0 ** -70, 2.0 ** 60, 2.0 ** 70])
def test_the_bits_of_the_division(cap):
    gen = torch.Generator(device="cuda").manual_seed(1)
    n = 1 << 20
    v = torch.randn(n, generator=gen, device="cuda") * torch.exp2(torch.randint(-30, 5, (n,), generator=gen, device="cuda").float()) * min(cap, 2.0 ** 60)
    v[:4] = torch.tensor([0.0, 16 * cap, -20 * cap, 9.01 * cap], device="cuda")
    # three bf16 pieces that add up to v without rounding, whatever their order
    a = torch.zeros(n, 8, dtype=torch.bfloat16, device="cuda")
    for i in range(3):
        a[:, i] = v.bfloat16()
        v = v - a[:, i].float()
    w = torch.zeros(2, 8, dtype=torch.bfloat16, device="cuda")
    w[:, :3] = 1
    with mo.full_precision_sums():
        assert torch.equal(mo.linear_cap(a, w, cap), mo.softcap(mo.product(a, w, f32_out=True), cap))
