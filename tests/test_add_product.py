"""Sums of two products: a result beside the first one, or in its place where the caller says so and no gradient is wanted."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo


def operands():
    gen = torch.Generator().manual_seed(1)
    return [torch.randn(*s, generator=gen) for s in ((5, 7), (5, 3), (7, 3))]


def test_the_first_one_stays():
    y, a, w = operands()
    kept = y.clone()
    got = mo.add_product(y, a, w, 0.5, 2.0)
    assert torch.equal(y, kept) and got is not y
    torch.testing.assert_close(got, 0.5 * kept + 2.0 * (a @ w.t()))


def test_in_its_place():
    y, a, w = operands()
    want = mo.add_product(y, a, w, 0.5, 2.0)
    assert mo.add_product_(y, a, w, 0.5, 2.0) is y and torch.equal(y, want)


@pytest.mark.parametrize("call", [mo.add_product, mo.add_product_])
@pytest.mark.parametrize("of", range(3))
def test_gradients(call, of):
    ts = operands()
    ts[of].requires_grad_()
    want = 0.5 * ts[0] + 2.0 * (ts[1] @ ts[2].t())
    got = call(*ts, 0.5, 2.0)
    torch.testing.assert_close(got, want)
    torch.testing.assert_close(*(torch.autograd.grad(z.square().sum(), ts[of])[0] for z in (got, want)))


@pytest.mark.gpu
def test_bf16_operands_give_the_same_bits():
    y, a, w = (t.cuda() for t in operands())
    a, w = (torch.nn.functional.pad(t, (0, 5)).bfloat16() for t in (a, w))
    kept, want = y.clone(), mo.add_product(y, a, w)
    assert torch.equal(y, kept) and torch.equal(mo.add_product_(y, a, w), want) and torch.equal(y, want)
