"""The recurrence's forms by key channels and decay, and the two of 32 channels with a decay per channel."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo
from tests.test_recurrent_chunks_gpu import test_chunk_edges as at_chunk_edges

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 33])
@pytest.mark.parametrize("dim,vdim,channel", [(128, 128, True), (96, 40, True), (100, 64, False), (256, 128, True), (256, 128, False), (200, 24, False)])
def test_forms(T, dim, vdim, channel):
    at_chunk_edges(T, dim, vdim, channel)


@pytest.mark.parametrize("T", [2, 5, 33])
@pytest.mark.parametrize("dim,vdim", [(32, 32), (24, 40), (64, 64)])
def test_many_rows_as_few(T, dim, vdim):
    """Enough rows for eight columns a lane (eight warps per SM; one batch of tokens where a lane has four key channels), against few at a time with four: the same bits."""
    gen = torch.Generator(device="cuda").manual_seed(T + vdim)
    B, H = 100, 24
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k, v = rand(B, T, H * dim).bfloat16(), rand(B, T, H * dim).bfloat16(), rand(B, T, H * vdim).bfloat16()
    x, x0, u, start = rand(B, T, H * dim) - 2, rand(H * dim) * 0.1, rand(H * dim), rand(B, H, dim, vdim)

    def run(lo, hi, state):
        part = lambda t: t[lo:hi].reshape((hi - lo) * T, -1)
        return mo.recurrent(part(q), part(k), part(v), state, hi - lo, T, H, dim, vdim, decay_logits=part(x), decay_bias=x0, bonus=u)
    many, few = start.clone(), start.clone()
    got = run(0, B, many)
    want = torch.cat([run(lo, lo + 20, few[lo:lo + 20]) for lo in range(0, B, 20)])
    assert torch.equal(got, want) and torch.equal(many, few)
