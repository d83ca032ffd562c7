"""The recurrence at the edges of its chunks (32 tokens) and batches (4): against 64 bits, and the same bits however a prompt is cut."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 4, 31, 32, 33, 65])
@pytest.mark.parametrize("dim,vdim,channel", [(64, 64, True), (32, 24, True), (128, 128, False), (64, 128, False)])
def test_chunk_edges(T, dim, vdim, channel):
    gen = torch.Generator(device="cuda").manual_seed(T * dim + vdim)
    B, H = 2, 3
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k, v = rand(B, T, H * dim).bfloat16(), rand(B, T, H * dim).bfloat16(), rand(B, T, H * vdim).bfloat16()
    x, x0, u, start = rand(B, T, H * dim) - 2, rand(H * dim) * 0.1, rand(H * dim), rand(B, H, dim, vdim)
    decay = torch.tensor([0.9, 0.99, 0.999], device="cuda")

    def run(lo, hi, state):
        n = hi - lo
        part = lambda t: t[:, lo:hi].reshape(B * n, -1)
        extra = dict(decay_logits=part(x), decay_bias=x0, bonus=u) if channel else dict(decay=decay)
        return mo.recurrent(part(q), part(k), part(v), state, B, n, H, dim, vdim, **extra).view(B, n, H, vdim)

    whole = start.clone()
    out = run(0, T, whole)
    S, want = start.double(), []
    qd, kd, vd = (t.double().view(B, T, H, -1) for t in (q, k, v))
    for t in range(T):
        kv = kd[:, t, :, :, None] * vd[:, t, :, None]
        w = torch.exp(-torch.exp(x[:, t].double() + x0.double())).view(B, H, dim, 1) if channel else decay.double()[None, :, None, None]
        seen = S + u.double().view(H, dim, 1) * kv if channel else w * S + kv
        want.append(torch.einsum("bhde,bhd->bhe", seen, qd[:, t]))
        S = w * S + kv
    want = torch.stack(want, 1)
    # fp32 throughout; the fast exponentials of a decay err by a few of its last places, over T tokens
    tol = (T + 16) * 2.0 ** -22
    assert (out.double() - want).norm() <= tol * want.norm() and (whole.double() - S).norm() <= tol * S.norm()
    half = T // 2
    if half > 1 and T - half > 1:
        cut = start.clone()
        assert torch.equal(torch.cat([run(0, half, cut), run(half, T, cut)], 1), out) and torch.equal(cut, whole)
