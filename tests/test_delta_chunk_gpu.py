"""The delta rule in chunks of 16 tokens: chunks' edges, widths that fill no group of columns, rows that allow no pairs, few heads (warps that share
columns) and many, against 64 bits."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo
from nanochat_b200 import ops

pytestmark = pytest.mark.gpu


def check(monkeypatch, B, T, H, G, Dk, Dv, shift=0):
    gen = torch.Generator(device="cuda").manual_seed(T * Dk + Dv)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k = rand(B * T, G * Dk).bfloat16(), rand(B * T, G * Dk).bfloat16()
    v = rand(B * T, H * Dv + 8).bfloat16()[:, shift:shift + H * Dv]
    x, x0, rate, b = rand(B * T, H * Dk) - 2, rand(H * Dk) * 0.3, torch.exp(rand(H) - 1), rand(B * T, H).bfloat16()
    start = rand(B, H, Dk, Dv)
    monkeypatch.setattr(mo, "gated_norm", lambda o, *a, **kw: o)  # the rule alone, fp32
    state = start.clone()
    out = mo.delta_rule(q, k, v, x, x0, rate, b, state, B, T, H, G, Dk, Dv, torch.zeros(B * T, H * Dv, dtype=torch.bfloat16, device="cuda"),
                        torch.ones(Dv, device="cuda"), 1e-6).double().view(B, T, H, Dv)
    unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
    group = torch.arange(H, device="cuda") // (H // G)
    qd, kd = (unit(z.double().view(B, T, G, Dk))[:, :, group] for z in (q, k))
    g = torch.exp(-rate.double()[:, None] * torch.nn.functional.softplus((x.double() + x0.double()).view(B, T, H, Dk)))
    beta, S, vd, want = torch.sigmoid(b.double()).view(B, T, H), start.double(), v.double().view(B, T, H, Dv), []
    for t in range(T):
        S = g[:, t, :, :, None] * S
        u = beta[:, t, :, None] * (vd[:, t] - torch.einsum("bhde,bhd->bhe", S, kd[:, t]))
        S = S + kd[:, t, :, :, None] * u[:, :, None]
        want.append(torch.einsum("bhde,bhd->bhe", S, qd[:, t]) * Dk ** -0.5)
    want = torch.stack(want, 1)
    # about 22 bits of every operand; the fast exponentials of a decay err by a few of its last places, over T tokens
    tol = (T + 32) * 2.0 ** -22
    assert ops.read_status("cuda") == 0
    assert (out - want).norm() <= tol * want.norm() and (state.double() - S).norm() <= tol * S.norm()


@pytest.mark.parametrize("T", [5, 15, 16, 17, 31, 33, 48, 49, 64, 65, 97])
@pytest.mark.parametrize("Dk,Dv", [(128, 128), (64, 40), (100, 17)])
def test_edges_of_chunks(monkeypatch, T, Dk, Dv):
    check(monkeypatch, 2, T, 3, 3, Dk, Dv)


# columns a warp takes alone: 16 at a time, few to many; and values at an odd place of a wider tensor
@pytest.mark.parametrize("B,H,G,Dk,Dv,shift", [(4, 10, 5, 128, 128, 0), (10, 12, 12, 128, 128, 0), (40, 12, 12, 64, 64, 0), (30, 10, 2, 32, 33, 0), (2, 3, 1, 128, 128, 1),
                                              (24, 16, 16, 128, 128, 1), (2, 2, 2, 64, 16, 2)])
def test_many_and_few_heads(monkeypatch, B, H, G, Dk, Dv, shift):
    check(monkeypatch, B, 50, H, G, Dk, Dv, shift)


# several rounds of the ring of three records, a ragged end: 7, 8 and 11 chunks; a warp to 16 columns at every padding of the channels, and shared ones
@pytest.mark.parametrize("T", [97, 113, 161])
@pytest.mark.parametrize("B,H,G,Dk,Dv", [(40, 16, 16, 128, 128), (40, 12, 12, 64, 64), (30, 10, 2, 32, 33), (2, 3, 3, 128, 128)])
def test_rounds_of_the_ring(monkeypatch, T, B, H, G, Dk, Dv):
    check(monkeypatch, B, T, H, G, Dk, Dv)


@pytest.mark.parametrize("T", [1000, 3001])
def test_long_prompts(monkeypatch, T):
    check(monkeypatch, 1, T, 4, 2, 128, 128)


def test_a_constant_decay_of_a_large_rate():
    """The same error of a decay, token after token: bounded by what the fast functions may err by, not by one rounding."""
    T, H, D = 2000, 3, 64
    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    k = torch.nn.functional.one_hot(torch.arange(T, device="cuda") % D, D).bfloat16().repeat(1, H)  # one channel a token
    v = (rand(T, H * D).abs() + 1).bfloat16()
    x, x0, rate = (rand(1, H * D) - 5).expand(T, -1).contiguous(), rand(H * D) * 0.3, torch.tensor([0.5, 3.0, 12.0], device="cuda")
    state, b = torch.zeros(1, H, D, D, device="cuda"), torch.zeros(T, H, device="cuda").bfloat16()
    mo.delta_rule(k, k, v, x, x0, rate, b, state, 1, T, H, H, D, D, torch.zeros(T, H * D, dtype=torch.bfloat16, device="cuda"), torch.ones(D, device="cuda"), 1e-6)
    g = rate.double()[:, None] * torch.nn.functional.softplus((x[0].double() + x0.double()).view(H, D))  # (H, D): -log of a token's decay
    unit = 1 / (1 + 1e-6) ** 0.5
    S = torch.zeros(H, D, D, dtype=torch.float64, device="cuda")
    seen = torch.zeros(D, dtype=torch.float64, device="cuda")
    for t in range(T):
        c = t % D  # the only channel that the token reads and writes; the others decay
        S *= torch.exp(-g)[:, :, None]
        S[:, c] += 0.5 * unit * (v[t].double().view(H, D) - unit * S[:, c])
    # per token: the argument by rate * (2^-21.4 of the logarithm + 2^-24 of its argument) + a rounding, the exponential by 3 + 1.2 |argument| of its
    # last places.  What is left of a write from D tokens ago carries D of these, with a half kept of the one before
    eps = rate.double()[:, None] * (2.0 ** -21.4 + 2.0 ** -24) + (4 + 2.4 * g) * 2.0 ** -24
    bound = 2 * D * eps + 64 * 2.0 ** -22
    assert ops.read_status("cuda") == 0
    assert ((state[0].double() - S).abs().amax(2) <= bound * S.abs().amax(2)).all()
