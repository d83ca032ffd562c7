"""The appends' launches for many head rows against the ones for few, and against the general kernels."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo
from nanochat_b200 import ops
from nanochat_b200.gpt import precompute_rotary_embeddings
from nanochat_b200.mixers import rotary_table

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def rand(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV, BF)


# rows just below and above the line between the two launches (32768), head counts that 4 does and does not divide
@pytest.mark.parametrize("B,T,H,G", [(1, 1638, 12, 4), (3, 700, 12, 4), (2, 6554, 1, 1), (1, 2001, 6, 6), (5, 1170, 3, 1)])
def test_many_rows_append_as_few_do(B, T, H, G):
    cap, lens = T + 64, torch.arange(B, dtype=torch.int32, device=DEV) * 7
    q, k, v = rand(B, T, H, 128, seed=1), rand(B, T, G, 128, seed=2), rand(B, T, G, 128, seed=3)
    cos, sin = precompute_rotary_embeddings(cap, 128, device=DEV)
    caches = [tuple(torch.zeros(B, cap, G, 128, dtype=BF, device=DEV) for _ in range(2)) for _ in range(2)]
    got = ops.append_rope_norm(q, k, v, *caches[0], lens, cos, sin)
    want, at = torch.empty_like(got), lens.clone()
    for t in range(0, T, 250):  # bit for bit, whatever the launch
        part = slice(t, min(t + 250, T))
        want[:, part] = ops.append_rope_norm(q[:, part], k[:, part], v[:, part], *caches[1], at, cos, sin)
        at += part.stop - part.start
    assert torch.equal(got, want) and all(torch.equal(a, b) for a, b in zip(*caches))
    assert ops.read_status(DEV) == 0


def slices(x, H, G):
    return x[:, :H * 128], x[:, H * 128:(H + G) * 128], x[:, (H + G) * 128:(H + 2 * G) * 128]


@pytest.mark.parametrize("B,T,H,G", [(2, 3, 1, 1), (7, 1, 12, 12), (1, 1638, 12, 4), (3, 700, 12, 4), (1, 2001, 6, 6)])
def test_whole_head_rope_unit(B, T, H, G):
    """Rows of an odd stride take the general kernel; sums of squares in another order move fp32 results by less than
    2^-18, so a bf16 value may land on the neighbour (2^-8 of it) and no further."""
    cap, lens = T + 64, torch.arange(B, dtype=torch.int32, device=DEV) * 7
    x = rand(B * T, (H + 2 * G) * 128 + 4)
    odd = torch.empty(B * T, x.size(1) + 1, dtype=BF, device=DEV)[:, :x.size(1)]
    odd.copy_(x)
    table, out = rotary_table(cap, 128, 5000.0, None, DEV), []
    for rows in (x, odd):
        kc, vc = (torch.zeros(B, cap, G, 128, dtype=BF, device=DEV) for _ in range(2))
        out.append((mo.rope_unit_append(*slices(rows, H, G), table, 128, kc, vc, lens, B, T, H, G, 128, 128, 0.7, 1e-5), kc, vc))
    assert torch.equal(out[0][2], out[1][2])
    for a, b in zip(out[0][:2], out[1][:2]):
        torch.testing.assert_close(a.float(), b.float(), rtol=2 ** -7, atol=1e-5)


# one to four pieces per thread, and more heads than that
@pytest.mark.parametrize("B,T,H,G", [(2, 3, 4, 4), (5, 1, 16, 4), (1, 37, 16, 16), (2, 9, 24, 12), (1, 5, 64, 2)])
@pytest.mark.parametrize("own", [True, False])
def test_whole_head_rms_rope(B, T, H, G, own):
    """As above, for the norm over the whole projection (fp32 sums in another order, within 2^-18)."""
    cap, lens = T + 64, torch.arange(B, dtype=torch.int32, device=DEV) * 7
    x = rand(B * T, (H + 2 * G) * 128 + 4)
    odd = torch.empty(B * T, x.size(1) + 1, dtype=BF, device=DEV)[:, :x.size(1)]
    odd.copy_(x)
    wq, wk = 1 + 0.1 * rand(H * 128, seed=4).float(), 1 + 0.1 * rand(G * 128, seed=5).float()
    table, out = rotary_table(cap, 128, 5000.0, None, DEV), []
    for rows in (x, odd):
        kc, vc = (torch.zeros(B, cap, G, 128, dtype=BF, device=DEV) for _ in range(2))
        q, k, v = slices(rows, H, G)
        out.append((mo.rms_rope_append(q, k if own else None, v if own else None, wq, wk if own else None, table, 128, kc, vc, lens, B, T,
                                       H, G, 128, 128, 0.7, 1e-5), kc, vc))
    assert torch.equal(out[0][2], out[1][2]) and bool(out[0][1].any()) == own
    for a, b in zip(out[0][:2], out[1][:2]):
        torch.testing.assert_close(a.float(), b.float(), rtol=2 ** -7, atol=1e-5)
