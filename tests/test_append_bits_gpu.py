"""The appends for whole heads of 128 channels give the bits of the general kernels, which a table off the 16-byte grid selects."""
import pytest
import torch

from nanochat_b200 import mixer_ops as mo
from nanochat_b200 import ops
from nanochat_b200.mixers import rotary_table

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def rows_of(n, H, G):
    """Values from 2^-9 to 2^9 of their like, so that the order of a sum shows in its last bits."""
    gen = torch.Generator().manual_seed(n + H)
    x = torch.randn(n, (H + 2 * G) * 128, generator=gen) * torch.exp2(torch.randint(-9, 10, (n, (H + 2 * G) * 128), generator=gen).float())
    return x.to(DEV, BF)


def tables(cap):
    on = rotary_table(cap, 128, 5000.0, None, DEV)
    off = torch.empty(on.numel() + 1, device=DEV)[1:].view(on.shape)
    off.copy_(on)
    assert on.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 4
    return on, off


def slices(x, H, G):
    return x[:, :H * 128], x[:, H * 128:(H + G) * 128], x[:, (H + G) * 128:]


@pytest.mark.parametrize("B,T,H,G", [(2, 3, 1, 1), (7, 1, 12, 12), (1, 1638, 12, 4), (3, 700, 12, 4), (1, 2001, 6, 6), (1, 5000, 16, 4)])
def test_rope_unit(B, T, H, G):
    cap, lens, x, out = T + 64, torch.arange(B, dtype=torch.int32, device=DEV) * 7, rows_of(B * T, H, G), []
    for table in tables(cap):
        kc, vc = (torch.zeros(B, cap, G, 128, dtype=BF, device=DEV) for _ in range(2))
        out.append((mo.rope_unit_append(*slices(x, H, G), table, 128, kc, vc, lens, B, T, H, G, 128, 128, 0.7, 1e-5), kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*out)) and ops.read_status(DEV) == 0


# two to eight pieces per thread, and more heads than that
@pytest.mark.parametrize("B,T,H,G", [(2, 3, 4, 4), (5, 1, 16, 4), (1, 37, 16, 16), (2, 9, 24, 12), (1, 5, 64, 2), (3, 11, 8, 1), (2, 7, 32, 16),
                                     (1, 3001, 24, 6), (1, 3, 48, 8)])
@pytest.mark.parametrize("own", [True, False])
def test_rms_rope(B, T, H, G, own):
    cap, lens, x, out = T + 64, torch.arange(B, dtype=torch.int32, device=DEV) * 7, rows_of(B * T, H, G), []
    gen = torch.Generator().manual_seed(4)
    wq, wk = (1 + 0.1 * torch.randn(n * 128, generator=gen).to(DEV) for n in (H, G))
    for table in tables(cap):
        kc, vc = (torch.zeros(B, cap, G, 128, dtype=BF, device=DEV) for _ in range(2))
        q, k, v = slices(x, H, G)
        out.append((mo.rms_rope_append(q, k if own else None, v if own else None, wq, wk if own else None, table, 128, kc, vc, lens, B, T,
                                       H, G, 128, 128, 0.7, 1e-5), kc, vc))
    assert all(torch.equal(a, b) for a, b in zip(*out)) and bool(out[0][1].any()) == own and ops.read_status(DEV) == 0
