"""The experts' products on pairs of CTAs (csrc/experts_pair.cu): ragged sizes, experts with none, one and a tile's edge of the positions, the bits of
the other form, and which calls take it."""
import pytest
import torch

from nanochat_b200 import _lib
from nanochat_b200 import mixer_ops as mo
from nanochat_b200 import ops

pytestmark = pytest.mark.gpu


def routed(counts, seed=0):
    """Logits under which expert e gets counts[e] tokens, one each, at random places."""
    rows, E = sum(counts), len(counts)
    gen = torch.Generator().manual_seed(seed)
    place = torch.randperm(rows, generator=gen)
    z = torch.randn(rows, E, generator=gen).clamp(-2, 2)
    z[place, torch.repeat_interleave(torch.arange(E), torch.tensor(counts))] = 4.0
    r = mo.Routing(z.cuda(), 1)
    assert (r.offsets[1:] - r.offsets[:-1]).tolist() == list(counts)
    return r


def general(a, w, r, up, N):
    """The same call without scratch, whose up product takes the other form; the down product in 64 bits, rounded."""
    E, _, K = w.shape
    if up:
        out = torch.empty(r.pairs, N, dtype=a.dtype, device="cuda")
        _lib.call("nckv_experts", *(t.data_ptr() for t in (a, w, out, r.offsets, r.slot, r.scale)), 1, r.pairs, E, r.top, N, K, 0,
                  ops.workspace(a.device, 1, 1, 1).data_ptr(), torch.cuda.current_stream().cuda_stream)
        return out
    out, at = torch.empty(r.pairs, N, dtype=torch.float64, device="cuda"), r.offsets.tolist()
    for e in range(E):
        out[r.slot[at[e]:at[e + 1]].long()] = a[at[e]:at[e + 1]].double() @ w[e].double().t()
    return out.view(-1, r.top, N)


@pytest.mark.parametrize("counts,W,ff", [
    ((0, 1, 255, 256, 257, 1024, 2500, 900), 648, 1288),    # neither channels nor widths fill their tiles
    ((2600, 2600, 0, 511, 513, 127, 128, 129), 1000, 1032),
    ((7000,), 328, 1032),
    ((640,) * 12, 1536, 1024),
])
def test_the_bits_of_the_other_form(counts, W, ff):
    r = routed(counts)
    gen = torch.Generator(device="cuda").manual_seed(W)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    E, rows = len(counts), sum(counts)
    h, w_in, w_down = rand(rows, W).bfloat16(), (rand(E, 2 * ff, W) * W ** -0.5).bfloat16(), (rand(E, W, ff) * ff ** -0.5).bfloat16()
    assert _lib.lib.nckv_experts_workspace_bytes(1, r.pairs, E, ff, W, 0) == 2 * r.pairs * W  # takes it
    act = mo.expert_product(h, w_in, r, True)
    assert torch.equal(act, general(h, w_in, r, True, ff))
    y, want = mo.expert_product(act, w_down, r, False), general(act, w_down, r, False, W)
    # fp32 sums of ff exact products, rounded to bf16
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + (ff + 1) * 2.0 ** -24 * ff ** 0.5 * act.double().abs().max()).all()
    assert ops.read_status("cuda") == 0


def test_few_positions_take_the_other_form():
    for R, E, N, K in ((256, 16, 1024, 1536), (1024, 16, 1024, 1536), (6000, 16, 1024, 1536), (40000, 300, 1024, 1536), (24028, 16, 1024, 1532)):
        assert _lib.lib.nckv_experts_workspace_bytes(1, R, E, N, K, 0) == 0
    assert _lib.lib.nckv_experts_workspace_bytes(0, 24028, 16, 1536, 1024, 0) == 0 == _lib.lib.nckv_experts_workspace_bytes(1, 24028, 16, 1024, 1536, 1)


def test_without_room_for_the_sorted_copy_the_other_form_answers(monkeypatch):
    r = routed((640,) * 12)
    gen = torch.Generator(device="cuda").manual_seed(3)
    h, w = torch.randn(640 * 12, 1536, generator=gen, device="cuda").bfloat16(), torch.randn(12, 2048, 1536, generator=gen, device="cuda").bfloat16()
    want, empty, need, refused = mo.expert_product(h, w, r, True), torch.empty, 2 * r.pairs * 1536, []

    def short(*size, **kw):
        if size == (need,) and kw.get("dtype") == torch.uint8:
            refused.append(size)
            raise torch.OutOfMemoryError("planted")
        return empty(*size, **kw)

    monkeypatch.setattr(torch, "empty", short)
    got = mo.expert_product(h, w, r, True)
    assert refused and torch.equal(got, want) and ops.read_status("cuda") == 0
