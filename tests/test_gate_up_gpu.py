"""The feed-forward's gate and up product with its activation in one launch (csrc/experts_pair.cu): edges of its tiles and of its rule."""
import pytest
import torch

from nanochat_b200 import _lib
from nanochat_b200 import mixer_ops as mo
from nanochat_b200 import ops

pytestmark = pytest.mark.gpu


def wanted(h, w):
    g, u = (h.double() @ w.double().t()).chunk(2, 1)
    return torch.nn.functional.silu(g) * u, g.abs() + u.abs()


@pytest.mark.parametrize("rows,N,K", [(1024, 2048, 64), (1025, 2056, 72), (1279, 4000, 200), (1281, 1801, 1000), (2600, 1024, 8192), (1024, 2049, 8),
                                      (9000, 257, 1536), (70000, 31, 40)])
def test_against_64_bits(rows, N, K):
    gen = torch.Generator(device="cuda").manual_seed(rows + N)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    h, w = rand(rows, K).bfloat16(), (rand(2 * N, K) * K ** -0.5).bfloat16()
    assert rows >= mo.GATE_UP_ROWS and rows * N >= mo.GATE_UP_VALUES
    got, (want, scale) = mo.gate_up_product(h, w), wanted(h, w)
    # one rounding to the 8 bits of bf16 (at most 2^-8 of the value), fp32 sums of up to 8192 terms of about K^-1/2 and the activation
    assert ((got.double() - want).abs() <= want.abs() / 256 + 1e-5 * scale * (1 + scale)).all()
    assert ops.read_status("cuda") == 0


@pytest.mark.parametrize("rows,N,K", [(1023, 4096, 64), (1024, 2047, 64), (3, 64, 64), (1100, 2048, 63), (1537, 1376, 4096), (1100, 2048, 2048)])
def test_the_rest_takes_two_launches(rows, N, K):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    h, w = rand(rows, K).bfloat16(), (rand(2 * N, K) * K ** -0.5).bfloat16()
    assert torch.equal(mo.gate_up(h, w), mo.silu_mul(mo.product(h, w)))


def test_the_largest_take_one():
    h, w = torch.randn(2048, 1536, device="cuda").bfloat16(), (torch.randn(8192, 1536, device="cuda") / 40).bfloat16()
    got = mo.gate_up(h, w)
    assert torch.equal(got, mo.gate_up_product(h, w)) and not torch.equal(got, mo.silu_mul(mo.product(h, w)))


def test_rows_that_are_not_packed_and_other_types():
    h, w = torch.randn(1024, 128, device="cuda").bfloat16()[:, :64], torch.randn(4096, 64, device="cuda").bfloat16()
    assert torch.equal(mo.gate_up(h, w), mo.silu_mul(mo.product(h, w)))
    h = torch.randn(1024 * 64 + 4, device="cuda").bfloat16()[4:].view(1024, 64)  # 8-byte aligned
    assert torch.equal(mo.gate_up(h, w), mo.silu_mul(mo.product(h, w)))
    h, w = torch.randn(1024, 64, device="cuda"), torch.randn(4096, 64, device="cuda")
    assert torch.equal(mo.gate_up(h, w), mo.silu_mul(mo.product(h, w)))


def test_so_many_weight_rows_that_a_group_of_tiles_had_no_number():
    """A group is 65536 / K tiles of positions by all tiles of weights, 2^13 x 2^19 here; few positions leave it at their own tiles."""
    rows, N, K = 3, 1 << 26, 8
    gen = torch.Generator(device="cuda").manual_seed(9)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda", dtype=torch.bfloat16)
    h, w, out = rand(rows, K), rand(2 * N, K), torch.zeros(rows, N, dtype=torch.bfloat16, device="cuda")
    _lib.call("nckv_gate_up", h.data_ptr(), w.data_ptr(), out.data_ptr(), rows, N, K, ops.workspace(h.device, 1, 1, 1).data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    assert ops.read_status("cuda") == 0
    for at in range(0, N, 1 << 23):
        part = slice(at, at + (1 << 23))
        want, scale = wanted(h, torch.cat([w[:N][part], w[N:][part]]))
        assert ((out[:, part].double() - want).abs() <= want.abs() / 256 + 1e-5 * scale * (1 + scale)).all()
