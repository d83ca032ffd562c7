"""The append's launch for many head rows (four per half-warp) in every form of its inputs and caches, against the one for few, bit for bit."""
import pytest
import torch

from nanochat_b200 import ops
from nanochat_b200.gpt import precompute_rotary_embeddings

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def rand(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV, BF)


def ints(*values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def caches(*shape):
    return [torch.zeros(*shape, 128, dtype=BF, device=DEV) for _ in range(2)]


def pieces(T, size=250):
    return [slice(t, min(t + size, T)) for t in range(0, T, size)]


B, T, H, G, CAP = 3, 700, 12, 4, 800  # 42000 head rows, of which a piece of 250 tokens and 3 rows has 15000


@pytest.fixture
def qkv():
    x = rand(B, T, (H + 2 * G) * 128, seed=1)
    return [z.unflatten(2, (-1, 128)) for z in x.split([H * 128, G * 128, G * 128], 2)]


@pytest.fixture
def tables():
    return precompute_rotary_embeddings(1024, 128, device=DEV)


def test_column_slices(qkv, tables):
    assert not qkv[0].is_contiguous() and ops._token_stride(qkv[0]) == (H + 2 * G) * 128
    lens, wide, few = ints(0, 33, 71), caches(B, CAP, G), caches(B, CAP, G)
    got = ops.append_rope_norm(*qkv, *wide, lens, *tables)
    for part in pieces(T):
        want = ops.append_rope_norm(*(t[:, part] for t in qkv), *few, lens + part.start, *tables)
        assert torch.equal(got[:, part], want)
    assert all(torch.equal(a, b) for a, b in zip(wide, few)) and ops.read_status(DEV) == 0


def test_write_slots(qkv, tables):
    lens, slots, wide, few = ints(5, 200, 300), ints(100, -1, 7), caches(B, CAP, G), caches(B, CAP, G)
    got = ops.append_rope_norm(*qkv, *wide, lens, *tables, write_slots=slots)
    for part in pieces(T):
        at = torch.where(slots < 0, slots, slots + part.start)
        want = ops.append_rope_norm(*(t[:, part] for t in qkv), *few, lens + part.start, *tables, write_slots=at)
        assert torch.equal(got[:, part], want)
    assert all(torch.equal(a, b) and not a[1].any() and a[0].any() for a, b in zip(wide, few)) and ops.read_status(DEV) == 0


def test_pages(qkv, tables):
    tokens = ops.PAGE_TILE * 2
    per = -(-CAP // tokens)
    table = torch.randperm(B * per, generator=torch.Generator().manual_seed(2)).view(B, per).to(DEV, torch.int32)
    lens, wide, few = ints(0, 33, 71), caches(B * per, tokens, G), caches(B * per, tokens, G)
    args = [t.contiguous() for t in qkv]
    got = ops.append_rope_norm_paged(*args, *wide, table, lens, *tables)
    for part in pieces(T):
        want = ops.append_rope_norm_paged(*(t[:, part] for t in args), *few, table, lens + part.start, *tables)
        assert torch.equal(got[:, part], want)
    assert all(torch.equal(a, b) for a, b in zip(wide, few)) and ops.read_status(DEV) == 0
    table[1, 1] = B * per  # a page outside the pool: its tokens are left out, the others written
    outside = caches(B * per, tokens, G)
    ops.append_rope_norm_paged(*args, *outside, table, lens, *tables)
    assert ops.read_status(DEV) == 8
    kept = torch.ones(B * per, dtype=torch.bool, device=DEV)
    kept[[p for p in range(B * per) if not (table == p).any()]] = False
    for a, b in zip(outside, wide):
        assert torch.equal(a[kept], b[kept]) and not a[~kept].any()


def test_split(tables):
    rows, heads = 2100, 12
    q, k, v = rand(rows, 1, heads, 128, seed=3), rand(rows, 1, 2, 128, seed=4), rand(rows, 1, 2, 128, seed=5)
    lens = torch.arange(rows, dtype=torch.int32, device=DEV) % 30
    for rank in (0, 1):
        wide, few = caches(rows, 32, 2), caches(rows, 32, 2)
        got = ops.append_rope_norm(q, k, v, *wide, lens, *tables, split=(2, rank, 4))
        for part in pieces(rows, 700):
            want = ops.append_rope_norm(q[part], k[part], v[part], *(c[part] for c in few), lens[part], *tables, split=(2, rank, 4))
            assert torch.equal(got[part], want)
        assert all(torch.equal(a, b) and a.any() for a, b in zip(wide, few)) and ops.read_status(DEV) == 0


def test_rows_that_do_not_fit(qkv, tables):
    """A row past the capacity, or of a negative length, is left out whole and reported; the others are written."""
    lens, wide, few = ints(0, CAP - T + 1, 71), caches(B, CAP, G), caches(B, CAP, G)
    got = ops.append_rope_norm(*qkv, *wide, lens, *tables)
    assert ops.read_status(DEV) == 1
    lens[1] = -2
    again = caches(B, CAP, G)
    ops.append_rope_norm(*qkv, *again, lens, *tables)
    assert ops.read_status(DEV) == 4
    lens[1] = 0
    want = ops.append_rope_norm(*qkv, *few, lens, *tables)
    for c in (*wide, *again):
        assert not c[1].any()
    for a, b, c in zip(wide, again, few):
        assert all(torch.equal(x[r], c[r]) for x in (a, b) for r in (0, 2))
    assert all(torch.equal(got[r], want[r]) for r in (0, 2))
