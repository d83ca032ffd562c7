"""A decode step of few rows in one launch (csrc/decode_small.cu): lengths around its groups of 16 keys, windows, group sizes, pages, slices of a
projection, garbage behind the length, rows that overflow."""
import pytest
import torch

from nanochat_b200 import _lib, ops
from nanochat_b200.engine import KVCache, PagedKVCache
from nanochat_b200.gpt import kv_attention, precompute_rotary_embeddings

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def attend(q, k, v, left):
    """In 64 bits: q (H, D) over keys (n, G, D), the newest last."""
    n, G = k.shape[:2]
    lo = max(0, n - 1 - left) if left >= 0 else 0
    k, v = (t[lo:].double().repeat_interleave(q.size(0) // G, 1) for t in (k, v))
    p = torch.softmax(torch.einsum("hd,nhd->hn", q.double(), k) * 128 ** -0.5, 1)
    return torch.einsum("hn,nhd->hd", p, v)


@pytest.mark.parametrize("H,G", [(2, 2), (6, 1), (12, 6), (8, 1), (16, 1), (9, 1), (16, 4)])
@pytest.mark.parametrize("cap,window", [(100, -1), (1024, -1), (512, 40), (512, 0), (5000, 300)])
def test_lengths_and_windows(H, G, cap, window):
    lens = [n for n in (0, 1, 15, 16, 17, 63, 99, 511, 1000, 4999) if n < cap]
    while len(lens) * G > 18 * (1 if cap > 512 else 2):
        lens.pop(len(lens) // 2)
    B = len(lens)
    if not _lib.lib.nckv_decode_small_fits(B, H, G, cap, window):
        pytest.skip("takes the other kernels")
    gen = torch.Generator(device="cuda").manual_seed(cap + H)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(BF)
    cos, sin = precompute_rotary_embeddings(cap, 128, device="cuda")
    kc, vc = (torch.full((B, cap, G, 128), float("nan"), dtype=BF, device="cuda") for _ in range(2))  # nothing behind a length is looked at
    for b, n in enumerate(lens):
        kc[b, :n], vc[b, :n] = rand(n, G, 128), rand(n, G, 128)
    seqlens = torch.tensor(lens, dtype=torch.int32, device="cuda")
    x = rand(B, 1, (H + 2 * G) * 128)
    q, k, v = (z.view(B, 1, -1, 128) for z in x.split([H * 128, G * 128, G * 128], 2))  # columns of one projection
    k2, v2 = kc.clone(), vc.clone()
    rotated = ops.append_rope_norm(q, k, v, k2, v2, seqlens, cos, sin)[:, 0]
    y = ops.append_and_attend_small(q, k, v, kc, vc, None, seqlens, cos, sin, window)[:, 0]
    bits = lambda t: t.view(torch.int16)
    assert torch.equal(bits(kc), bits(k2)) and torch.equal(bits(vc), bits(v2)) and ops.read_status("cuda") == 0
    for b, n in enumerate(lens):
        want = attend(rotated[b], kc[b, :n + 1], vc[b, :n + 1], window)
        # weights and outputs in bf16
        assert (y[b].double() - want).abs().max() <= 1e-2 * want.abs().max().clamp(min=0.1)


def test_pages_give_the_bits_of_dense_rows():
    B, H, G, cap, pt = 3, 8, 2, 480, 96
    cos, sin = precompute_rotary_embeddings(cap, 128, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(2)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(BF)
    dense, paged = KVCache(B, G, cap, 128, 2, "cuda", BF), PagedKVCache(B, G, cap, 128, 2, "cuda", BF, page_tokens=pt)
    paged.reserve(cap)
    dense.k_cache.copy_(rand(*dense.k_cache.shape))
    dense.v_cache.copy_(rand(*dense.v_cache.shape))
    for b in range(B):
        for i, page in enumerate(paged.block_table[b].tolist()):
            paged.k_cache[:, page], paged.v_cache[:, page] = dense.k_cache[:, b, i * pt:(i + 1) * pt], dense.v_cache[:, b, i * pt:(i + 1) * pt]
    for lens in ([0, 95, 96], [97, 200, 479]):
        for window in (-1, 70):
            q, k, v = rand(B, 1, H, 128), rand(B, 1, G, 128), rand(B, 1, G, 128)
            out = []
            for cache in (dense, paged):
                cache.cache_seqlens.copy_(torch.tensor(lens))
                out.append(kv_attention(q, k, v, (cos, sin), (window, 0), cache, 0))
            assert torch.equal(*out)
    assert ops.read_status("cuda") == 0


def test_rows_that_do_not_fit_are_flagged_and_leave_the_cache():
    B, H, G, cap = 4, 2, 2, 64
    cos, sin = precompute_rotary_embeddings(cap, 128, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(BF)
    kc, vc, q, k, v = rand(B, cap, G, 128), rand(B, cap, G, 128), rand(B, 1, H, 128), rand(B, 1, G, 128), rand(B, 1, G, 128)
    good = torch.tensor([5, 5, 5, 5], dtype=torch.int32, device="cuda")
    want = ops.append_and_attend_small(q, k, v, kc.clone(), vc.clone(), None, good, cos, sin, -1)
    k2, v2 = kc.clone(), vc.clone()
    y = ops.append_and_attend_small(q, k, v, k2, v2, None, torch.tensor([5, cap, -3, 5], dtype=torch.int32, device="cuda"), cos, sin, -1)
    assert ops.read_status("cuda") == _lib.ST_OVERFLOW | _lib.ST_BAD_SEQLEN
    assert torch.equal(y[[0, 3]], want[[0, 3]]) and not y[1:3].any()
    assert torch.equal(k2[1:3], kc[1:3]) and torch.equal(v2[1:3], vc[1:3])


@pytest.mark.parametrize("B,H,G,cap,window,last", [(1, 2, 2, 3072, -1, True), (1, 2, 2, 65536, 3071, True), (36, 2, 1, 512, -1, False),
                                                    (140, 1, 1, 384, -1, True), (140, 16, 1, 256, -1, True), (1, 16, 1, 1024, -1, True)])
def test_the_longest_caches_it_takes(B, H, G, cap, window, last):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("another device")
    fits = _lib.lib.nckv_decode_small_fits
    assert fits(B, H, G, cap, window) and not (last and fits(B, H, G, cap + 1, window + 1 if window >= 0 else -1))
    assert not fits(149, 1, 1, 16, -1) and not fits(2, 34, 2, 64, -1) and not fits(0, 1, 1, 16, -1)
    gen = torch.Generator(device="cuda").manual_seed(B)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(BF)
    cos, sin = precompute_rotary_embeddings(cap, 128, device="cuda")
    kc, vc, q, k, v = rand(B, cap, G, 128), rand(B, cap, G, 128), rand(B, 1, H, 128), rand(B, 1, G, 128), rand(B, 1, G, 128)
    seqlens = torch.full((B,), cap - 1, dtype=torch.int32, device="cuda")
    k2, v2 = kc.clone(), vc.clone()
    rotated = ops.append_rope_norm(q, k, v, k2, v2, seqlens, cos, sin)[:, 0]
    y = ops.append_and_attend_small(q, k, v, kc, vc, None, seqlens, cos, sin, window)[:, 0]
    assert torch.equal(kc, k2) and torch.equal(vc, v2) and ops.read_status("cuda") == 0
    for b in (0, B - 1):
        want = attend(rotated[b], kc[b], vc[b], window)
        assert (y[b].double() - want).abs().max() <= 1e-2 * want.abs().max()


def test_scores_of_minus_infinity_have_no_weight():
    B, H, G, cap, n = 1, 2, 2, 64, 40
    cos, sin = precompute_rotary_embeddings(cap, 128, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(BF)
    kc, vc, q, k, v = rand(B, cap, G, 128), rand(B, cap, G, 128), rand(B, 1, H, 128), rand(B, 1, G, 128), rand(B, 1, G, 128)
    seqlens = torch.tensor([n], dtype=torch.int32, device="cuda")
    rotated = ops.append_rope_norm(q, k, v, kc.clone(), vc.clone(), seqlens, cos, sin)[0, 0]
    kc[0, :32] = 0
    for h in range(G):  # the first two groups of keys: -inf against the first channel of q
        kc[0, :32, h, 0] = -float("inf") * rotated[h, 0].sign().float()
    y = ops.append_and_attend_small(q, k, v, kc, vc, None, seqlens, cos, sin, -1)[0, 0]
    want = attend(rotated, kc[0, 32:n + 1], vc[0, 32:n + 1], -1)
    assert (y.double() - want).abs().max() <= 1e-2 * want.abs().max()


def test_steps_and_a_chunk_in_turn_on_the_same_rows():
    """What a step leaves in the cache is what the next call, of whichever kernels, reads: beside a cache too long for the one launch."""
    B, H, G, short, long = 3, 6, 2, 512, 16384
    assert _lib.lib.nckv_decode_small_fits(B, H, G, short, -1) and not _lib.lib.nckv_decode_small_fits(B, H, G, long, -1)
    cos, sin = precompute_rotary_embeddings(long, 128, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(6)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(BF)
    caches = [KVCache(B, G, n, 128, 1, "cuda", BF) for n in (short, long)]
    k0, v0 = rand(1, B, 200, G, 128), rand(1, B, 200, G, 128)
    for c in caches:
        c.k_cache[:, :, :200], c.v_cache[:, :, :200] = k0, v0
        c.cache_seqlens.copy_(torch.tensor([30, 111, 200]))
    for T in (1, 1, 1, 7, 1, 130, 1, 1):
        q, k, v = rand(B, T, H, 128), rand(B, T, G, 128), rand(B, T, G, 128)
        y, want = (kv_attention(q, k, v, (cos, sin), (-1, 0), c, 0) for c in caches)
        # weights and outputs in bf16
        assert (y.double() - want.double()).abs().max() <= 1e-2 * want.double().abs().max()
    n = caches[0].cache_seqlens.tolist()
    assert n == caches[1].cache_seqlens.tolist() == [30 + 143, 111 + 143, 200 + 143]
    for b in range(B):
        for a, c in zip((caches[0].k_cache, caches[0].v_cache), (caches[1].k_cache, caches[1].v_cache)):
            assert torch.equal(a[0, b, :n[b]].view(torch.int16), c[0, b, :n[b]].view(torch.int16))
    assert ops.read_status("cuda") == 0
