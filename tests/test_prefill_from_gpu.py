"""KVCache.prefill with the lengths read on the device (csrc/prefill_broadcast.cu): every length, and what it refuses leaves the cache as it was."""
import pytest
import torch

from nanochat_b200 import ops
from nanochat_b200.engine import KVCache

pytestmark = pytest.mark.gpu


def caches(T_src, T_dst, rows=3, layers=2, heads=2, dtype=torch.bfloat16):
    src, dst = KVCache(1, heads, T_src, 128, layers, "cuda", dtype), KVCache(rows, heads, T_dst, 128, layers, "cuda", dtype)
    for t in (src.k_cache, src.v_cache, dst.k_cache, dst.v_cache):
        t.copy_(torch.randn(t.shape, device="cuda"))
    return src, dst


@pytest.mark.parametrize("p,T_src,T_dst", [(0, 8, 8), (1, 8, 9), (7, 8, 64), (8, 8, 8), (513, 700, 701), (5, 70000, 70000)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_row_gets_the_prompt_and_nothing_else(p, T_src, T_dst, dtype):
    src, dst = caches(T_src, T_dst, dtype=dtype)
    src.cache_seqlens.fill_(p)
    want = [t.clone() for t in (dst.k_cache, dst.v_cache)]
    for w, s in zip(want, (src.k_cache, src.v_cache)):
        w[:, :, :p] = s[:, :, :p]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        dst.prefill(src)
    stream.synchronize()
    assert torch.equal(dst.k_cache, want[0]) and torch.equal(dst.v_cache, want[1]) and dst.cache_seqlens.tolist() == [p] * 3


@pytest.mark.parametrize("length,start,error", [(4, 1, AssertionError), (4, -1, AssertionError), (9, 0, RuntimeError), (-2, 0, RuntimeError)])
def test_what_is_refused_is_left_alone(length, start, error):
    src, dst = caches(8, 8)
    src.cache_seqlens.fill_(length)
    dst.cache_seqlens.fill_(start)
    before = [t.clone() for t in (dst.k_cache, dst.v_cache, dst.cache_seqlens)]
    with pytest.raises(error):
        dst.prefill(src)
    assert all(torch.equal(a, b) for a, b in zip(before, (dst.k_cache, dst.v_cache, dst.cache_seqlens)))


def test_tensors_that_the_single_call_looks_at():
    src, dst = caches(8, 8, layers=1)
    assert ops.prefill_broadcast_from(src.k_cache, src.v_cache, src.cache_seqlens.long(), dst.k_cache, dst.v_cache, dst.cache_seqlens) is None
    strided = dst.k_cache[:, :, ::2]
    assert ops.prefill_broadcast_from(src.k_cache, src.v_cache, src.cache_seqlens, strided, strided, dst.cache_seqlens) is None
    wide = torch.zeros(1, 3, 8, 2, 128, device="cuda")
    assert ops.prefill_broadcast_from(src.k_cache, src.v_cache, src.cache_seqlens, wide, wide, dst.cache_seqlens) is None


def test_an_error_waits_for_the_note(monkeypatch):
    """The pinned memory of the note goes back to its pool with the call, so nothing may still write to it."""
    src, dst = caches(8, 8)
    call = ops._lib.call

    def failing(name, *args):
        if name == "nckv_prefill_broadcast_from":
            raise RuntimeError("planted")
        return call(name, *args)

    monkeypatch.setattr(ops._lib, "call", failing)
    torch.cuda.synchronize()
    torch.cuda._sleep(int(0.2 * 1.9e9))  # the note waits behind it
    with pytest.raises(RuntimeError, match="planted"):
        dst.prefill(src)
    assert torch.cuda.current_stream().query()
