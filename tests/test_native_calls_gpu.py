"""The native calls against the general Python path: same bits where they apply, None where they do not, same errors."""
import pytest
import torch

from nanochat_b200 import _lib, ops
from nanochat_b200.engine import KVCache, PagedKVCache
from nanochat_b200.gpt import kv_attention, precompute_rotary_embeddings

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


class General:
    """Stands in for the native module and takes nothing."""

    set_workspace = staticmethod(_lib.native.set_workspace)

    def __getattr__(self, name):
        return lambda *a: None


class Counting:
    """The native module, with a count of the calls that it took."""

    def __init__(self):
        self.taken = 0

    def __getattr__(self, name):
        fn = getattr(_native, name)

        def call(*a):
            out = fn(*a)
            self.taken += out is not None and name != "set_workspace"
            return out
        return call


_native = _lib.native


def rand(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV, BF)


def state(kind, B, T, H, G, cap):
    cache = (PagedKVCache if kind == "paged" else KVCache)(B, G, cap, 128, 2, DEV, BF)
    if kind == "paged":
        cache.reserve(cap)
    for i, t in enumerate(cache.get_layer_cache(0)):
        t.copy_(rand(*t.shape, seed=10 + i))
    cache.cache_seqlens.copy_(torch.arange(B, dtype=torch.int32) * 3 % (cap - T + 1))
    x = rand(B, T, (H + 2 * G) * 128, seed=3)
    q, k, v = (z.view(B, T, -1, 128) for z in x.split([H * 128, G * 128, G * 128], 2))
    if kind == "slices":
        return cache, q, k, v
    if kind == "transposed":  # heads outermost: no common token stride
        return cache, *(z.transpose(1, 2).contiguous().transpose(1, 2) for z in (q, k, v))
    return cache, q.contiguous(), k.contiguous(), v.contiguous()


@pytest.mark.parametrize("kind,B,T,H,G,window,native", [
    ("packed", 1, 1, 2, 2, -1, True), ("packed", 33, 1, 16, 4, 7, True), ("packed", 2, 5, 12, 12, -1, True), ("packed", 1, 130, 4, 1, 64, True),
    ("slices", 7, 1, 12, 12, 100, True), ("slices", 2, 9, 6, 2, -1, True), ("paged", 5, 1, 8, 2, -1, True), ("transposed", 2, 6, 4, 4, -1, False),
    ("transposed", 3, 1, 4, 4, 2, True), ("packed", 2, 1, 16, 1, -1, True)])
def test_kv_attention(monkeypatch, kind, B, T, H, G, window, native):
    cos, sin = precompute_rotary_embeddings(512, 128, device=DEV)
    out = []
    for module in (General(), Counting()):
        monkeypatch.setattr(_lib, "native", module)
        cache, q, k, v = state(kind, B, T, H, G, 400)
        ops.workspace(torch.device("cuda", 0), B, H, G)
        for layer in (0, 1):  # the second is the last: the lengths move on
            y = kv_attention(q, k, v, (cos, sin), (window, 0), cache, layer)
        kc, vc = cache.get_layer_cache(0)
        lens = cache.cache_seqlens.clone()
        out.append((kv_attention(q, k, v, (cos, sin), (window, 0), cache, 0), kc, vc, lens, y.shape))
    taken = _lib.native.taken
    assert taken == (3 if native else 0)
    for a, b in zip(*out):
        assert a == b if isinstance(a, torch.Size) else torch.equal(a, b)
    assert ops.read_status(DEV) == 0


def test_what_the_general_path_refuses_is_refused():
    cos, sin = precompute_rotary_embeddings(512, 128, device=DEV)
    cache, q, k, v = state("packed", 2, 3, 4, 2, 64)
    call = lambda **kw: kv_attention(kw.get("q", q), kw.get("k", k), kw.get("v", v), kw.get("t", (cos, sin)), (-1, 0), kw.get("c", cache), 0)
    call()
    short = KVCache(2, 2, 2, 128, 2, DEV, BF)
    with pytest.raises(_lib.NckvError) as e:  # three tokens into rows of two
        call(c=short)
    assert e.value.code == -3
    other = KVCache(3, 2, 64, 128, 2, DEV, BF)
    for kw in (dict(q=q.float()), dict(k=k[:, :2]), dict(v=v.half()), dict(c=other), dict(q=q.cpu()), dict(q=q[..., :64].contiguous()),
               dict(t=(cos.float(), sin.float()))):
        with pytest.raises(RuntimeError):
            call(**kw)


def test_another_stream_has_its_own_scratch():
    cos, sin = precompute_rotary_embeddings(512, 128, device=DEV)
    cache, q, k, v = state("packed", 4, 1, 4, 2, 300)
    want = kv_attention(q, k, v, (cos, sin), (-1, 0), cache, 0)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        first = kv_attention(q, k, v, (cos, sin), (-1, 0), cache, 0)   # the general path makes this stream's scratch
        second = kv_attention(q, k, v, (cos, sin), (-1, 0), cache, 0)  # the native call finds it
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(first, want) and torch.equal(second, want)


@pytest.mark.parametrize("shape", [(1, 1, 128), (5, 1, 256), (2, 37, 1536), (3, 640)])
def test_glue(monkeypatch, shape):
    x, add, x0 = (rand(*shape, seed=i) for i in range(3))
    out = []
    for module in (General(), Counting()):
        monkeypatch.setattr(_lib, "native", module)
        out.append([ops.glue_mix_norm(x, want_x=False), ops.glue_mix_norm(x, add=add, x0=x0, resid_lambda=1.1, x0_lambda=0.3, want_sum=True),
                    ops.glue_mix_norm(x, add=add, x_backout=x0, backout_lambda=0.2), ops.glue_mix_norm(x, want_sum=True, want_norm=False),
                    (ops.glue_relu_sq(x),)])
    assert _lib.native.taken == 5
    for a, b in zip(*out):
        for s, t in zip(a, b):
            assert (s is None) == (t is None) and (s is None or torch.equal(s, t))
    with pytest.raises(RuntimeError):
        ops.glue_mix_norm(x, add=add[..., 1:])
    with pytest.raises(RuntimeError):
        ops.glue_relu_sq(x.float())
