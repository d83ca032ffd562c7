"""Prompts through the fused trunk, logits at chosen places, the soft cap in one launch."""
import pytest
import torch

from nanochat_b200 import ops
from nanochat_b200.engine import KVCache, forward_at
from nanochat_b200.gpt import GPT, GPTConfig

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


@pytest.mark.parametrize("rows,width,cols", [(1, 8, 8), (3, 64, 61), (5, 64, 64), (2, 4160, 4104), (70000, 16, 16), (1, 32768, 32768)])
def test_logit_cap_is_the_eager_sequence(rows, width, cols):
    z = (torch.randn(rows, width, generator=torch.Generator().manual_seed(1)) * 20).to(DEV, BF)
    z[0, 0], z[-1, cols - 1] = float("inf"), float("nan")
    want = 15 * torch.tanh(z[..., :cols].float() / 15)
    got = ops.glue_logit_cap(z, cols, 15.0)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert ops.glue_logit_cap(z[:0], cols, 15.0).shape == (0, cols)


def model_of(n_layer, n_embd, n_head, vocab=4096):
    torch.manual_seed(5)
    with torch.device("meta"):
        model = GPT(GPTConfig(sequence_len=512, vocab_size=vocab, n_layer=n_layer, n_head=n_head, n_kv_head=n_head, n_embd=n_embd),
                    compute_dtype=BF)
    model.to_empty(device=DEV)
    model.init_weights()
    for blk in model.transformer.h:  # let attention and MLP reach the residual stream
        torch.nn.init.normal_(blk.attn.c_proj.weight, std=n_embd ** -0.5)
        torch.nn.init.normal_(blk.mlp.c_proj.weight, std=n_embd ** -0.5)
    torch.nn.init.normal_(model.lm_head.weight, std=0.02)
    model.smear_lambda.data.fill_(0.5)
    return model.to(BF)


def cache_of(model, rows, length):
    cfg = model.config
    return KVCache(rows, cfg.n_kv_head, length, cfg.n_embd // cfg.n_head, cfg.n_layer, DEV, BF)


@pytest.mark.parametrize("n_layer,n_embd,n_head,B,T", [(1, 128, 1, 2, 2), (2, 256, 2, 1, 129), (3, 640, 5, 3, 40), (4, 1536, 12, 1, 700)])
def test_prompt_logits_and_cache_are_those_of_the_eager_trunk(n_layer, n_embd, n_head, B, T):
    model = model_of(n_layer, n_embd, n_head, vocab=4093)
    ids = torch.randint(0, 4093, (B, T), generator=torch.Generator().manual_seed(9)).to(DEV)
    runs = []
    for fused in (False, True):
        model.fused_glue = fused
        cache = cache_of(model, B, T + 3)
        runs.append((model.forward(ids, kv_cache=cache), model.forward(ids[:, :3], kv_cache=cache), cache))
    (a, a2, ca), (b, b2, cb) = runs
    assert torch.equal(a, b) and torch.equal(a2, b2)
    assert all(torch.equal(x, y) for x, y in ((ca.k_cache, cb.k_cache), (ca.v_cache, cb.v_cache), (ca.cache_seqlens, cb.cache_seqlens)))


def test_logits_at_chosen_places():
    """A product over fewer rows may be cut differently: bf16 logits agree to one rounding (2^-8 of values up to 3)."""
    model, T = model_of(2, 256, 2), 37
    ids = torch.randint(0, 4096, (2, T), generator=torch.Generator().manual_seed(9)).to(DEV)
    for fused in (False, True):
        model.fused_glue = fused
        every = model.forward(ids, kv_cache=cache_of(model, 2, T))
        for places in ([T - 1], [3, -1, 0], []):
            some = forward_at(model, ids, cache_of(model, 2, T), places)
            assert some.shape == (2, len(places), 4096)
            torch.testing.assert_close(some, every[:, places], rtol=2 ** -7, atol=2 ** -8 * 3)


def test_a_captured_prompt_takes_the_eager_trunk_until_the_lambdas_are_known():
    model, T = model_of(2, 256, 2), 20
    ids = torch.randint(0, 4096, (1, T), generator=torch.Generator().manual_seed(9)).to(DEV)
    model.fused_glue = False
    want = model.forward(ids, kv_cache=cache_of(model, 1, T))
    model.fused_glue = True
    cache = cache_of(model, 1, T)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        ops.workspace(torch.device("cuda", 0), 1, 2, 2)  # scratch and cuBLAS are set up ahead of a capture
        model.fused_glue = False
        model.forward(ids, kv_cache=cache)
        model.fused_glue = True
        cache.reset()
        side.synchronize()
        assert model._lambda_cache is None
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            got = model.forward(ids, kv_cache=cache)
    torch.cuda.current_stream().wait_stream(side)
    cache.reset()
    graph.replay()
    assert torch.equal(got, want)
