"""Prompts over a cache run the modules' hooks, subclasses' forwards and forwards that were put in a module's place."""
import pytest
import torch
import torch.nn as nn

from nanochat_b200 import gpt
from tests.test_prompt_trunk_gpu import DEV, cache_of, model_of

pytestmark = pytest.mark.gpu


def parts(model):
    block = model.transformer.h[1]
    return {"block": block, "attn": block.attn, "mlp": block.mlp, "c_v": block.attn.c_v, "c_fc": block.mlp.c_fc, "c_proj": block.mlp.c_proj}


def hooked(module, calls):
    module.register_forward_hook(lambda m, a, out: (calls.append(1), out * 0.5)[1])


def hooked_before(module, calls):
    module.register_forward_pre_hook(lambda m, a: (calls.append(1), (a[0] * 0.5, *a[1:]))[1])


def replaced(module, calls):
    own = module.forward
    module.forward = lambda *a: (calls.append(1), own(*a) * 0.5)[1]


def subclassed(module, calls):
    cls = type(module)
    module.__class__ = type("Other", (cls,), {"forward": lambda self, *a: (calls.append(1), cls.forward(self, *a) * 0.5)[1]})


def in_fp32(module, calls):
    own = module.forward
    module.forward = lambda *a: (calls.append(1), own(*a).float())[1]


@pytest.mark.parametrize("name", ["block", "attn", "mlp", "c_v", "c_fc", "c_proj"])
@pytest.mark.parametrize("change", [hooked, hooked_before, replaced, subclassed])
def test_what_is_put_around_a_module_runs(name, change):
    model = model_of(3, 256, 2)
    ids = torch.randint(0, 4096, (2, 9), generator=torch.Generator().manual_seed(3)).to(DEV)
    plain = model.forward(ids, kv_cache=cache_of(model, 2, 16))
    calls = []
    change(parts(model)[name], calls)
    got = model.forward(ids, kv_cache=cache_of(model, 2, 16))
    assert len(calls) == 1
    model.fused_glue = False
    want = model.forward(ids, kv_cache=cache_of(model, 2, 16))
    assert torch.equal(got, want) and not torch.equal(got, plain)


def test_a_product_of_another_type_runs():
    """An activation that is not bf16 goes through the eager ops, as it does in a pass without a cache."""
    model = model_of(3, 256, 2)
    ids = torch.randint(0, 4096, (2, 9), generator=torch.Generator().manual_seed(3)).to(DEV)
    plain = model.forward(ids, kv_cache=cache_of(model, 2, 16))
    in_fp32(model.transformer.h[2].mlp.c_fc, calls := [])
    got = model.forward(ids, kv_cache=cache_of(model, 2, 16))
    assert calls and got.dtype == torch.float32 and (got - plain).abs().max() < 0.1


def test_global_hooks_and_class_forwards_run(monkeypatch):
    model = model_of(2, 256, 2)
    ids = torch.randint(0, 4096, (1, 9), generator=torch.Generator().manual_seed(3)).to(DEV)
    seen = []
    handle = nn.modules.module.register_module_forward_hook(lambda m, a, out: seen.append(type(m)))
    try:
        model.forward(ids, kv_cache=cache_of(model, 1, 16))
    finally:
        handle.remove()
    assert seen.count(gpt.Block) == seen.count(gpt.Attention) == seen.count(gpt.MLP) == 2
    own, calls = gpt.MLP.forward, []
    monkeypatch.setattr(gpt.MLP, "forward", lambda self, x: (calls.append(1), own(self, x))[1])
    model.forward(ids, kv_cache=cache_of(model, 1, 16))
    assert len(calls) == 2


@pytest.mark.parametrize("of_head", [lambda z: z[..., :4000], lambda z: z.transpose(0, 1).contiguous().transpose(0, 1), lambda z: z.float()])
@pytest.mark.parametrize("T", [1, 9])
def test_logits_of_another_layout(of_head, T):
    model = model_of(2, 256, 2)
    ids = torch.randint(0, 4096, (2, T), generator=torch.Generator().manual_seed(3)).to(DEV)
    want = of_head(model.forward(ids, kv_cache=cache_of(model, 2, 16)))
    model.lm_head.register_forward_hook(lambda m, a, out: of_head(out))
    assert torch.equal(model.forward(ids, kv_cache=cache_of(model, 2, 16)), want)
