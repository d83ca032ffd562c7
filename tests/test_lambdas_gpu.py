"""The trunk's scalar parameters written or replaced between passes: prompts and decode steps see them as they are now."""
import pytest
import torch
import torch.nn as nn

from nanochat_b200 import ops
from nanochat_b200.engine import GraphedDecodeStep
from tests.test_prompt_trunk_gpu import BF, DEV, cache_of, model_of

pytestmark = pytest.mark.gpu


def replaced(model, name):
    old = getattr(model, name)
    setattr(model, name, nn.Parameter((old.detach() + 0.25).to(old.dtype)))


def written(model, name):
    getattr(model, name).data.add_(0.25)


def loaded(model, name):
    model.load_state_dict({name: (getattr(model, name).detach() + 0.25)}, strict=False, assign=True)


def passes(model, ids):
    cache = cache_of(model, 2, 64)
    prompt = model.forward(ids, kv_cache=cache)
    return prompt, model.forward(ids[:, :1], kv_cache=cache), cache.k_cache, cache.v_cache


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("change", [replaced, written, loaded])
@pytest.mark.parametrize("name", ["resid_lambdas", "x0_lambdas", "backout_lambda"])
def test_a_changed_scalar_is_seen(name, change, dtype):
    model = model_of(3, 256, 2)
    for n in ("resid_lambdas", "x0_lambdas", "backout_lambda"):
        getattr(model, n).data = getattr(model, n).data.to(dtype)
    ids = torch.randint(0, 4096, (2, 21), generator=torch.Generator().manual_seed(3)).to(DEV)
    before = passes(model, ids)
    change(model, name)
    got = passes(model, ids)
    model.fused_glue = False
    want = passes(model, ids)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert not torch.equal(got[0], before[0]) and not torch.equal(got[1], before[1])


def test_a_replayed_step_sees_a_written_scalar():
    replayed_step(model_of(3, 256, 2))


@torch.inference_mode()
def replayed_step(model):
    ids = torch.randint(0, 4096, (2, 5), generator=torch.Generator().manual_seed(3)).to(DEV)
    cache = cache_of(model, 2, 64)
    model.forward(ids, kv_cache=cache)
    step = GraphedDecodeStep(model, cache, ids[:, :1])
    step.step(ids[:, :1])
    for name in ("resid_lambdas", "x0_lambdas", "backout_lambda"):
        written(model, name)
    before = [t.clone() for t in (cache.cache_seqlens, cache.prev_embedding)]
    got = step.step(ids[:, 1:2]).clone()
    cache.cache_seqlens.copy_(before[0])
    cache.prev_embedding = before[1]
    assert torch.equal(got, model.forward(ids[:, 1:2], kv_cache=cache)[:, -1])


@pytest.mark.parametrize("C", [4, 512, 8192])
@pytest.mark.parametrize("dtypes", [(BF, BF, BF), (torch.float32, BF, torch.float32)])
def test_scalars_on_the_device_mix_as_numbers_do(monkeypatch, C, dtypes):
    from nanochat_b200 import _lib
    gen = torch.Generator().manual_seed(C)
    x, add, other = (torch.randn(5, C, generator=gen).to(DEV, BF) for _ in range(3))
    lam = [torch.tensor([0.1, v], device=DEV).to(t) for v, t in zip((1.083, 0.1337, 0.2), dtypes)]
    lam[2] = lam[2][1:]
    num = [float(t[-1].to(BF)) for t in lam]
    native = _lib.native

    class General:
        def __getattr__(self, name):
            return lambda *a: None
    for module in (native, General()):
        monkeypatch.setattr(_lib, "native", module)
        got = (*ops.glue_mix_norm_at(x, add=add, x0=other, resid_lambdas=lam[0], x0_lambdas=lam[1], layer=1, want_sum=True),
               *ops.glue_mix_norm_at(x, add=add, x_backout=other, backout_lambda=lam[2]), *ops.glue_mix_norm_at(x, want_x=False))
        want = (*ops.glue_mix_norm(x, add=add, x0=other, resid_lambda=num[0], x0_lambda=num[1], want_sum=True),
                *ops.glue_mix_norm(x, add=add, x_backout=other, backout_lambda=num[2]), *ops.glue_mix_norm(x, want_x=False))
        assert all((a is None) == (b is None) and (a is None or torch.equal(a, b)) for a, b in zip(got, want))
        for bad in (dict(resid_lambdas=lam[0]), dict(resid_lambdas=lam[0].cpu(), x0_lambdas=lam[1]),
                    dict(resid_lambdas=lam[0].double(), x0_lambdas=lam[1]), dict(resid_lambdas=lam[0], x0_lambdas=lam[1], layer=2),
                    dict(resid_lambdas=lam[0], x0_lambdas=lam[1], layer=-1)):
            with pytest.raises(RuntimeError):
                ops.glue_mix_norm_at(x, x0=other, **bad)
