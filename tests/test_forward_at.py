"""forward_at over models whose forward is another than GPT's."""
import torch

from nanochat_b200.engine import forward_at
from nanochat_b200.gpt import GPT, GPTConfig


def whole(self, idx, targets=None, kv_cache=None, loss_reduction="mean"):
    return torch.arange(idx.numel() * 3.0).view(*idx.shape, 3)


class Own(GPT):
    forward = whole


class Placing(GPT):
    accepts_logits_at = True

    def forward(self, idx, kv_cache=None, logits_at=None):
        return whole(self, idx)[:, logits_at] + 1


def model(cls):
    with torch.device("meta"):
        return cls(GPTConfig(n_layer=1, n_head=1, n_kv_head=1, n_embd=128, vocab_size=64))


def test_a_forward_without_places(monkeypatch):
    ids = torch.zeros(2, 4, dtype=torch.long)
    want = whole(None, ids)[:, [3, -2]]
    replaced = model(GPT)
    replaced.forward = whole.__get__(replaced)
    for m in (model(Own), replaced):
        assert torch.equal(forward_at(m, ids, None, [3, -2]), want)
    assert torch.equal(forward_at(model(Placing), ids, None, [3, -2]), want + 1)
    assert model(GPT).accepts_logits_at
    monkeypatch.setattr(GPT, "forward", whole)
    assert torch.equal(forward_at(model(GPT), ids, None, [3, -2]), want)
