"""Pages of a size that the attention refuses are refused before anything is written."""
import types

import pytest
import torch

from nanochat_b200 import ops
from nanochat_b200.gpt import kv_attention, precompute_rotary_embeddings
from tests.test_native_calls_gpu import BF, DEV, rand

pytestmark = pytest.mark.gpu


def test_pages_of_another_size():
    tokens, G = ops.PAGE_TILE + 8, 2
    pool = [torch.zeros(3, tokens, G, 128, dtype=BF, device=DEV) for _ in range(2)]
    cache = types.SimpleNamespace(paged=True, n_layers=1, block_table=torch.tensor([[1, 0], [2, 0]], dtype=torch.int32, device=DEV),
                                  cache_seqlens=torch.tensor([3, 9], dtype=torch.int32, device=DEV), get_layer_cache=lambda i: pool)
    cos, sin = precompute_rotary_embeddings(512, 128, device=DEV)
    ops.workspace(torch.device("cuda", 0), 2, 4, G)
    with pytest.raises(RuntimeError):
        kv_attention(rand(2, 1, 4, 128), rand(2, 1, G, 128, seed=1), rand(2, 1, G, 128, seed=2), (cos, sin), (-1, 0), cache, 0)
    assert not any(t.any() for t in pool)
