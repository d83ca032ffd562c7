"""Native calls that find no memory raise what torch raises."""
import pytest
import torch

from nanochat_b200 import ops
from nanochat_b200.gpt import kv_attention, precompute_rotary_embeddings
from tests.test_native_calls_gpu import BF, DEV, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["relu", "mix", "mix_at", "attention"])
def test_out_of_memory(call):
    """The allocator of this process is limited to what it holds, 64 MB of outputs asked for."""
    x = torch.zeros(1 << 15, 1024, dtype=BF, device=DEV)
    lam = torch.zeros(1, device=DEV)
    cos, sin = precompute_rotary_embeddings(4096, 128, device=DEV)
    cache, q, k, v = state("packed", 8, 2048, 16, 1, 2100)
    run = {"relu": lambda: ops.glue_relu_sq(x), "mix": lambda: ops.glue_mix_norm(x),
           "mix_at": lambda: ops.glue_mix_norm_at(x, x_backout=x, backout_lambda=lam),
           "attention": lambda: kv_attention(q, k, v, (cos, sin), (-1, 0), cache, 0)}[call]
    ops.workspace(torch.device("cuda", 0), 8, 16, 1)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            run()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    out = run()
    assert out is not None and ops.read_status(DEV) == 0
