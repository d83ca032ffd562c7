"""Off the GPU the native calls take nothing, and the general path says why."""
import pytest
import torch

from nanochat_b200 import _lib, ops


def test_nothing_is_taken_off_the_gpu():
    x = torch.zeros(2, 1, 128, dtype=torch.bfloat16)
    assert _lib.native.glue_relu_sq(x) is None
    assert _lib.native.glue_mix_norm(x, None, None, None, 1.0, 0.0, 0.0, False, True, True, 1e-6) is None
    q, cache, lens, table = (torch.zeros(*s, dtype=t) for s, t in (((2, 1, 4, 128), torch.bfloat16), ((2, 8, 4, 128), torch.bfloat16),
                                                                   ((2,), torch.int32), ((8, 64), torch.bfloat16)))
    assert ops.append_and_attend(q, q, q, cache, cache, None, lens, table, table, -1) is None
    with pytest.raises(RuntimeError):
        ops.glue_relu_sq(x)
    with pytest.raises(RuntimeError):
        ops.append_rope_norm(q, q, q, cache, cache, lens, table, table)
