"""The scratch of a recurrence belongs to the call: nothing of it is shared between threads or kept behind the call."""
import contextlib
import gc
import threading
import types

import pytest
import torch

from nanochat_b200 import mixer_ops as mo

B, T, H, D = 1, 2, 1, 4


@pytest.fixture
def native(monkeypatch):
    """The binding's side replaced: calls are noted with the address of their scratch, the argument before last but two."""
    fake = types.SimpleNamespace(calls=[], meet=None)

    def call(name, *args):
        fake.calls.append(args[-4])
        if fake.meet is not None:
            fake.meet.wait(10)

    monkeypatch.setattr(mo, "_lib", types.SimpleNamespace(call=call, lib=types.SimpleNamespace(nckv_recurrent_workspace_bytes=lambda *a: 4096)))
    monkeypatch.setattr(mo, "_ctx", lambda t: (0, 0))
    monkeypatch.setattr(mo.ops, "_require_cuda", lambda *a: None)
    monkeypatch.setattr(mo.ops, "_device_guard", lambda idx: contextlib.nullcontext())
    monkeypatch.setattr(mo.ops, "workspace", lambda *a: torch.zeros(1))
    return fake


def run():
    rows = torch.zeros(B * T, H * D, dtype=torch.bfloat16)
    mo.recurrent(rows, rows, rows, torch.zeros(B, H, D, D), B, T, H, D, D, decay=torch.ones(H))


def test_calls_at_the_same_time_have_scratch_of_their_own(native):
    run()
    native.calls.clear()
    native.meet = threading.Barrier(2)
    threads = [threading.Thread(target=run) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(set(native.calls)) == 2 and None not in native.calls


def test_nothing_is_kept_behind_the_call(native):
    run()
    gc.collect()
    assert not [t for t in gc.get_objects() if type(t) is torch.Tensor and t.data_ptr() == native.calls[0]]
