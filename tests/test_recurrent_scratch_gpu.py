"""Recurrences whose calls need scratch (heads that take turns, segments): from two threads on one stream, and replayed behind calls that need more."""
import threading

import pytest
import torch

from nanochat_b200 import _lib, mixer_ops as mo
from nanochat_b200 import ops

pytestmark = pytest.mark.gpu

SMS = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 148
FORMS = [(SMS + 12, 256, 1, 64), (2, 2048, 2, 64)]  # one head or more than an SM; few heads, in segments


def inputs(B, T, H, D, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k, v = (rand(B * T, H * D).bfloat16() for _ in range(3))
    decay, state = torch.rand(H, generator=gen, device="cuda"), rand(B, H, D, D)
    assert _lib.lib.nckv_recurrent_workspace_bytes(B, T, H, D, D) > 0
    return lambda S: mo.recurrent(q, k, v, S, B, T, H, D, D, decay=decay), state


@pytest.mark.parametrize("form", FORMS)
def test_two_threads_on_one_stream(form):
    work = [inputs(*form, seed) for seed in (1, 2)]
    want = []
    for run, S0 in work:
        S = S0.clone()
        want.append((run(S), S))
    torch.cuda.synchronize()
    got, start = [None, None], threading.Barrier(2)

    def several(i):
        run, S0 = work[i]
        states, outs = [S0.clone() for _ in range(40)], []
        start.wait()
        for S in states:
            outs.append(run(S))
        got[i] = states, outs

    threads = [threading.Thread(target=several, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for (states, outs), (out, S) in zip(got, want):
        assert all(torch.equal(o, out) for o in outs) and all(torch.equal(s, S) for s in states)
    assert ops.read_status("cuda") == 0


@pytest.mark.parametrize("form", FORMS)
def test_replayed_behind_a_call_that_needs_more(form):
    run, S0 = inputs(*form, 3)
    larger, L0 = inputs(4, 4096, 2, 128, 4)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        S = S0.clone()
        want = run(S)
        want_S = S.clone()
        S.copy_(S0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = run(S)
        L = L0.clone()
        larger_want = larger(L)
        others = [torch.full((n,), 7, dtype=torch.int32, device="cuda") for n in (16, 100, 160, 1000, 10000, 1 << 20) for _ in range(20)]
        for _ in range(3):
            S.copy_(S0)
            graph.replay()
            L.copy_(L0)
            larger_got = larger(L)
            assert torch.equal(out, want) and torch.equal(S, want_S) and torch.equal(larger_got, larger_want)
        assert all((t == 7).all() for t in others)
        side.synchronize()
    assert ops.read_status("cuda") == 0


def test_heads_take_turns_while_other_kernels_hold_sms():
    """Part of the grid is resident at first: whoever waits for a head, its CTA has started."""
    run, S0 = inputs(SMS + SMS // 3, 256, 1, 64, 5)
    S = S0.clone()
    want = run(S)
    a = torch.randn(8192, 8192, device="cuda").bfloat16()
    b = a @ a
    states, outs = [S0.clone() for _ in range(20)], []
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        for _ in range(6):
            torch.mm(a, a, out=b)
    for s in states:
        outs.append(run(s))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs) and all(torch.equal(s, S) for s in states) and ops.read_status("cuda") == 0
