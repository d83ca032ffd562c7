"""Somewhat more heads than SMs (csrc/recurrent.cuh: recurrent_turns_kernel): heads that move between SMs give the bits of a CTA to a head."""
import pytest
import torch

from nanochat_b200 import _lib, mixer_ops as mo
from nanochat_b200 import ops

pytestmark = pytest.mark.gpu


def sizes():
    sm = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 148
    return [sm + 1, sm + 2, sm + 12, sm + sm // 3]


@pytest.mark.parametrize("pairs", sizes())
@pytest.mark.parametrize("T,D,V,form", [(256, 64, 64, "gated"), (257, 64, 64, "gated"), (1000, 64, 64, "channel"), (333, 36, 60, "gated"), (300, 64, 128, "constant"),
                                        (515, 48, 120, "constant"), (256, 64, 60, "constant")])
def test_bits(pairs, T, D, V, form):
    gen = torch.Generator(device="cuda").manual_seed(pairs + T)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    B, H = (pairs, 1) if pairs % 2 else (pairs // 2, 2)
    q, k, v, gate = rand(B * T, H * D).bfloat16(), rand(B * T, H * D).bfloat16(), rand(B * T, H * V).bfloat16(), rand(B * T, H * V).bfloat16()
    x, x0, u, nw, S0 = rand(B * T, H * D) - 2, rand(H * D), rand(H * D), rand(H * V), rand(B, H, D, V)
    decay = torch.rand(H, generator=gen, device="cuda")
    gated, channel = form == "gated", form != "constant"
    kw = dict(decay_logits=x, decay_bias=x0, bonus=u) if channel else dict(decay=decay, silu_inputs=True)
    if gated:
        kw.update(gate=gate, norm_weight=nw, eps=1e-6)
    S, want_S = S0.clone(), S0.clone()
    out = mo.recurrent(q, k, v, S, B, T, H, D, V, **kw)
    want = torch.empty_like(out)
    p = lambda t: t.data_ptr()
    _lib.call("nckv_recurrent", p(q), p(k), p(v), H * D, H * D, H * V, p(x) if channel else None, H * D, p(x0) if channel else None, p(u) if channel else None,
              None if channel else p(decay), p(gate) if gated else None, H * V if gated else 0, p(nw) if gated else None, 1e-6, p(want), H * V, p(want_S),
              B, T, H, D, V, int(not channel), 0, None, 0, torch.cuda.current_stream().cuda_stream)
    assert _lib.lib.nckv_recurrent_workspace_bytes(B, T, H, D, V) == 4 * pairs
    bits = lambda t: t.view(torch.int16 if t.element_size() == 2 else torch.int32)
    assert torch.equal(bits(out), bits(want)) and torch.equal(bits(S), bits(want_S)) and ops.read_status("cuda") == 0


def test_twice_in_a_graph_and_on_two_streams():
    B, T, H, D = sizes()[2], 256, 1, 64
    rand = lambda *s: torch.randn(*s, device="cuda")
    q, k, v, decay, S0 = rand(B * T, D).bfloat16(), rand(B * T, D).bfloat16(), rand(B * T, D).bfloat16(), torch.rand(H, device="cuda"), rand(B, H, D, D)
    run = lambda S: mo.recurrent(q, k, v, S, B, T, H, D, D, decay=decay)
    S = S0.clone()
    want = [run(S), run(S)]
    want_S = S.clone()
    streams = [torch.cuda.Stream() for _ in range(2)]
    results = []
    torch.cuda.synchronize()
    for st in streams:
        with torch.cuda.stream(st):
            S = S0.clone()
            results.append(([run(S), run(S)], S))
    torch.cuda.synchronize()
    for got, S in results:
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and torch.equal(S, want_S)
    graph, S = torch.cuda.CUDAGraph(), S0.clone()
    with torch.cuda.stream(streams[0]):
        with torch.cuda.graph(graph, stream=streams[0]):
            out = run(S)
        for i in range(2):
            graph.replay()
            streams[0].synchronize()
            assert torch.equal(out, want[i])
