"""Native calls from several threads: each other's results, and the interpreter while a launch waits."""
import threading
import time

import pytest
import torch

from nanochat_b200 import ops
from nanochat_b200.gpt import kv_attention, precompute_rotary_embeddings
from tests.test_native_calls_gpu import BF, DEV, rand, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["relu", "mix", "attention"])
def test_other_threads_run_while_a_launch_waits(call):
    """A thread fills its launch queue behind a third of a second of work on the device; another one counts on."""
    x = rand(4, 1, 512)
    cos, sin = precompute_rotary_embeddings(512, 128, device=DEV)
    cache, q, k, v = state("packed", 2, 1, 4, 2, 400)
    run = {"relu": lambda: ops.glue_relu_sq(x), "mix": lambda: ops.glue_mix_norm(x, add=x),
           "attention": lambda: kv_attention(q, k, v, (cos, sin), (-1, 0), cache, 0)}[call]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        run()
        run()
    torch.cuda.synchronize()
    done = threading.Event()

    def launches():
        with torch.cuda.stream(side):
            torch.cuda._sleep(int(0.35 * 1.9e9))
            for _ in range(4000):
                run()
        done.set()

    thread = threading.Thread(target=launches)
    longest, last = 0.0, time.perf_counter()
    thread.start()
    while not done.is_set():
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
    thread.join()
    torch.cuda.synchronize()
    assert longest < 0.15, f"the interpreter stood still for {longest:.3f} s"


def test_threads_on_streams_of_their_own():
    cos, sin = precompute_rotary_embeddings(512, 128, device=DEV)
    want, got = {}, {}

    def work(n, out):
        cache, q, k, v = state("packed", 1 + n, 1, 8, 2, 400)
        x = rand(3 + n, 256, seed=n)
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
            for _ in range(50):
                y = kv_attention(q, k, v, (cos, sin), (64, 0), cache, 0)
                z = ops.glue_mix_norm(x, add=x, want_sum=True)
            torch.cuda.current_stream().synchronize()
        out[n] = (y, *z)
    for n in range(4):
        work(n, want)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(n, got)) for n in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for n in range(4):
        assert all(torch.equal(a, b) for a, b in zip(got[n], want[n]))
