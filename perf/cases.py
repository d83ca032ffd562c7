"""The work that a user of this package has it do, as cases that can be timed and compared.

One path per entry point:
  decode    ``gpt.kv_attention`` with one new token per row: RoPE, norm, append and attention of one layer, ragged rows
  pages     the same over a ``PagedKVCache``
  chunk     ``gpt.kv_attention`` with several new tokens per row behind what the cache holds (prompts and their portions)
  train     ``flash_attn.flash_attn_func`` with its backward pass
  broadcast ``KVCache.prefill``: one prompt to all sample rows
  prompt    a whole model over new tokens: logits at the last place (what generation needs) or at all (scoring)
  step      a whole model's decode step, replayed as ``Engine`` does (``GraphedDecodeStep``)
The models are the three designs of the package: ``gpt``, ``sipadra`` (recurrent and windowed layers) and ``zuvulorn``
(gated recurrences, delta rule, attention, experts), at the widths 1536 and 2048 with the sizes of the benchmark.
Everything is bfloat16, the type that the package serves and trains in; weights and activations are random.
"""
import math

import torch
import torch.nn.functional as F

from nanochat_b200.engine import GraphedDecodeStep, KVCache, PagedKVCache, forward_at, new_cache
from nanochat_b200.flash_attention import flash_attn
from nanochat_b200.gpt import GPT, kv_attention
from nanochat_b200.models import model_class

D, VOCAB, BF, F64 = 128, 32768, torch.bfloat16, torch.float64

# width -> sizes of a layer in the three designs (the benchmark's d24 and d32)
GPT_SIZES = {1536: dict(heads=12, kv_heads=12), 2048: dict(heads=16, kv_heads=4)}
SIPADRA_SIZES = {1536: dict(ff=4096, wkv_heads=24, left=(12, 12), window=1024, right=(12, 64, 128), rank=64),
                 2048: dict(ff=5504, wkv_heads=32, left=(16, 4), window=2048, right=(16, 128, 128), rank=96)}
ZUVULORN_SIZES = {1536: dict(ff=1024, blocks=12, delta=12, attn=(12, 12), rank=64),
                  2048: dict(ff=1376, blocks=16, delta=16, attn=(16, 4), rank=96)}
EXPERTS, TOP, STREAMS, TAPS = 16, 4, 4, 4


def listed():
    return [
        # four samples just behind a short prompt on the smallest configuration: launches and latency only
        dict(name="decode_few", path="decode", rows=4, heads=2, kv_heads=2, capacity=2048, low=32, high=96, window=-1),
        # the op-level benchmark: 32 ragged rows, full causal
        dict(name="decode_ragged", path="decode", rows=32, heads=12, kv_heads=12, capacity=2048, low=1, high=2047, window=-1),
        # long context, few rows, grouped heads
        dict(name="decode_long", path="decode", rows=8, heads=16, kv_heads=4, capacity=65536, low=32768, high=65535, window=-1),
        # a serving batch in pages on a layer with a short window
        dict(name="decode_pages", path="pages", rows=256, heads=16, kv_heads=4, capacity=4096, low=128, high=3071, window=2048),
        # a portion of odd length behind a ragged context, grouped heads, window
        dict(name="chunk_window", path="chunk", rows=3, tokens=1531, heads=16, kv_heads=4, capacity=6144, low=1024, high=4096,
             window=2048),
        # attention of a training step, both directions
        dict(name="train_attention", path="train", rows=8, tokens=2048, heads=12, kv_heads=12, window=-1),
        # an 8192-token prompt to 64 sample rows
        dict(name="broadcast", path="broadcast", rows=64, tokens=8192, kv_heads=4, layers=1, capacity=8192),
        # the prompt of a generation: one row, logits at its end
        dict(name="gpt_prompt", path="prompt", model="gpt", width=1536, layers=8, rows=1, tokens=2048, logits="last"),
        # the decode step of a served batch, all 24 layers
        dict(name="gpt_step", path="step", model="gpt", width=1536, layers=24, rows=64, low=512, high=1023),
        # scoring a batch of texts: logits at every place
        dict(name="sipadra_prompt", path="prompt", model="sipadra", width=1536, layers=3, rows=8, tokens=2048, logits="all"),
        # scoring one long text of odd length, all kinds of layers
        dict(name="zuvulorn_prompt", path="prompt", model="zuvulorn", width=1536, layers=6, rows=1, tokens=6007, logits="all"),
        # a served batch on the design with experts
        dict(name="zuvulorn_step", path="step", model="zuvulorn", width=1536, layers=6, rows=64, low=512, high=1023),
    ]


def draw(rng):
    def spread(low, high):
        return min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))

    path = rng.choice(["decode", "decode", "pages", "chunk", "train", "broadcast", "prompt", "prompt", "prompt", "step", "step", "step"])
    heads, kv_heads = rng.choice([(2, 2), (6, 6), (12, 12), (16, 4), (16, 16), (16, 2)])
    if path in ("decode", "pages"):
        rows = spread(1, 256)
        high = spread(16, min(32768, max(16, (1 << 22) // (rows * kv_heads))))
        return dict(path=path, rows=rows, heads=heads, kv_heads=kv_heads, capacity=-(-(high + 1) // 64) * 64, low=spread(1, high), high=high,
                    window=rng.choice([-1, -1, 1024, spread(8, high)]))
    if path == "chunk":
        rows = spread(1, 16)
        tokens = spread(2, min(8192, 32768 // rows))
        high = spread(1, 16384)
        return dict(path=path, rows=rows, tokens=tokens, heads=heads, kv_heads=kv_heads, capacity=high + tokens, low=rng.choice([0, spread(1, high)]),
                    high=high, window=rng.choice([-1, 1024, spread(8, high + tokens)]))
    if path == "train":
        rows = spread(1, 16)
        return dict(path=path, rows=rows, tokens=spread(16, min(4096, 24576 // rows)), heads=heads, kv_heads=kv_heads,
                    window=rng.choice([-1, -1, 512, 1024]))
    if path == "broadcast":
        rows, layers = spread(1, 64), rng.choice([1, 2, 4, 8])
        tokens = spread(1, min(32768, max(1, (1 << 21) // (rows * layers * kv_heads))))
        return dict(path=path, rows=rows, tokens=tokens, kv_heads=kv_heads, layers=layers, capacity=tokens + rng.randrange(64))
    model, width = rng.choice(["gpt", "sipadra", "zuvulorn"]), rng.choice([1536, 2048])
    if path == "prompt":
        rows = spread(1, 8)
        return dict(path=path, model=model, width=width, layers=rng.choice([3, 4, 6]) if width == 1536 else 3, rows=rows,
                    tokens=spread(2, min(8192, 8192 // rows)), logits="all" if model == "zuvulorn" else rng.choice(["last", "all"]))
    low = spread(1, 2048)
    return dict(path=path, model=model, width=width, layers=rng.choice([3, 6]), rows=spread(1, 128), low=low, high=low + rng.randrange(512))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
class Draws:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, dtype=BF, scale=1.0):
        return (torch.randn(*shape, generator=self.gen, device="cuda") * scale).to(dtype)

    def whole(self, low, high, *shape, dtype=torch.int32):
        return torch.randint(low, high + 1, shape, generator=self.gen, device="cuda", dtype=dtype)

    def fill(self, t, scale=1.0):
        """Normal values in place, slice by slice: a cache can be most of what fits."""
        for part in t.view(-1).split(1 << 28):
            part.copy_(torch.randn(part.numel(), generator=self.gen, device=part.device) * scale)


def rotary(length):
    """The tables of the GPT design, (1, length, 1, 64) cosines and sines in bfloat16."""
    freq = 1.0 / (100000 ** (torch.arange(0, D, 2, dtype=torch.float32, device="cuda") / D))
    angle = torch.outer(torch.arange(length, dtype=torch.float32, device="cuda"), freq)
    return angle.cos().to(BF)[None, :, None], angle.sin().to(BF)[None, :, None]


def attention_state(c, seed):
    """A cache of two layers, so that a call for the first one leaves the rows' lengths alone."""
    d = Draws(seed)
    tokens = c.get("tokens", 1)
    lengths = d.whole(c["low"], c["high"], c["rows"])
    args = (c["rows"], c["kv_heads"], c["capacity"], D, 2, "cuda", BF)
    if c["path"] == "pages":
        cache = PagedKVCache(*args)
        cache.reserve(c["capacity"])
    else:
        cache = KVCache(*args)
    for t in cache.get_layer_cache(0):
        d.fill(t)
    cache.cache_seqlens.copy_(lengths)
    q, k, v = (d.normal(c["rows"], tokens, h, D) for h in (c["heads"], c["kv_heads"], c["kv_heads"]))
    return dict(cache=cache, q=q, k=k, v=v, tables=rotary(c["capacity"] + 1), window=(c["window"], 0))


def train_state(c, seed):
    d = Draws(seed)
    q, k, v = (d.normal(c["rows"], c["tokens"], h, D).requires_grad_() for h in (c["heads"], c["kv_heads"], c["kv_heads"]))
    return dict(q=q, k=k, v=v, grad=d.normal(c["rows"], c["tokens"], c["heads"], D), window=(c["window"], 0))


def broadcast_state(c, seed):
    d = Draws(seed)
    src = KVCache(1, c["kv_heads"], c["tokens"], D, c["layers"], "cuda", BF)
    dst = KVCache(c["rows"], c["kv_heads"], c["capacity"], D, c["layers"], "cuda", BF)
    d.fill(src.k_cache)
    d.fill(src.v_cache)
    src.cache_seqlens.fill_(c["tokens"])
    return dict(src=src, dst=dst)


def design(c):
    """config.json of the case's model."""
    W, n = c["width"], c["layers"]
    if c["model"] == "gpt":
        s = GPT_SIZES[W]
        return dict(sequence_len=4096, vocab_size=VOCAB, n_layer=n, n_head=s["heads"], n_kv_head=s["kv_heads"], n_embd=W)
    if c["model"] == "sipadra":
        s = SIPADRA_SIZES[W]
        mlp, (h, g), (rh, rd, rv) = {"kind": "dense", "ff": s["ff"]}, s["left"], s["right"]
        rot = {"base": 500000.0, "dims": D, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
        wkv = {"type": "wkv", "mixer": {"heads": s["wkv_heads"], "dim": 64}, "mlp": mlp}
        par = {"type": "parallel", "mlp": mlp, "mixer": {
            "left": {"heads": h, "kv_heads": g, "dim": D, "vdim": D, "mask": {"size": s["window"]}, "scale": D ** -0.5, "rot": rot},
            "right": {"heads": rh, "dim": rd, "vdim": rv, "decay": [1 - 2.0 ** -(3 + 6 * i / rh) for i in range(rh)]},
            "left_scale": 1.0, "right_scale": 1.0}}
        return {"architecture": "Sipadra", "vocab": VOCAB, "width": W, "norm": {"eps": 1e-6}, "logit_softcap": 30.0,
                "layers": [par if i % 3 == 2 else wkv for i in range(n)]}
    s = ZUVULORN_SIZES[W]
    mlp = {"kind": "moe", "expert": {"ff": s["ff"]}, "router": {"experts": EXPERTS, "top": TOP}}
    rot = {"base": 500000.0, "dims": D, "scaling": {"factor": 4.0, "low": 1.0, "high": 4.0, "original": 8192}}
    layers = []
    for i in range(n):
        kind, m = [("rglru", {"width": W, "blocks": s["blocks"], "conv": TAPS}),
                   ("channel_delta", {"heads": s["delta"], "kv_heads": s["delta"], "dim": D, "vdim": D, "conv": TAPS}),
                   ("attention", {"heads": s["attn"][0], "kv_heads": s["attn"][1], "dim": D, "vdim": D, "scale": D ** -0.5, "rot": rot})][i % 3]
        if i % 6 == 5:
            m["kv_from"] = i - 3
        layers.append({"type": kind, "mixer": m, "mlp": mlp})
    return {"architecture": "Zuvulorn", "vocab": VOCAB, "width": W, "norm": {"eps": 1e-6}, "streams": STREAMS, "layers": layers}


def shapes(c):
    """name -> shape of the model's tensors, under the names that its folder has them."""
    W, n = c["width"], c["layers"]
    if c["model"] == "gpt":
        kv = GPT_SIZES[W]["kv_heads"]
        out = {"transformer.wte.weight": (VOCAB, W), "lm_head.weight": (VOCAB, W), "resid_lambdas": (n,), "x0_lambdas": (n,),
               "smear_gate.weight": (1, 24), "smear_lambda": (1,), "backout_lambda": (1,)}
        for i in range(n):
            p = f"transformer.h.{i}."
            out.update({p + "attn.c_q.weight": (W, W), p + "attn.c_k.weight": (kv * D, W), p + "attn.c_v.weight": (kv * D, W),
                        p + "attn.c_proj.weight": (W, W), p + "mlp.c_fc.weight": (4 * W, W), p + "mlp.c_proj.weight": (W, 4 * W)})
            if i % 2 == (n - 1) % 2:
                out.update({p + "attn.ve_gate.weight": (kv, 12), f"value_embeds.{i}.weight": (VOCAB, kv * D)})
        return out
    rank = (SIPADRA_SIZES if c["model"] == "sipadra" else ZUVULORN_SIZES)[W]["rank"]
    out = {"embed": (VOCAB, W), "final.norm": (W,)}
    if c["model"] == "zuvulorn":
        out["head"] = (VOCAB, W)
    for i, layer in enumerate(design(c)["layers"]):
        m, p, mix = layer["mixer"], f"l{i}.", {}
        subs = 2
        if layer["type"] == "wkv":
            k = m["heads"] * m["dim"]
            mix = {**{"mu." + s: (W,) for s in "rkvgw"}, **{s: (k, W) for s in "rkvg"}, "w1": (rank, W), "w2": (k, rank), "w0": (k,),
                   "u": (m["heads"], m["dim"]), "norm": (k,), "o": (W, k)}
        elif layer["type"] == "parallel":
            a, b = m["left"], m["right"]
            nq, nk, k, e = a["heads"] * D, a["kv_heads"] * D, b["heads"] * b["dim"], b["heads"] * b["vdim"]
            mix = {"left.q": (nq, W), "left.k": (nk, W), "left.v": (nk, W), "left.o": (W, nq), "right.q": (k, W), "right.k": (k, W),
                   "right.v": (e, W), "right.g": (e, W), "right.norm": (e,), "right.o": (W, e)}
        elif layer["type"] == "rglru":
            k, part = m["width"], m["width"] // m["blocks"]
            mix = {"y": (k, W), "y.b": (k,), "x": (k, W), "x.b": (k,), "conv": (k, TAPS), "conv.b": (k,), "lam": (k,), "o": (W, k),
                   "ra": (m["blocks"], part, part), "ra.b": (m["blocks"], part), "ri": (m["blocks"], part, part), "ri.b": (m["blocks"], part)}
        elif layer["type"] == "attention":
            nq, nk = m["heads"] * D, m["kv_heads"] * D
            mix = {"q": (nq, W), "q.norm": (nq,), "g": (m["heads"], W), "o": (W, nq)}
            if "kv_from" not in m:
                mix.update({"k": (nk, W), "k.norm": (nk,), "v": (nk, W)})
        else:
            k = m["heads"] * D
            mix = {**{s: (k, W) for s in "qkv"}, **{s + ".conv": (k, TAPS) for s in "qkv"}, "b": (m["heads"], W), "A_log": (m["heads"],),
                   "dt_bias": (k,), "norm": (D,), "a1": (rank, W), "a2": (k, rank), "g1": (rank, W), "g2": (k, rank), "o": (W, k)}
        out.update({f"{p}mix.{k}": v for k, v in mix.items()})
        if c["model"] == "sipadra":
            ff = layer["mlp"]["ff"]
            out.update({p + "norm2": (W,), p + "mlp.gate": (ff, W), p + "mlp.up": (ff, W), p + "mlp.down": (W, ff)})
        else:
            ff = layer["mlp"]["expert"]["ff"]
            out[p + "mlp.router"] = (EXPERTS, W)
            for e in range(EXPERTS):
                out.update({f"{p}mlp.e{e}.gate": (ff, W), f"{p}mlp.e{e}.up": (ff, W), f"{p}mlp.e{e}.down": (W, ff)})
            for s in range(1, subs + 1):
                out.update({f"{p}hc{s}.in": (STREAMS,), f"{p}hc{s}.out": (STREAMS,), f"{p}hc{s}.mix": (STREAMS, STREAMS)})
        for s in range(1, subs + 1):
            out[f"{p}norm{s}"] = (W,)
    return out


def weights(c, d):
    """Random bfloat16 weights under which every part moves the logits; what writes to the residual is scaled down for the
    48 sublayers of the whole model, and a router's scores lie apart, as in a trained one."""
    out, quiet = {}, 48 ** -0.5
    for name, shape in shapes(c).items():
        z = torch.randn(shape, generator=d.gen, device="cuda")
        leaf = name.split(".", 1)[-1]
        if name in ("resid_lambdas", "x0_lambdas", "smear_lambda", "backout_lambda"):
            z = {"resid_lambdas": 1.05, "x0_lambdas": 0.1, "smear_lambda": 0.1, "backout_lambda": 0.2}[name] + 0.02 * z
        elif "norm" in leaf:
            z = 1 + 0.1 * z
        elif ".hc" in name:
            z = {"in": (1 + 0.2 * z) / STREAMS, "out": 1 + 0.2 * z, "mix": torch.eye(STREAMS, device="cuda") + 0.05 * z if z.dim() == 2 else z}[
                leaf.rsplit(".", 1)[-1]]
        elif ".mu." in name:
            z = z.sigmoid()
        elif leaf.endswith(("lam", "A_log", "dt_bias", "w0")):
            z = z - 2
        elif leaf.endswith("mlp.router"):
            z = 3 * z * shape[-1] ** -0.5
        elif len(shape) > 1 and "embed" not in name and "wte" not in name:
            z = z * shape[-1] ** -0.5
            if leaf.endswith(("mix.o", "left.o", "right.o", "down", "c_proj.weight")):
                z = z * quiet
        elif len(shape) == 1:
            z = 0.5 * z
        out[name] = z.to(BF)
    return out


def model_state(c, seed):
    """(weights, model, empty or filled cache, ids)."""
    d = Draws(seed)
    tensors = weights(c, d)
    cls = GPT if c["model"] == "gpt" else model_class(design(c)["architecture"])
    model = cls.from_dict(design(c), tensors, BF, torch.device("cuda", torch.cuda.current_device()))
    tokens = c.get("tokens", 1)
    ids = d.whole(0, VOCAB - 1, c["rows"], tokens, dtype=torch.int64)
    cache = new_cache(model, c["rows"], tokens if c["path"] == "prompt" else c["high"] + 64, BF)
    lengths = None
    if c["path"] == "step":  # as behind prompts: keys and values, states, lengths
        if c["model"] == "gpt":
            d.fill(cache.k_cache, 1.2)
            d.fill(cache.v_cache)
            cache.prev_embedding = d.normal(c["rows"], 1, c["width"])
        else:
            for key in sorted(cache.kv):
                for t in cache.kv[key]:
                    d.fill(t)
            for key in sorted(cache.state):
                d.fill(cache.state[key], 0.5)
        lengths = d.whole(c["low"], c["high"], c["rows"])
        cache.cache_seqlens.copy_(lengths)
    return dict(tensors=tensors, model=model, cache=cache, ids=ids, lengths=lengths, places=list(range(tokens)) if c.get("logits") == "all" else [tokens - 1])


def prepare(case, seed):
    path = case["path"]
    if path == "train":
        s = train_state(case, seed)
    elif path == "broadcast":
        s = broadcast_state(case, seed)
    elif path in ("prompt", "step"):
        s = model_state(case, seed)
        del s["tensors"]
        if path == "step":
            s["graphed"] = GraphedDecodeStep(s["model"], s["cache"], s["ids"])
    else:
        s = attention_state(case, seed)
    s["path"] = path
    return s


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(s):
    path = s["path"]
    if path in ("decode", "pages", "chunk"):
        y = kv_attention(s["q"], s["k"], s["v"], s["tables"], s["window"], s["cache"], 0)
        k, v = s["cache"].get_layer_cache(0)
        return dict(y=y, k=k, v=v)
    if path == "train":
        y = flash_attn.flash_attn_func(s["q"], s["k"], s["v"], causal=True, window_size=s["window"])
        dq, dk, dv = torch.autograd.grad(y, (s["q"], s["k"], s["v"]), s["grad"])
        return dict(y=y, dq=dq, dk=dk, dv=dv)
    if path == "broadcast":
        s["dst"].reset()
        s["dst"].prefill(s["src"])
        return dict(k=s["dst"].k_cache, v=s["dst"].v_cache, lengths=s["dst"].cache_seqlens)
    cache, model = s["cache"], s["model"]
    if path == "prompt":
        cache.reset()
        if len(s["places"]) > 1:
            logits = model.forward(s["ids"], kv_cache=cache)
        else:
            logits = forward_at(model, s["ids"], cache, s["places"])
    else:
        cache.cache_seqlens.copy_(s["lengths"])
        logits = s["graphed"].step(s["ids"])
    return dict(logits=logits, **kept(cache))


def kept(cache):
    """What a forward pass leaves in the cache."""
    out = {"lengths": cache.cache_seqlens}
    if hasattr(cache, "kv"):
        out["kv"] = {key: list(pair) for key, pair in cache.kv.items()}
        out["state"] = dict(cache.state)
    else:
        out["kv"] = [cache.k_cache, cache.v_cache]
    return out


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def seen(low, high, tokens, left):
    """(keys read, query-key pairs) of a row of mean length, ``tokens`` new ones; left < 0: all."""
    L = (low + high) // 2
    if left < 0 or left >= L + tokens:
        return L + tokens, tokens * L + tokens * (tokens + 1) // 2
    first = max(0, L - left)
    pairs = sum(min(L + t, left) + 1 for t in range(tokens))
    return L + tokens - first, pairs


def layer_work(c):
    """(bytes, flops) of the layers beside their weights' products, per pass: keys and values, states, pairs."""
    B, T, W, n = c["rows"], c.get("tokens", 1), c["width"], c["layers"]
    low, high = (c["low"], c["high"]) if c["path"] == "step" else (0, 0)
    nbytes = flops = 0

    def attention(heads, kv_heads, left):
        keys, pairs = seen(low, high, T, left)
        # the keys and values of a prompt are written here and need not be read back from memory
        return 4 * B * kv_heads * D * (keys if c["path"] == "step" else T), 4 * D * heads * B * pairs

    for i in range(n):
        if c["model"] == "gpt":
            s = GPT_SIZES[W]
            x = attention(s["heads"], s["kv_heads"], -1 if i == n - 1 or i % 4 == 3 else 1024)
            ve = 2 * B * T * s["kv_heads"] * D if i % 2 == (n - 1) % 2 else 0
            x = (x[0] + ve, x[1])
        elif c["model"] == "sipadra":
            s = SIPADRA_SIZES[W]
            h, dk, dv = s["right"]
            if i % 3 == 2:
                x = attention(*s["left"], s["window"] - 1)
                x = (x[0] + 8 * B * h * dk * dv, x[1] + 6 * B * T * h * dk * dv)
            else:
                x = (8 * B * s["wkv_heads"] * 64 * 64, 6 * B * T * s["wkv_heads"] * 64 * 64)
        else:
            s = ZUVULORN_SIZES[W]
            x = {0: (8 * B * W, 10 * B * T * W), 1: (8 * B * s["delta"] * D * D, 8 * B * T * s["delta"] * D * D),
                 2: attention(*s["attn"], -1)}[i % 3]
        nbytes, flops = nbytes + x[0], flops + x[1]
    return nbytes, flops


def work(case):
    c = case
    B, T = c["rows"], c.get("tokens", 1)
    if c["path"] in ("decode", "pages", "chunk"):
        H, G = c["heads"], c["kv_heads"]
        keys, pairs = seen(c["low"], c["high"], T, c["window"])
        return {"bytes": B * (4 * G * D * (keys - T) + T * (4 * H * D + 8 * G * D + 2 * D)), "flops": 4 * D * H * B * pairs}
    if c["path"] == "train":
        H, G = c["heads"], c["kv_heads"]
        return {"bytes": 2 * B * T * D * (4 * H + 4 * G), "flops": 14 * D * H * B * seen(0, 0, T, c["window"])[1]}
    if c["path"] == "broadcast":
        return {"bytes": 4 * c["layers"] * T * c["kv_heads"] * D * (1 + B), "flops": 0}
    nbytes, flops = layer_work(c)
    places = T if c.get("logits") == "all" else 1
    for name, shape in shapes(c).items():
        n = math.prod(shape)
        if "embed" in name or "wte" in name:
            if c["model"] != "sipadra" or name != "embed":
                nbytes += 2 * min(n, B * T * shape[-1]) if "value_embeds" not in name else 0
                continue
        here = B * (places if name in ("lm_head.weight", "embed", "head") else T)
        if ".e" in name and ".mlp.e" in name:  # an expert's weights are read if any token goes there, and used by its share
            nbytes += 2 * n * (1 - (1 - TOP / EXPERTS) ** (B * T))
            flops += 2 * n * here * TOP / EXPERTS
        else:
            nbytes += 2 * n
            flops += 2 * n * here if len(shape) == 2 else 2 * n / shape[0] * here * shape[0] if len(shape) == 3 else 0
    nbytes += 4 * B * places * VOCAB
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    path = case["path"]
    if path == "broadcast":
        return "exact"
    if path == "train":
        return {"rel": 1e-2, "max": 0.5}
    if path in ("prompt", "step"):
        return {"rel": 3e-2, "max": 0.9}
    return {"rel": 1e-2, "max": 0.2}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------
def exact(case, seed):
    with torch.no_grad():
        path = case["path"]
        if path in ("decode", "pages", "chunk"):
            return exact_attention(case, seed)
        if path == "train":
            return exact_train(case, seed)
        if path == "broadcast":
            return None
        return exact_model(case, seed)


def rms64(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def turn64(x, cos, sin):
    """GPT's rotation, then norm and factor: x (T, H, D) at the positions of cos / sin (T, 64)."""
    a, b = x[..., :D // 2], x[..., D // 2:]
    cos, sin = cos[:, None], sin[:, None]
    return rms64(torch.cat([a * cos + b * sin, b * cos - a * sin], -1), 2.0 ** -23) * 1.2


def hidden(first, T, n, left):
    """True where query t at position first + t does not see key j."""
    at = first + torch.arange(T, device="cuda")[:, None]
    j = torch.arange(n, device="cuda")[None]
    return (j > at) | (at - j > left) if left >= 0 else j > at


def attend64(q, k, v, first, left, sink=False, scale=D ** -0.5):
    """q (T, H, D) at positions first.., k and v (n, G, D): (T, H, D)."""
    T, H, _ = q.shape
    G = k.size(1)
    out = torch.empty_like(q)
    for t0 in range(0, T, 2048):
        mask = hidden(first + t0, min(2048, T - t0), k.size(0), left)
        for h in range(H):
            g = h // (H // G)
            s = (q[t0:t0 + 2048, h] @ k[:, g].T * scale).masked_fill_(mask, -math.inf)
            top = s.amax(1, keepdim=True)
            if sink:
                top = top.clamp(min=0)
            e = torch.exp(s - top)
            total = e.sum(1, keepdim=True)
            if sink:
                total = total + torch.exp(-top)
            out[t0:t0 + 2048, h] = e @ v[:, g] / total
    return out


def exact_attention(c, seed):
    s = attention_state(c, seed)
    cache, T = s["cache"], c.get("tokens", 1)
    cos, sin = (t[0, :, 0].double() for t in s["tables"])
    kc, vc = cache.get_layer_cache(0)
    paged = c["path"] == "pages"
    # None in the pools' place: which page a token lies in is the cache's affair
    k_out, v_out = (None, None) if paged else (kc.double(), vc.double())
    ys = []
    for b, L in enumerate(cache.cache_seqlens.tolist()):
        at = slice(L, L + T)
        q, k = (turn64(s[x][b].double(), cos[at], sin[at]) for x in "qk")
        if paged:
            pages = cache.block_table[b].long()
            old = [t[pages].flatten(0, 1)[:L].double() for t in (kc, vc)]
        else:
            old = [t[b, :L].double() for t in (kc, vc)]
            k_out[b, at], v_out[b, at] = k, s["v"][b].double()
        # a new key is read back in the type that the cache has
        ys.append(attend64(q, torch.cat([old[0], k]), torch.cat([old[1], s["v"][b].double()]), L, c["window"]))
    return dict(y=torch.stack(ys), k=k_out, v=v_out)


def exact_train(c, seed):
    s = train_state(c, seed)
    H, G, T = c["heads"], c["kv_heads"], c["tokens"]
    q, k, v, do = (s[x].detach().double() for x in ("q", "k", "v", "grad"))
    y, dq, dk, dv = (torch.zeros_like(x) for x in (q, q, k, v))
    mask, scale = hidden(0, T, T, c["window"]), D ** -0.5
    for b in range(c["rows"]):
        for h in range(H):
            g = h // (H // G)
            p = torch.softmax((q[b, :, h] @ k[b, :, g].T * scale).masked_fill_(mask, -math.inf), 1)
            y[b, :, h] = p @ v[b, :, g]
            dp = do[b, :, h] @ v[b, :, g].T
            ds = p * (dp - (do[b, :, h] * y[b, :, h]).sum(-1, keepdim=True)) * scale
            dq[b, :, h] = ds @ k[b, :, g]
            dk[b, :, g] += ds.T @ q[b, :, h]
            dv[b, :, g] += p.T @ do[b, :, h]
    return dict(y=y, dq=dq, dk=dk, dv=dv)


class Wide:
    """The model's tensors in 64 bits, one at a time."""

    def __init__(self, tensors, prefix=""):
        self.tensors, self.prefix = tensors, prefix

    def __getitem__(self, name):
        return self.tensors[self.prefix + name].double()

    def __contains__(self, name):
        return self.prefix + name in self.tensors

    def under(self, prefix):
        return Wide(self.tensors, self.prefix + prefix)


def exact_model(c, seed):
    s = model_state(c, seed)
    w, cache, ids = Wide(s["tensors"]), s["cache"], s["ids"]
    s["model"] = None
    first = s["lengths"].tolist() if s["lengths"] is not None else [0] * c["rows"]
    left = {}  # what the pass leaves in the cache's states; the new keys and values show in the logits
    logits = {"gpt": gpt64, "sipadra": sipadra64, "zuvulorn": zuvulorn64}[c["model"]](c, w, cache, ids, first, s["places"], left)
    if c["path"] == "step":
        logits = logits[:, -1]
    return dict(logits=logits, lengths=None, kv=None, **({"state": left} if left else {}))


def over_cache(c, q, k, v, kept_kv, first, left, sink=False):
    """Attention of the new tokens (B, T, H, D), (B, T, G, D) behind what the cache's rows hold."""
    out = []
    for b, L in enumerate(first):
        old_k, old_v = (t[b, :L].double() for t in kept_kv)
        out.append(attend64(q[b], torch.cat([old_k, k[b]]), torch.cat([old_v, v[b]]), L, left, sink))
    return torch.stack(out)


def gpt64(c, w, cache, ids, first, places, states):
    B, T, W, n = c["rows"], c.get("tokens", 1), c["width"], c["layers"]
    s, eps = GPT_SIZES[W], 2.0 ** -23
    cos, sin = (t[0, :, 0].double() for t in rotary(max(first) + T))
    x = rms64(w.tensors["transformer.wte.weight"][ids].double(), eps)
    lam, gate_w = w["smear_lambda"], w["smear_gate.weight"]
    if T > 1:
        x = torch.cat([x[:, :1], x[:, 1:] + lam * torch.sigmoid(x[:, 1:, :24] @ gate_w.T) * x[:, :-1]], 1)
    else:
        x = x + lam * torch.sigmoid(x[..., :24] @ gate_w.T) * cache.prev_embedding.double()
    x0, saved = x, None
    resid, x0l = w["resid_lambdas"], w["x0_lambdas"]
    for i in range(n):
        p = w.under(f"transformer.h.{i}.")
        x = resid[i] * x + x0l[i] * x0
        h = rms64(x, eps)
        q, k, v = ((h @ p[f"attn.c_{t}.weight"].T).view(B, T, -1, D) for t in "qkv")
        if f"value_embeds.{i}.weight" in w:
            gate = 3 * torch.sigmoid(h[..., :12] @ p["attn.ve_gate.weight"].T)
            v = v + gate[..., None] * w.tensors[f"value_embeds.{i}.weight"][ids].double().view(v.shape)
        at = [slice(L, L + T) for L in first]
        q = torch.stack([turn64(q[b], cos[at[b]], sin[at[b]]) for b in range(B)])
        k = torch.stack([turn64(k[b], cos[at[b]], sin[at[b]]) for b in range(B)])
        left = 4096 if i == n - 1 or i % 4 == 3 else 1024
        y = over_cache(c, q, k, v, (cache.k_cache[i], cache.v_cache[i]), first, left)
        x = x + y.reshape(B, T, W) @ p["attn.c_proj.weight"].T
        x = x + torch.relu(rms64(x, eps) @ p["mlp.c_fc.weight"].T).square() @ p["mlp.c_proj.weight"].T
        if i == n // 2:
            saved = x
    x = rms64(x - w["backout_lambda"] * saved, eps)[:, places]
    return 15 * torch.tanh(x @ w["lm_head.weight"].T / 15)


def yarn_angles(length, rot):
    """(angles (length, 64), amplitude) of Sipadra's rotation."""
    s, base, i = rot["scaling"], rot["base"], torch.arange(D // 2, dtype=F64, device="cuda")
    freq = base ** (-2 * i / D)

    def pair_of(turns):
        return D * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(pair_of(s["fast"])), 0), min(math.ceil(pair_of(s["slow"])), D - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    freq = freq / s["factor"] * ramp + freq * (1 - ramp)
    return torch.outer(torch.arange(length, dtype=F64, device="cuda"), freq), 0.1 * math.log(s["factor"]) + 1


def banded_angles(length, rot):
    """(angles (length, 64), amplitude) of Zuvulorn's rotation."""
    s = rot["scaling"]
    freq = rot["base"] ** (-2 * torch.arange(D // 2, dtype=F64, device="cuda") / D)
    keep = ((s["original"] * freq / (2 * math.pi) - s["low"]) / (s["high"] - s["low"])).clamp(0, 1)
    freq = keep * freq + (1 - keep) * freq / s["factor"]
    return torch.outer(torch.arange(length, dtype=F64, device="cuda"), freq), 1.0


def turned(x, angles, amplitude, first):
    """x (B, T, H, D) rotated, row b from position first[b] on."""
    T = x.size(1)
    a = torch.stack([angles[L:L + T] for L in first])[:, :, None]
    cos, sin = a.cos() * amplitude, a.sin() * amplitude
    u, v = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)


def sipadra64(c, w, cache, ids, first, places, states):
    B, T, eps = c["rows"], c.get("tokens", 1), 1e-6
    x = w.tensors["embed"][ids].double()
    for i, layer in enumerate(design(c)["layers"]):
        p, m = w.under(f"l{i}.mix."), layer["mixer"]
        if layer["type"] == "wkv":
            h, d = m["heads"], m["dim"]
            shifted = torch.cat([cache.state[f"l{i}.wkv.shift"].double()[:, None], x[:, :-1]], 1)
            mix = {s: x + (shifted - x) * p["mu." + s] for s in "rkvgw"}
            r, k, v = ((mix[s] @ p[s].T).view(B, T, h, d) for s in "rkv")
            g = torch.exp(-torch.exp(torch.tanh(mix["w"] @ p["w1"].T) @ p["w2"].T + p["w0"])).view(B, T, h, d)
            S, o, u = cache.state[f"l{i}.wkv"].double(), torch.empty_like(v), p["u"]
            for t in range(T):
                kv = k[:, t, :, :, None] * v[:, t, :, None]
                o[:, t] = torch.einsum("bhde,bhd->bhe", S + u[..., None] * kv, r[:, t])
                S = g[:, t, :, :, None] * S + kv
            states.update({f"l{i}.wkv": S, f"l{i}.wkv.shift": x[:, -1]})
            y = (rms64(o, eps).flatten(2) * p["norm"] * F.silu(mix["g"] @ p["g"].T)) @ p["o"].T
        else:
            a, b, pl, pr = m["left"], m["right"], p.under("left."), p.under("right.")
            angles, amp = yarn_angles(max(first) + T, a["rot"])
            q, k, v = ((x @ pl[s].T).view(B, T, -1, D) for s in "qkv")
            q, k = (rms64(turned(z, angles, amp, first), eps) for z in (q, k))
            left = over_cache(c, q, k, v, cache.kv[f"l{i}.left"], first, a["mask"]["size"] - 1).flatten(2) @ pl["o"].T
            q, k, v = (F.silu(x @ pr[s].T).view(B, T, b["heads"], -1) for s in "qkv")
            S, o = cache.state[f"l{i}.right"].double(), torch.empty_like(v)
            decay = torch.tensor(b["decay"], dtype=F64, device="cuda")[:, None, None]
            for t in range(T):
                S = decay * S + k[:, t, :, :, None] * v[:, t, :, None]
                o[:, t] = torch.einsum("bhde,bhd->bhe", S, q[:, t])
            states[f"l{i}.right"] = S
            y = left + (rms64(o.flatten(2), eps) * pr["norm"] * torch.sigmoid(x @ pr["g"].T)) @ pr["o"].T
        p = w.under(f"l{i}.")
        x = x + rms64(y, eps) * p["norm1"]
        y = (F.silu(x @ p["mlp.gate"].T) * (x @ p["mlp.up"].T)) @ p["mlp.down"].T
        x = x + rms64(y, eps) * p["norm2"]
    logits = rms64(x[:, places], eps) * w["final.norm"] @ w["embed"].T
    return logits.div_(30).tanh_().mul_(30)


def conv64(x, carry, taps, bias=0):
    """x (B, T, C), carry (B, K - 1, C) the inputs before, taps (C, K); (outputs, the new carry)."""
    z = torch.cat([carry.double(), x], 1)
    return z[:, 1 - TAPS:], sum(z[:, j:j + x.size(1)] * taps[:, j] for j in range(TAPS)) + bias


def zuvulorn64(c, w, cache, ids, first, places, states):
    B, T, W, eps = c["rows"], c.get("tokens", 1), c["width"], 1e-6
    streams = w.tensors["embed"][ids].double()[..., None, :].expand(B, T, STREAMS, W)
    keys = {}

    def norm(u, weight):
        u = u - u.mean(-1, keepdim=True)
        return rms64(u, eps) * weight

    def rglru(p, h, m, key):
        y = F.gelu(h @ p["y"].T + p["y.b"], approximate="tanh")
        states[key + ".conv"], u = conv64(h @ p["x"].T + p["x.b"], cache.state[key + ".conv"], p["conv"], p["conv.b"])
        part = u.view(B, T, m["blocks"], -1)
        r, i = (torch.sigmoid(torch.einsum("bij,ntbj->ntbi", p[s], part) + p[s + ".b"]).reshape(u.shape) for s in ("ra", "ri"))
        log_a = -8 * r * F.softplus(p["lam"])
        a, drive = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * i * u
        S, o = cache.state[key].double(), torch.empty_like(u)
        for t in range(T):
            S = a[:, t] * S + drive[:, t]
            o[:, t] = S
        states[key] = S
        return (o * y) @ p["o"].T

    def attention(p, h, m, key):
        angles, amp = banded_angles(max(first) + T, m["rot"])
        q = turned((rms64(h @ p["q"].T, eps) * p["q.norm"]).view(B, T, -1, D), angles, amp, first)
        source = key
        if "kv_from" in m:
            source = f"l{m['kv_from']}.attention"
        else:
            k = turned((rms64(h @ p["k"].T, eps) * p["k.norm"]).view(B, T, -1, D), angles, amp, first)
            keys[key] = k, (h @ p["v"].T).view(B, T, -1, D)
        o = over_cache(c, q, *keys[source], cache.kv[source], first, -1, sink=True)
        return (o * torch.sigmoid(h @ p["g"].T)[..., None]).flatten(2) @ p["o"].T

    def delta(p, h, m, key):
        H = m["heads"]
        taps = torch.cat([p[s + ".conv"] for s in "qkv"])
        states[key + ".conv"], z = conv64(h @ torch.cat([p[s] for s in "qkv"]).T, cache.state[key + ".conv"], taps)
        q, k, v = F.silu(z).view(B, T, 3, H, D).unbind(2)
        q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        beta = torch.sigmoid(h @ p["b"].T)
        rate = F.softplus(h @ p["a1"].T @ p["a2"].T + p["dt_bias"]).view(B, T, H, D)
        g = torch.exp(-torch.exp(p["A_log"])[:, None] * rate)
        S, o = cache.state[key].double(), torch.empty_like(v)
        for t in range(T):
            S = g[:, t, :, :, None] * S
            u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhde,bhd->bhe", S, k[:, t]))
            S = S + k[:, t, :, :, None] * u[:, :, None]
            o[:, t] = torch.einsum("bhde,bhd->bhe", S, q[:, t]) * D ** -0.5
        states[key] = S
        gate = torch.sigmoid(h @ p["g1"].T @ p["g2"].T).view(o.shape)
        return (rms64(o, eps) * p["norm"] * gate).flatten(2) @ p["o"].T

    def experts(p, h):
        h = h.flatten(0, 1)
        score, pick = torch.sigmoid(h @ p["router"].T).topk(TOP, 1)
        out = torch.zeros_like(h)
        for e in range(EXPERTS):
            row, slot = (pick == e).nonzero(as_tuple=True)
            z = score[row, slot, None] * h[row]
            out.index_add_(0, row, (F.silu(z @ p[f"e{e}.gate"].T) * (z @ p[f"e{e}.up"].T)) @ p[f"e{e}.down"].T)
        return out.view(B, T, W)

    def through(x, p, s, norm_weight, sublayer):
        y = sublayer(norm(torch.einsum("btsw,s->btw", x, p[f"hc{s}.in"]), norm_weight))
        return torch.einsum("btsw,su->btuw", x, p[f"hc{s}.mix"]) + p[f"hc{s}.out"][:, None] * y[:, :, None]

    for i, layer in enumerate(design(c)["layers"]):
        p, kind = w.under(f"l{i}."), layer["type"]
        mixer = {"rglru": rglru, "attention": attention, "channel_delta": delta}[kind]
        streams = through(streams, p, 1, p["norm1"], lambda h: mixer(p.under("mix."), h, layer["mixer"], f"l{i}.{kind}"))
        streams = through(streams, p, 2, p["norm2"], lambda h: experts(p.under("mlp."), h))
    return norm(streams.sum(2)[:, places], w["final.norm"]) @ w["head"].T
