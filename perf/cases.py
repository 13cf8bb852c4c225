"""The work users have this package do, as cases that can be timed.

A case is a plain dict.  Its ``kind`` names one way of using the package:

``step``     one decode step of attention on a filled cache: a query of every sequence against
             all stored tokens, layer after layer (``KVContext.decode``), or through the
             reference's cache class for one layer and one sequence
             (``TurboQuantKVCache.fused_decode``, ``"api": "cache"``).
``prompt``   a prompt enters an empty cache and its first token is attended: ``clear``,
             ``append`` of all tokens at once, ``decode``.
``turn``     a short conversation turn: a prompt, then token by token ``append`` + ``decode``.
``read``     the dequantised keys and values of a token range (``KVContext.dequant``): what the
             dense fallbacks of the model adapters attend.
``paged``    an engine's paged tensor saved under a request id and restored into other pages
             (``DeviceBlockStore.save_paged`` / ``load_into_paged``).
``handoff``  one cache moved to another context through its wire format (``export_state`` /
             ``import_state``): host bytes by nature.

Keys and values are what the benchmark draws: standard normal times a per-channel log-normal
scale, with 3 of 128 key channels per head a further x20; queries are standard normal.
"""

import math

import numpy as np
import torch

from turboquant_pro_b200 import KVContext, TurboQuantKVCache
from turboquant_pro_b200.connector import DeviceBlockStore

D = 128
WINDOW, BLOCK = 512, 256        # tokens kept uncompressed; tokens of a compressed block
PAGE_TOKENS = 16                # tokens per page of the engine's paged tensor
DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}

# (KV heads, query heads, value bits) of the geometries the configurations and the model table
# name: multi-head, Llama-3-8B / Mistral-7B, Llama-3-70B, Gemma-2-27B, Qwen2.5-7B
SHAPES = {"mha": (32, 32, 4), "8b": (8, 32, 3), "70b": (8, 64, 4), "27b": (16, 32, 3),
          "7b": (4, 28, 3)}


def _case(kind, shape, tokens, *, name=None, batch=1, low=0, layers=1, dtype="float16", steps=0,
          api="context", bits=None, order="bthd"):
    h, hq, vb = SHAPES[shape]
    c = {"kind": kind, "heads": h, "q_heads": hq, "value_bits": bits or vb, "tokens": tokens,
         "low": low or tokens, "batch": batch, "layers": layers, "dtype": dtype, "steps": steps,
         "api": api, "order": order}
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one layer of a single user's multi-head cache, float32 as the cache class defaults to:
        # the smallest call, launches and latency
        _case("step", "mha", 4096, name="step_mha_4k_f32", dtype="float32", api="cache"),
        # a serving batch of the 8B model at its full context: the headline workload
        _case("step", "8b", 8192, name="step_8b_b32_8k", batch=32, layers=2),
        # one very long document
        _case("step", "8b", 131072, name="step_8b_b1_128k", layers=2, dtype="bfloat16"),
        # a large batch of requests of every length, eight query heads per KV head
        _case("step", "70b", 32768, name="step_70b_b64_ragged", batch=64, low=1024),
        # seven query heads per KV head, ragged batch
        _case("step", "7b", 12000, name="step_7b_b16_ragged", batch=16, low=700, layers=2,
              dtype="bfloat16"),
        # a chat turn of a few users: prompt, then tokens one by one (the last of them flush a block)
        _case("turn", "8b", 1010, name="turn_8b_b4", batch=4, layers=2, steps=24,
              dtype="bfloat16", order="bhtd"),
        # a batch of long prompts
        _case("prompt", "8b", 16384, name="prompt_8b_b8_16k", batch=8),
        # one prompt through the cache class, float32 tokens, odd length
        _case("prompt", "mha", 4001, name="prompt_mha_4k_f32", dtype="float32", api="cache"),
        # dense keys and values of one sequence, as the adapters' fallbacks read them
        _case("read", "8b", 8000, name="read_8b_8k", dtype="bfloat16"),
        # an engine stores a request and restores it elsewhere
        _case("paged", "8b", 3333, name="paged_8b_3k", layers=2, dtype="bfloat16", bits=4),
        # a request leaves for another worker
        _case("handoff", "8b", 2100, name="handoff_8b_2k"),
    ]


def _spread(rng, low, high):
    """A whole number of [low, high], even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "prompt", "prompt", "turn", "read", "paged",
                       "handoff"])
    shape = rng.choice(list(SHAPES))
    h = SHAPES[shape][0]
    dtype = rng.choice(["float16", "float16", "bfloat16", "bfloat16", "float32"])
    bits = rng.choice([3, 4])
    if kind == "step":
        tokens = _spread(rng, 40, 131072)
        batch = _spread(rng, 1, max(1, min(64, 4_000_000 // (tokens * h))))
        if rng.random() < 0.15:
            return _case("step", "mha", min(tokens, 16384), dtype="float32", api="cache")
        low = max(1, tokens // rng.choice([1, 2, 20]))
        return _case("step", shape, tokens, batch=batch, low=low, dtype=dtype, bits=bits,
                     layers=rng.choice([1, 2]))
    if kind == "prompt":
        tokens = _spread(rng, 100, 16384)
        if rng.random() < 0.25:
            return _case("prompt", "mha", min(tokens, 8192), dtype="float32", api="cache")
        batch = _spread(rng, 1, max(1, min(16, 900_000 // (tokens * h))))
        return _case("prompt", shape, tokens, batch=batch, dtype=dtype, bits=bits,
                     order=rng.choice(["bthd", "bhtd"]))
    if kind == "turn":
        return _case("turn", shape, _spread(rng, 20, 2000), batch=rng.randint(1, 8), layers=2,
                     steps=rng.randint(8, 24), dtype=dtype, bits=bits,
                     order=rng.choice(["bthd", "bhtd"]))
    if kind == "read":
        return _case("read", shape, _spread(rng, 300, 16384 if h <= 8 else 6000), dtype=dtype,
                     bits=bits)
    if kind == "paged":
        return _case("paged", shape, _spread(rng, 300, 8000 if h <= 8 else 3000), layers=2,
                     dtype=dtype, bits=bits)
    return _case("handoff", shape, _spread(rng, 530, 2500 if h <= 8 else 1100), dtype=dtype,
                 bits=bits)


# ---- inputs --------------------------------------------------------------------------------
class _Source:
    """Tokens of one model from a seed: fixed channel scales, fresh normals."""

    def __init__(self, seed, heads, dtype):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(int(seed) * 7919 + 17)
        self.dtype = dtype
        self.sk = torch.exp(0.5 * self.normal((heads, D), torch.float32))
        self.sv = torch.exp(0.5 * self.normal((heads, D), torch.float32))
        wide = torch.rand((heads, D), generator=self.gen, device="cuda").argsort(dim=1)[:, :3]
        self.sk.scatter_(1, wide, 20.0 * self.sk.gather(1, wide))

    def normal(self, shape, dtype=None):
        return torch.randn(shape, generator=self.gen, device="cuda", dtype=dtype or self.dtype)

    def tokens(self, batch, n):
        """Keys and values ``[batch, n, heads, D]``."""
        h = self.sk.shape[0]
        k = self.normal((batch, n, h, D)).mul_(self.sk.to(self.dtype))
        v = self.normal((batch, n, h, D)).mul_(self.sv.to(self.dtype))
        return k, v


def _ordered(t, order):
    """``[B, T, H, D]`` as a model hands it over: as it is, or a view of ``[B, H, T, D]``."""
    return t if order == "bthd" else t.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)


def _lengths(case):
    """Tokens of every sequence: evenly spread over [low, tokens] in a scattered order."""
    b, lo, hi = case["batch"], case["low"], case["tokens"]
    if lo == hi:
        return [hi] * b
    order = sorted(range(b), key=lambda i: (i * 0.6180339887) % 1.0)
    return [lo + int((hi - lo) * (order[i] + 0.5) / b) for i in range(b)]


def _context(case, max_tokens):
    return KVContext(n_layers=case["layers"], n_seqs=case["batch"],
                     n_kv_heads=case["heads"], n_q_heads=case["q_heads"],
                     value_bits=case["value_bits"], hot_window=WINDOW,
                     max_tokens_per_seq=max_tokens, kv_dtype=case["dtype"], seed=0)


def _fill(ctx, case, src, chunk_values=1 << 26):
    """Every sequence of every layer to its length, in appends of a bounded size."""
    lens = _lengths(case)
    groups = [(0, case["batch"], lens[0])] if len(set(lens)) == 1 else \
        [(i, 1, n) for i, n in enumerate(lens)]
    for layer in range(ctx.n_layers):
        for s0, b, n in groups:
            step = max(BLOCK, chunk_values // (b * case["heads"] * D))
            for t in range(0, n, step):
                k, v = src.tokens(b, min(step, n - t))
                ctx.append(layer, k, v, seq_begin=s0)


def _cache(case):
    return TurboQuantKVCache.robust(head_dim=D, n_heads=case["heads"],
                                    value_bits=case["value_bits"], hot_window=WINDOW,
                                    max_tokens=case["tokens"] + 1, dtype=case["dtype"],
                                    n_q_heads=case["q_heads"], seed=0)


def prepare(case, seed):
    kind, h, hq, n = case["kind"], case["heads"], case["q_heads"], case["tokens"]
    dtype, layers, batch = DTYPES[case["dtype"]], case["layers"], case["batch"]
    src = _Source(seed, h, dtype)
    s = {"case": case}
    if case["api"] == "cache":
        s["cache"] = _cache(case)
        s["q"] = src.normal((hq, D))
        k, v = src.tokens(1, n)
        if kind == "step":
            s["cache"].append_many(k[0], v[0])
        else:
            s["k"], s["v"] = k[0], v[0]
        return s
    q_dtype = torch.bfloat16 if dtype == torch.float16 else dtype
    if kind == "step":
        s["ctx"] = _context(case, n)
        _fill(s["ctx"], case, src)
        s["q"] = src.normal((layers, batch, hq, D), q_dtype)
    elif kind == "prompt":
        s["ctx"] = _context(case, n + 1)
        s["k"], s["v"] = (_ordered(t, case["order"]) for t in src.tokens(batch, n))
        s["q"] = src.normal((layers, batch, hq, D), q_dtype)
    elif kind == "turn":
        steps = case["steps"]
        s["ctx"] = _context(case, n + steps)
        s["prompt"] = [[_ordered(t, case["order"]) for t in src.tokens(batch, n)]
                       for _ in range(layers)]
        s["token"] = [[[_ordered(t, case["order"]) for t in src.tokens(batch, 1)]
                       for _ in range(layers)] for _ in range(steps)]
        s["q"] = src.normal((steps, layers, batch, hq, D), q_dtype)
        s["out"] = torch.empty((steps, layers, batch, hq, D), device="cuda")
    elif kind == "read":
        s["ctx"] = _context(case, n)
        _fill(s["ctx"], case, src)
    elif kind == "paged":
        s["store"] = DeviceBlockStore(layers, h, n_q_heads=hq, max_requests=2, max_tokens=n,
                                      value_bits=case["value_bits"], hot_window=WINDOW,
                                      dtype=case["dtype"], seed=0)
        need = -(-n // PAGE_TOKENS)
        s["from"], s["to"] = [], []
        for _ in range(layers):
            k, v = src.tokens(need + 3, PAGE_TOKENS)
            s["from"].append(torch.stack([k, v]))
            s["to"].append(torch.zeros_like(s["from"][-1]))
        s["tables"] = [torch.randperm(need + 3, generator=src.gen, device="cuda")[:need].int()
                       for _ in range(2)]
    else:
        s["ctx"] = _context(case, n)
        _fill(s["ctx"], case, src)
        s["other"] = _context(case, n)
        s["message_bytes"] = int(1.1 * h * _stored_bytes(case, n)) + (1 << 16)
    return s


# ---- one pass ------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind, layers, n = case["kind"], case["layers"], case["tokens"]
    if case["api"] == "cache":
        if kind == "prompt":
            s["cache"].clear()
            s["cache"].append_many(s["k"], s["v"])
        return s["cache"].fused_decode(s["q"])
    if kind == "step":
        return [s["ctx"].decode(layer, s["q"][layer]) for layer in range(layers)]
    if kind == "prompt":
        ctx = s["ctx"]
        ctx.clear(0)
        ctx.append(0, s["k"], s["v"])
        return ctx.decode(0, s["q"][0])
    if kind == "turn":
        ctx = s["ctx"]
        for layer in range(layers):
            ctx.clear(layer)
            ctx.append(layer, *s["prompt"][layer])
        for i in range(case["steps"]):
            for layer in range(layers):
                ctx.append(layer, *s["token"][i][layer])
                ctx.decode(layer, s["q"][i, layer], out=s["out"][i, layer])
        return s["out"]
    if kind == "read":
        return [s["ctx"].dequant(layer, 0, 0, n) for layer in range(layers)]
    if kind == "paged":
        for layer in range(layers):
            s["store"].save_paged("request", f"model.layers.{layer}.attn", s["from"][layer],
                                  s["tables"][0], n)
        for layer in range(layers):
            s["store"].load_into_paged("request", f"model.layers.{layer}.attn", s["to"][layer],
                                       s["tables"][1])
        return s["to"]
    moved = s["ctx"].export_state(0, 0)
    s["other"].import_state(0, 0, moved)
    # the blocks as one message of a fixed size (ties make the side-lists a little longer or shorter)
    message = b"".join(moved["blocks"]).ljust(s["message_bytes"], b"\0")
    return [np.frombuffer(message, dtype=np.uint8), moved["hot_k"], moved["hot_v"],
            s["other"].dequant(0, 0, 0, n)]


# ---- what a pass cannot do without -----------------------------------------------------------
def _stored_bytes(case, n):
    """Bytes of one cached sequence of one KV head: compressed blocks and the window."""
    blocks = 0 if n <= WINDOW else 1 + (n - WINDOW - 1) // BLOCK
    elem = 4 if case["dtype"] == "float32" else 2
    block = BLOCK * D * (4 + case["value_bits"]) // 8 + 4 * BLOCK + 8 * D + 6 * 5 * D
    return blocks * block + 2 * (n - blocks * BLOCK) * D * elem


def work(case):
    kind, h, hq, layers = case["kind"], case["heads"], case["q_heads"], case["layers"]
    n, batch = case["tokens"], case["batch"]
    elem = 4 if case["dtype"] == "float32" else 2
    raw = 2 * D * elem                     # key and value of one token of one head
    rotate = 2 * D * D                     # multiply-adds of one value's rotation, as operations

    def attend(lens):                      # one decode of one layer
        return (sum(h * _stored_bytes(case, m) for m in lens) + len(lens) * hq * D * (elem + 4),
                sum(4 * hq * D * m for m in lens))

    if kind == "step":
        b, f = attend(_lengths(case))
    elif kind == "prompt":
        b, f = attend([n] * batch)
        b += batch * h * (n * raw + _stored_bytes(case, n))
        f += batch * h * n * rotate
    elif kind == "turn":
        b = batch * h * (n * raw + _stored_bytes(case, n))
        f = batch * h * n * rotate
        for i in range(1, case["steps"] + 1):
            db, df = attend([n + i] * batch)
            b, f = b + db + 2 * batch * h * raw, f + df
    elif kind == "read":
        b, f = h * (_stored_bytes(case, n) + 8 * D * n), h * n * rotate
    elif kind == "paged":
        b, f = h * (2 * n * raw + 2 * _stored_bytes(case, n)), 2 * h * n * rotate
    else:
        b, f = h * (4 * _stored_bytes(case, n) + 8 * D * n), h * n * rotate
    return {"bytes": layers * b, "flops": layers * f}


def tolerance(case):
    # What is stored is exact.  Attention multiplies fp16 operands (11-bit tables, weights and
    # probabilities) with float32 sums; a score of magnitude 10 carries that rounding into the
    # exponent.
    return {"rel": 3e-3} if case["kind"] in ("step", "prompt", "turn") else "exact"
