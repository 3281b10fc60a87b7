"""Performance cases of the attention path: what a program built on `hy3_b200.Hy3Attn` has it do, over the sizes, cache types
and batch shapes it is used with.

Two kinds of pass, each through the public entry points in the order a generation loop calls them:

  decode   one new token per sequence: `batch_set` for the step, then `decode_step` for every layer (eagerly, as
           `EvalSession` walks a token, or as one captured CUDA graph replayed per token, as the benchmark does);
  prefill  a run of new tokens on top of a cached prefix, in chunks: per chunk `batch_set`, then per layer `append` (queries
           out as fp16) and `prefill`.

A pass always works at the same positions: the new token's slot (or the chunk's slots) is written again, as after a
rolled-back cache length, so that a pass can be repeated on the same state.
"""
import math

import numpy as np
import torch

from hy3_b200 import D, G, H, Hy3Attn

KV_BYTES_PER_TOKEN_HEAD = {"fp16": 512, "int8": 260, "int4": 132}   # K and V of one token and KV head: codes + fp16 scales


def listed():
    return [
        # configuration "single-layer decode over 4096 positions", FP16 cache: the smallest call, one layer of one token, latency only
        {"name": "decode_fp16_b1_4096_1layer", "kind": "decode", "kv": "fp16", "layers": 1, "batch": 1, "lo": 4096, "hi": 4096, "heads": 8, "yarn": False, "graph": False},
        # a token early in a conversation (default INT8 cache, all 80 layers, layer by layer from the host): launches and latency
        {"name": "decode_int8_b1_700_80layers", "kind": "decode", "kv": "int8", "layers": 80, "batch": 1, "lo": 700, "hi": 700, "heads": 8, "yarn": False, "graph": False},
        # the benchmark's headline: INT8 cache, batch 1, 80 layer caches of 32768 positions, one graph per token
        {"name": "decode_int8_b1_32768_80layers", "kind": "decode", "kv": "int8", "layers": 80, "batch": 1, "lo": 32768, "hi": 32768, "heads": 8, "yarn": False, "graph": True},
        # the same shape with an FP16 cache, 16 layer caches
        {"name": "decode_fp16_b1_32768_16layers", "kind": "decode", "kv": "fp16", "layers": 16, "batch": 1, "lo": 32768, "hi": 32768, "heads": 8, "yarn": False, "graph": True},
        # long context: INT4 cache, YaRN factor 4, 262144 positions, 4 layer caches
        {"name": "decode_int4_b1_262144_4layers", "kind": "decode", "kv": "int4", "layers": 4, "batch": 1, "lo": 262144, "hi": 262144, "heads": 8, "yarn": True, "graph": False},
        # a small server: 8 conversations of a few thousand tokens, INT4 cache, 8 layers
        {"name": "decode_int4_b8_ragged_8layers", "kind": "decode", "kv": "int4", "layers": 8, "batch": 8, "lo": 300, "hi": 8000, "heads": 8, "yarn": False, "graph": False},
        # batched serving: 64 sequences with lengths uniform in [1024, 65536], INT8 cache, one layer (4.3 GB per call)
        {"name": "decode_int8_b64_ragged_1layer", "kind": "decode", "kv": "int8", "layers": 1, "batch": 64, "lo": 1024, "hi": 65536, "heads": 8, "yarn": False, "graph": False},
        # the same batch as one of 8 GPUs sees it when the KV heads are split: one KV head per GPU
        {"name": "decode_int8_b64_ragged_1head", "kind": "decode", "kv": "int8", "layers": 1, "batch": 64, "lo": 1024, "hi": 65536, "heads": 1, "yarn": False, "graph": False},
        # a short question in a running conversation: 45 new tokens on a history of 1001, INT8 cache, 16 layers
        {"name": "prefill_int8_45_on_1001_16layers", "kind": "prefill", "kv": "int8", "layers": 16, "prefix": 1001, "new": 45, "chunk": 512},
        # multi-turn: 1024 new tokens on a cached prefix of 4096, chunks of 512, INT8 cache
        {"name": "prefill_int8_1024_on_4096_4layers", "kind": "prefill", "kv": "int8", "layers": 4, "prefix": 4096, "new": 1024, "chunk": 512},
        # a fresh prompt of an odd length in the largest chunks the backend takes, INT4 cache
        {"name": "prefill_int4_3001_chunk2048_2layers", "kind": "prefill", "kv": "int4", "layers": 2, "prefix": 0, "new": 3001, "chunk": 2048},
        # a fresh long prompt: 8192 tokens in 512-token chunks, FP16 cache
        {"name": "prefill_fp16_8192_chunk512_2layers", "kind": "prefill", "kv": "fp16", "layers": 2, "prefix": 0, "new": 8192, "chunk": 512},
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kv = rng.choice(["fp16", "int8", "int8", "int4"])
    if rng.random() < 0.6:
        batch = rng.choice([1, 1, 1, _log_int(rng, 2, 64)])
        heads = rng.choice([8, 8, 8, 8, 4, 2, 1])
        hi = _log_int(rng, 128, 262144 if batch == 1 else 65536)
        lo = hi if batch == 1 else max(1, int(hi * rng.uniform(0.02, 1.0)))
        # a call's caches stay below 4 GB, the sequence lengths being what is spread
        per_layer = batch * (lo + hi) / 2 * heads * KV_BYTES_PER_TOKEN_HEAD[kv]
        if per_layer > 4e9:
            hi = max(128, int(hi * 4e9 / per_layer))
            lo = max(1, min(lo, hi))
            per_layer = batch * (lo + hi) / 2 * heads * KV_BYTES_PER_TOKEN_HEAD[kv]
        layers = min(_log_int(rng, 1, 80), max(1, int(4e9 / per_layer)))
        return {"kind": "decode", "kv": kv, "layers": layers, "batch": batch, "lo": lo, "hi": hi, "heads": heads,
                "yarn": rng.random() < 0.25, "graph": rng.random() < 0.3}
    new = _log_int(rng, 2, 8192)
    prefix = rng.choice([0, _log_int(rng, 16, 16384)])
    chunk = rng.choice([256, 512, 512, 1000, 2048])
    # no more than 2e12 operations and 1.5 GB of rows
    flops = _prefill_flops({"prefix": prefix, "new": new, "layers": 1})
    if flops > 2e12:
        prefix = max(0, min(prefix, int(2e12 / (4.0 * D * H * new) - new / 2)))
        flops = _prefill_flops({"prefix": prefix, "new": new, "layers": 1})
    layers = min(_log_int(rng, 1, 32), max(1, int(2e12 / flops)), max(1, 16384 // new))
    return {"kind": "prefill", "kv": kv, "layers": layers, "prefix": prefix, "new": new, "chunk": chunk}


def _lengths(case):
    """Tokens in each sequence's cache before the step (a function of the case alone)."""
    if case["batch"] == 1:
        return [case["hi"]]
    rng = np.random.default_rng(case["batch"] * 1000003 + case["hi"])
    return [int(x) for x in rng.integers(case["lo"], case["hi"] + 1, case["batch"])]


def _yarn4():
    """A YaRN table with factor 4, every frequency interpolated."""
    inv = (1.0 / (11158840.0 ** (np.arange(64) / 64.0))).astype(np.float32)
    return inv / 4.0, 1.0 + 0.1 * math.log(4.0)


def _norm_weights(ctx, layers, seed):
    rng = np.random.default_rng(seed)
    w = (1.0 + 0.02 * rng.standard_normal((layers, 2, D))).astype(np.float32)
    for layer in range(layers):
        ctx.set_norm_weights(layer, w[layer, 0], w[layer, 1])


def _normal(shape, gen):
    return torch.randn(shape, device="cuda", dtype=torch.float32, generator=gen)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    layers = case["layers"]
    if case["kind"] == "decode":
        lens, batch = _lengths(case), case["batch"]
        ctx = Hy3Attn(kv_dtype=case["kv"], n_layers=layers, kv_head_count=case["heads"], max_seqs=batch, max_batch=batch,
                      max_tokens=sum(n + 1 for n in lens), max_tokens_per_seq=max(lens) + 129)
        _norm_weights(ctx, layers, seed)
        if case["yarn"]:
            ctx.set_rope(*_yarn4())
        for layer in range(layers):
            for i, n in enumerate(lens):
                ctx.fill_random(layer, i, 0, n, seed * 1000003 + 1000 * layer + i)
        s = {"case": case, "ctx": ctx, "seqs": np.arange(batch, dtype=np.int32), "slots": np.array(lens, np.int32),
             "q": list(_normal((layers, batch, H, D), gen).unbind(0)), "k": list(_normal((layers, batch, G, D), gen).unbind(0)),
             "v": list(_normal((layers, batch, G, D), gen).unbind(0))}
        s["out"] = torch.zeros((layers, batch, H, D), device="cuda")
        s["out_l"] = list(s["out"].unbind(0))
        ctx.batch_set(s["seqs"], s["slots"])
        if case["graph"]:
            # one graph per token, replayed with new positions; captured on a stream of its own
            torch.cuda.synchronize()
            side = torch.cuda.Stream()
            ctx.set_stream(side)
            with torch.cuda.stream(side):
                _decode_layers(s)
            side.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"], stream=side):
                _decode_layers(s)
            side.synchronize()
            ctx.use_torch_stream()
        return s
    prefix, new, chunk = case["prefix"], case["new"], case["chunk"]
    ctx = Hy3Attn(kv_dtype=case["kv"], n_layers=layers, max_batch=chunk, max_tokens=prefix + new + 128)
    _norm_weights(ctx, layers, seed)
    s = {"case": case, "ctx": ctx, "q": list(_normal((layers, new, H, D), gen).unbind(0)),
         "k": list(_normal((layers, new, G, D), gen).unbind(0)), "v": list(_normal((layers, new, G, D), gen).unbind(0)),
         "q16": torch.empty((chunk, H, D), dtype=torch.float16, device="cuda"), "out": torch.zeros((layers, new, H, D), device="cuda")}
    s["chunks"] = [(c0, min(chunk, new - c0)) for c0 in range(0, new, chunk)]
    s["seqs"] = np.zeros(chunk, np.int32)
    # the cached prefix was ingested by earlier turns, in the same chunks
    for c0 in range(0, prefix, chunk):
        n = min(chunk, prefix - c0)
        ctx.batch_set(s["seqs"][:n], np.arange(c0, c0 + n, dtype=np.int32))
        for layer in range(layers):
            q16 = s["q16"][:n]
            ctx.append(layer, _normal((n, H, D), gen), _normal((n, G, D), gen), _normal((n, G, D), gen), q_out=False, q_out16=q16)
            if c0 + n == prefix:
                ctx.prefill(layer, 0, c0, q16)
    return s


def _decode_layers(s):
    ctx, q, k, v, out = s["ctx"], s["q"], s["k"], s["v"], s["out_l"]
    for layer in range(s["case"]["layers"]):
        ctx.decode_step(layer, q[layer], k[layer], v[layer], out=out[layer])


def run(state):
    s, case = state, state["case"]
    ctx = s["ctx"]
    if case["kind"] == "decode":
        ctx.batch_set(s["seqs"], s["slots"])
        if case["graph"]:
            s["graph"].replay()
        else:
            _decode_layers(s)
        return s["out"]
    base, out = case["prefix"], s["out"]
    for c0, n in s["chunks"]:
        ctx.batch_set(s["seqs"][:n], np.arange(base + c0, base + c0 + n, dtype=np.int32))
        q16 = s["q16"][:n]
        for layer in range(case["layers"]):
            ctx.append(layer, s["q"][layer][c0:c0 + n], s["k"][layer][c0:c0 + n], s["v"][layer][c0:c0 + n], q_out=False, q_out16=q16)
            ctx.prefill(layer, 0, base + c0, q16, out=out[layer, c0:c0 + n])
    return out


def _prefill_flops(case):
    new, prefix = case["new"], case["prefix"]
    return case["layers"] * 4.0 * D * H * (new * prefix + new * (new + 1) / 2)


def work(case):
    per_token = KV_BYTES_PER_TOKEN_HEAD[case["kv"]]
    if case["kind"] == "decode":
        heads, batch = case["heads"], case["batch"]
        tokens = sum(n + 1 for n in _lengths(case))
        rows = batch * heads * (8 + 1 + 1 + 8) * D * 4              # q, k, v in, out
        # every cached token read once, the new one written once
        return {"bytes": float(case["layers"] * (tokens * heads * per_token + batch * heads * per_token + rows)),
                "flops": float(case["layers"] * tokens * heads * 8 * 4 * D)}
    new, prefix = case["new"], case["prefix"]
    rows = new * (H + G + G + H) * D * 4
    return {"bytes": float(case["layers"] * ((prefix + new) * G * per_token + rows)), "flops": _prefill_flops(case)}


def tolerance(case):
    # Outputs are fp32.  decode: scores and weights are carried in two 8-bit or two fp16 digits (about 2^-15 of the largest)
    # into fp32 sums; prefill: queries and weights are rounded to fp16 (2^-11 each) before fp32 sums.
    return {"rel": 3e-4} if case["kind"] == "decode" else {"rel": 1e-3}
