"""Workloads whose speed this framework is judged by: what a user of it runs, through its public entry points.

Six kinds of work, each over the sizes it meets in use:

  linear     one LinearCompressed.forward (ops.PackedLinear): one token of a single stream up to a prompt's tokens; 8 / 4 / 2-bit
             and binary factors, low-rank and full-rank, with and without bias, bf16 and fp32
  attention  one layer's paged decode attention (ops.paged_decode_attention) over a filled quantized cache
  append     one layer's prompt written to its cache: FP8 scales, RoPE on the keys, quantize-and-append (ops.PagedKV)
  step       one captured decode step of an engine (decoder.CompressedDecoder.step), logits returned
  prefill    one batched prompt pass of an engine (CompressedDecoder.prefill)
  generate   prompt and greedy decoding in one call (CompressedDecoder.generate)
  quantize   one weight matrix to packed codes and scales (ops.Factor.quantize), as a model is packed layer by layer

Architectures are the three that the repository's configurations use: Llama-3-8B, Qwen2-0.5B and the language tower of
Qwen2.5-VL-7B (full widths; fewer layers where a pass would only repeat the same layer).  Weights, prompts and cached
values are random with the configurations' distributions: weights N(0, 0.02^2), cached keys and values N(0, 1) with four
outlier channels per head (x 20).
"""
import math
import random

import torch

from transformer_surgeon_b200 import ops
from transformer_surgeon_b200.decoder import CompressedDecoder, DecoderConfig, LayerWeights, fuse_rows, rope_tables

ARCHS = {
    "llama3-8b": dict(hidden=4096, num_heads=32, num_kv_heads=8, head_dim=128, intermediate=14336, vocab=128256,
                      rope_theta=5e5, rms_eps=1e-5),
    "qwen2.5-vl-7b": dict(hidden=3584, num_heads=28, num_kv_heads=4, head_dim=128, intermediate=18944, vocab=152064,
                          rope_theta=1e6, rms_eps=1e-6),
    "qwen2-0.5b": dict(hidden=896, num_heads=14, num_kv_heads=2, head_dim=64, intermediate=4864, vocab=151936,
                       rope_theta=1e6, rms_eps=1e-6),
}
KV_BYTES = {"int8": 1.0, "fp8": 1.0, "nvfp4": 0.5625, "fp32": 4.0, "bf16": 2.0}      # per cached element, without int8's token scales
CHUNK = 2048                                                                          # tokens appended at a time while a cache is filled


def listed():
    return [
        # one token of one stream through a rank-256 4-bit layer: all latency
        dict(name="linear_m1", kind="linear", m=1, inp=4096, out=4096, rank=256, precision="4", bias=False, dtype="bf16"),
        # a small decode batch, 8-bit factors of rank 1024
        dict(name="linear_m16", kind="linear", m=16, inp=4096, out=4096, rank=1024, precision="8", bias=False, dtype="bf16"),
        # an odd number of tokens (a short prompt) through a full-rank projection with bias, binary weights
        dict(name="linear_m77", kind="linear", m=77, inp=3584, out=4608, rank=0, precision="binary", bias=True, dtype="bf16"),
        # a prompt's tokens
        dict(name="linear_m2048", kind="linear", m=2048, inp=4096, out=4096, rank=1024, precision="4", bias=False, dtype="bf16"),
        # a large decode batch of unequal lengths, int8 pages
        dict(name="attn_int8", kind="attention", kv="int8", batch=64, heads=32, kv_heads=8, head_dim=128, context=4096),
        # few sequences with long contexts, NVFP4 pages, seven query heads to a kv head
        dict(name="attn_nvfp4", kind="attention", kv="nvfp4", batch=8, heads=28, kv_heads=4, head_dim=128, context=32768),
        # the prompts of a batch written to FP8 pages
        dict(name="append_fp8", kind="append", kv="fp8", batch=32, kv_heads=8, head_dim=128, tokens=2048),
        # decode at the headline configuration: batch 32, 2k contexts, 4-bit low-rank MLPs, FP8 pages
        dict(name="step_batch32", kind="step", arch="llama3-8b", layers=8, batch=32, context=2048, kv="fp8", bits="4", rank=1024),
        # one interactive stream on a model of mixed precisions and ranks, NVFP4 pages
        dict(name="step_single", kind="step", arch="qwen2.5-vl-7b", layers=8, batch=1, context=4001, kv="nvfp4", bits="mixed", rank=-1),
        # prompts of a batch through the model
        dict(name="prefill", kind="prefill", arch="llama3-8b", layers=4, batch=8, tokens=2048, kv="fp8", bits="4", rank=1024),
        # an fp32 model end to end: 128 prompt tokens, 32 new ones, rank 128 everywhere
        dict(name="generate_fp32", kind="generate", arch="qwen2-0.5b", layers=24, batch=1, tokens=128, new=32, rank=128),
        # packing a model: one MLP matrix
        dict(name="quantize", kind="quantize", rows=14336, cols=4096, precision="4", dtype="bf16"),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "attention", "attention", "append", "step", "step", "prefill", "generate", "quantize"])
    if kind == "linear":
        inp, out = rng.choice([(4096, 4096), (4096, 6144), (4096, 14336), (14336, 4096), (3584, 3584), (3584, 18944), (18944, 3584), (896, 4864)])
        rank = rng.choice([0, 128, 256, 8 * _log(rng, 8, 224)])
        if rng.random() < 0.15:
            return dict(kind=kind, m=_log(rng, 1, 128), inp=inp, out=out, rank=rank, precision=rng.choice(["none", "8", "4"]),
                        bias=rng.random() < 0.5, dtype="fp32")
        return dict(kind=kind, m=_log(rng, 1, 4096), inp=inp, out=out, rank=rank, precision=rng.choice(["8", "4", "4", "2", "binary"]),
                    bias=rng.random() < 0.5, dtype="bf16")
    if kind == "attention":
        heads, kv_heads, head_dim = rng.choice([(32, 8, 128), (28, 4, 128), (14, 2, 64)])
        batch = _log(rng, 1, 64)
        return dict(kind=kind, kv=rng.choice(["int8", "fp8", "nvfp4"]), batch=batch, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
                    context=_log(rng, 64, min(32768, 524288 // batch)))
    if kind == "append":
        kv_heads, head_dim = rng.choice([(8, 128), (4, 128), (2, 64)])
        return dict(kind=kind, kv=rng.choice(["int8", "fp8", "nvfp4"]), batch=_log(rng, 1, 32), kv_heads=kv_heads, head_dim=head_dim,
                    tokens=_log(rng, 1, 2048))
    if kind == "step":
        arch = rng.choice(["llama3-8b", "qwen2.5-vl-7b"])
        batch = _log(rng, 1, 64)
        mixed = rng.random() < 0.5
        return dict(kind=kind, arch=arch, layers=rng.randint(2, 8), batch=batch, context=_log(rng, 128, min(16384, 131072 // batch)),
                    kv=rng.choice(["fp8", "int8", "nvfp4"]), bits="mixed" if mixed else rng.choice(["4", "8", "2"]),
                    rank=-1 if mixed else 8 * rng.randint(64, 224))
    if kind == "prefill":
        arch = rng.choice(["llama3-8b", "qwen2.5-vl-7b"])
        batch = _log(rng, 1, 8)
        return dict(kind=kind, arch=arch, layers=rng.randint(1, 3), batch=batch, tokens=_log(rng, 33, 12288 // batch),
                    kv=rng.choice(["fp8", "int8", "nvfp4"]), bits=rng.choice(["4", "8"]), rank=8 * rng.randint(64, 160))
    if kind == "generate":
        return dict(kind=kind, arch="qwen2-0.5b", layers=rng.randint(4, 24), batch=_log(rng, 1, 4), tokens=_log(rng, 7, 128), new=rng.randint(8, 32),
                    rank=rng.choice([64, 128, 224]))
    rows, cols = rng.choice([14336, 4096, 3584, 18944, 1024, 896, 8 * _log(rng, 16, 448)]), rng.choice([4096, 14336, 3584, 1024, 896, 4864, 8 * _log(rng, 16, 448)])
    return dict(kind=kind, rows=rows, cols=cols, precision=rng.choice(["8", "4", "3", "2", "binary"]), dtype=rng.choice(["bf16", "bf16", "fp32"]))


# ------------------------------------------------------------------------------------------------ inputs
def _dtype(name):
    return torch.bfloat16 if name == "bf16" else torch.float32


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, shape, std, dtype):
    return (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)


def _factor(g, rows, cols, std, precision, dtype):
    w = _randn(g, (rows, cols), std, dtype)
    if precision == "none":
        return ops.Factor.dense(w)
    return ops.Factor.quantize(w, precision if precision == "binary" else int(precision))


def _linear(g, out, inp, rank, precision, dtype, bias=False):
    b = _randn(g, (out,), 0.1, dtype) if bias else None
    if rank == 0:
        return ops.PackedLinear(_factor(g, out, inp, 0.02, precision, dtype), None, b, dtype)
    # the product has the scale of a N(0, 0.02^2) dense weight
    u = _factor(g, out, rank, 0.005 * (inp / rank) ** 0.5, precision, dtype)
    return ops.PackedLinear(u, _factor(g, rank, inp, inp ** -0.5, precision, dtype), b, dtype)


def _outliers(g, kv_heads, head_dim):
    o = torch.ones((kv_heads, head_dim), device="cuda")
    for h in range(kv_heads):
        o[h, torch.randperm(head_dim, generator=g, device="cuda")[:4]] = 20.0
    return o


def _fill(g, kv, seq_lens, batch, context):
    """`context` tokens per sequence into an empty cache; leaves seq_lens at `context`."""
    o = _outliers(g, kv.hkv, kv.head_dim)
    if kv.k_scale is not None:
        kv.fill_fp8_scales(110.0 / 448.0, 110.0 / 448.0)
    seq_lens.zero_()
    for t in range(0, context, CHUNK):
        n = min(CHUNK, context - t)
        k, v = (torch.randn((batch, n, kv.hkv, kv.head_dim), generator=g, device="cuda").mul_(o).bfloat16() for _ in range(2))
        kv.append(k, v)
        seq_lens.add_(n)


def _lengths(c):
    """Tokens per sequence of an attention case: from half the context to all of it."""
    return [c["context"] - (i * (c["context"] // 2)) // c["batch"] for i in range(c["batch"])]


def _recipe(c):
    """Precision and MLP rank (0 = full) of every layer.  Mixed: precisions of {2, 4, 8} with the first and last layer at 8,
    ranks of {25 %, 50 %, 100 %} of the hidden size, from a fixed seed (they are part of the case, not of its inputs)."""
    if c["bits"] != "mixed":
        return [(c["bits"], c["rank"])] * c["layers"]
    r, hidden, n = random.Random(2), ARCHS[c["arch"]]["hidden"], c["layers"]
    bits = ["8" if i in (0, n - 1) else r.choice(["2", "4", "8"]) for i in range(n)]
    return list(zip(bits, [r.choice([hidden // 4, hidden // 2, 0]) for _ in range(n)]))


def _engine(g, c, kv_format, dtype, max_seq, recipe, attn_rank):
    a = ARCHS[c["arch"]]
    h, hkv, d, hid, inter = a["num_heads"], a["num_kv_heads"], a["head_dim"], a["hidden"], a["intermediate"]
    cfg = DecoderConfig(num_layers=c["layers"], dtype=dtype, kv_format=kv_format, max_positions=max_seq + 16, **a)
    biased = c["arch"].startswith("qwen")                  # Qwen2: biases on q, k, v
    layers = []
    for bits, rank in recipe:
        ln = [torch.ones(hid, dtype=dtype, device="cuda") for _ in range(2)]
        mlp = [_linear(g, *s, rank, bits, dtype) for s in ((inter, hid), (inter, hid), (hid, inter))]
        if attn_rank:
            q, k, v = (_linear(g, n * d, hid, attn_rank, bits, dtype, biased) for n in (h, hkv, hkv))
            layers.append(LayerWeights(*ln, _linear(g, hid, h * d, attn_rank, bits, dtype), *mlp, q=q, k=k, v=v))
        else:
            f = [_factor(g, n * d, hid, 0.02, bits, dtype) for n in (h, hkv, hkv)]
            b = [_randn(g, (n * d,), 0.1, dtype) if biased else None for n in (h, hkv, hkv)]
            layers.append(LayerWeights(*ln, _linear(g, hid, h * d, 0, bits, dtype), *mlp, qkv=fuse_rows(f, b, dtype)))
    embed = _randn(g, (a["vocab"], hid), 0.02, dtype)
    head = ops.PackedLinear(ops.Factor.dense(_randn(g, (a["vocab"], hid), 0.02, dtype)), None, None, dtype)
    return CompressedDecoder(cfg, embed, layers, torch.ones(hid, dtype=dtype, device="cuda"), head, c["batch"], max_seq, "cuda")


def _tokens(seed, c, shape):
    return torch.randint(0, ARCHS[c["arch"]]["vocab"], shape, generator=torch.Generator().manual_seed(seed)).cuda()


def prepare(case, seed):
    c, g = case, _gen(seed)
    kind = c["kind"]
    if kind == "linear":
        dt = _dtype(c["dtype"])
        return dict(c, layer=_linear(g, c["out"], c["inp"], c["rank"], c["precision"], dt, c["bias"]), x=_randn(g, (c["m"], c["inp"]), 1.0, dt))
    if kind == "attention":
        b, pages = c["batch"], (c["context"] + 15) // 16
        table = torch.randperm(b * pages, generator=g, device="cuda").to(torch.int32).reshape(b, pages)
        seq = torch.zeros(b, dtype=torch.int32, device="cuda")
        cache = ops.PagedKV(c["kv"], b * pages, c["kv_heads"], c["head_dim"], table, seq, "cuda")
        _fill(g, cache, seq, b, c["context"])
        seq.copy_(torch.tensor(_lengths(c), dtype=torch.int32))
        return dict(c, cache=cache, q=_randn(g, (b, c["heads"], c["head_dim"]), 1.0, torch.bfloat16))
    if kind == "append":
        b, pages = c["batch"], (c["tokens"] + 15) // 16
        table = torch.randperm(b * pages, generator=g, device="cuda").to(torch.int32).reshape(b, pages)
        cache = ops.PagedKV(c["kv"], b * pages, c["kv_heads"], c["head_dim"], table, torch.zeros(b, dtype=torch.int32, device="cuda"), "cuda")
        o = _outliers(g, c["kv_heads"], c["head_dim"])
        k, v = ((torch.randn((b, c["tokens"], c["kv_heads"], c["head_dim"]), generator=g, device="cuda") * o).bfloat16() for _ in range(2))
        return dict(c, cache=cache, k=k, v=v, rope=rope_tables(c["head_dim"], 1e6, c["tokens"], "cuda"))
    if kind == "step":
        e = _engine(g, c, c["kv"], torch.bfloat16, c["context"] + 16, _recipe(c), 0)
        for cache in e.kv:
            _fill(g, cache, e.seq_lens, c["batch"], c["context"])
        e.capture()
        return dict(c, engine=e, lens=e.seq_lens.clone(), ids=_tokens(seed, c, (c["batch"],)))
    if kind == "prefill":
        e = _engine(g, c, c["kv"], torch.bfloat16, c["tokens"] + 16, _recipe(c), 0)
        return dict(c, engine=e, ids=_tokens(seed, c, (c["batch"], c["tokens"])))
    if kind == "generate":
        e = _engine(g, c, "fp32", torch.float32, c["tokens"] + c["new"] + 8, [("none", c["rank"])] * c["layers"], c["rank"])
        e.capture()
        return dict(c, engine=e, ids=_tokens(seed, c, (c["batch"], c["tokens"])))
    return dict(c, w=_randn(g, (c["rows"], c["cols"]), 0.02, _dtype(c["dtype"])))


# ------------------------------------------------------------------------------------------------ one pass
def _caches(e, fmt):
    """The engine's caches: FP8 pages as the numbers they hold, others as bytes."""
    pools = [p for kv in e.kv for p in (kv.k_pool, kv.v_pool)]
    return [p.view(torch.float8_e4m3fn) for p in pools] if fmt == "fp8" else pools


def run(state):
    s = state
    kind = s["kind"]
    if kind == "linear":
        return s["layer"](s["x"])
    if kind == "attention":
        return ops.paged_decode_attention(s["cache"], s["q"], s["context"])
    if kind == "append":
        cache = s["cache"]
        if s["kv"] == "fp8":
            cache.set_fp8_scales(s["k"], s["v"], rope=s["rope"])
        cache.append(s["k"], s["v"], rope=s["rope"])
        return [cache.k_pool, cache.v_pool] + ([cache.k_scale, cache.v_scale] if s["kv"] == "fp8" else [])
    e = s.get("engine")
    if kind == "step":
        e.seq_lens.copy_(s["lens"])          # the same token position on every pass
        return [e.step(s["ids"])] + _caches(e, s["kv"])
    if kind == "prefill":
        logits = e.prefill(s["ids"])
        return [logits] + (_caches(e, "fp8") if s["kv"] == "fp8" else [])
    if kind == "generate":
        return list(e.generate(s["ids"], s["new"], batched_prefill=True))
    f = ops.Factor.quantize(s["w"], s["precision"] if s["precision"] == "binary" else int(s["precision"]))
    return [f.data, f.scales]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _bits(precision):
    return {"binary": 1, "2": 2, "3": 4, "4": 4, "8": 8, "none": 32}[precision]


def _weights(out, inp, rank, precision):
    """(elements, bytes) of a layer's factors with their scales."""
    shapes = [(out, rank), (rank, inp)] if rank else [(out, inp)]
    n = sum(r * k for r, k in shapes)
    return n, n * _bits(precision) / 8 + (4 * sum(r for r, _ in shapes) if precision != "none" else 0)


def _layer_work(a, bits, rank, attn_rank):
    h, hkv, d, hid, inter = a["num_heads"], a["num_kv_heads"], a["head_dim"], a["hidden"], a["intermediate"]
    parts = [_weights(n * d, hid, attn_rank, bits) for n in (h, hkv, hkv)] + [_weights(hid, h * d, attn_rank, bits)]
    parts += [_weights(inter, hid, rank, bits)] * 2 + [_weights(hid, inter, rank, bits)]
    return sum(p[0] for p in parts), sum(p[1] for p in parts)


def work(case):
    c = case
    kind = c["kind"]
    if kind == "linear":
        n, b = _weights(c["out"], c["inp"], c["rank"], c["precision"])
        elt = 2 if c["dtype"] == "bf16" else 4
        return {"bytes": b + elt * c["m"] * (c["inp"] + c["out"]) + (elt * c["out"] if c["bias"] else 0), "flops": 2.0 * c["m"] * n}
    if kind == "attention":
        tokens, d = sum(_lengths(c)), c["head_dim"]
        per = 2 * c["kv_heads"] * (d * KV_BYTES[c["kv"]] + (4 if c["kv"] == "int8" else 0))
        return {"bytes": tokens * per + 4 * c["batch"] * c["heads"] * d, "flops": 4.0 * tokens * c["heads"] * d}
    if kind == "append":
        n = 2.0 * c["batch"] * c["tokens"] * c["kv_heads"] * c["head_dim"]
        return {"bytes": n * (2 + KV_BYTES[c["kv"]]), "flops": 0.0}
    if kind == "quantize":
        n = float(c["rows"] * c["cols"])
        return {"bytes": n * (2 if c["dtype"] == "bf16" else 4) + n * _bits(c["precision"]) / 8 + 4 * c["rows"], "flops": 0.0}
    a = ARCHS[c["arch"]]
    h, hkv, d = a["num_heads"], a["num_kv_heads"], a["head_dim"]
    if kind == "generate":
        n, b = _layer_work(a, "none", c["rank"], c["rank"])
        head, t, layers, batch = a["vocab"] * a["hidden"], c["tokens"], c["layers"], c["batch"]
        passes = 1 + c["new"]
        kv = sum(batch * (t + i) * 2 * hkv * d * 4 for i in range(c["new"])) * layers
        attn = 4.0 * batch * layers * h * d * (t * t / 2 + sum(t + i for i in range(c["new"])))
        return {"bytes": passes * (layers * b + 4.0 * head) + kv, "flops": 2.0 * batch * (layers * n * (t + c["new"]) + head * passes) + attn}
    per_layer = [_layer_work(a, bits, rank, 0) for bits, rank in _recipe(c)]
    n, b = sum(p[0] for p in per_layer), sum(p[1] for p in per_layer)
    head, batch, layers, kvb = a["vocab"] * a["hidden"], c["batch"], c["layers"], KV_BYTES[c["kv"]]
    if kind == "step":
        cached = float(batch * c["context"] * layers)
        return {"bytes": b + 2.0 * head + cached * 2 * hkv * d * kvb + 2.0 * batch * a["vocab"],
                "flops": 2.0 * batch * (n + head) + 4.0 * cached * h * d}
    t = c["tokens"]
    return {"bytes": b + 2.0 * head + batch * t * (2.0 * a["hidden"] + layers * 2 * hkv * d * kvb),
            "flops": 2.0 * batch * (t * n + head) + layers * 4.0 * batch * h * d * t * t / 2}


def tolerance(case):
    kind = case["kind"]
    if kind == "append":
        return "exact"                                   # codes and scales are defined bit for bit
    if kind == "quantize":
        return {"rel": 4e-3} if case["precision"] == "binary" else "exact"       # binary: a mean, rounded to the weights' type
    if kind == "generate":
        return {"rel": 1e-4}                             # fp32 through all layers; the tokens are the same
    if kind == "linear":
        return {"rel": 1e-5} if case["dtype"] == "fp32" else {"rel": 1e-2}
    if kind == "attention":
        return {"rel": 1e-2}
    # bf16 through all layers; an appended code may be its neighbour where a key or value lies between two
    return {"rel": 2e-2, "differ": 1e-2}
