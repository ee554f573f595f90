"""The work this package is used for, as cases that can be timed one pass at a time.

Four directions: the quantized linears of a decoder layer called as a model calls them (decode with a few rows of
activations, prefill with many), fp16 weights quantized into the hybrid format, quantized streams taken into use (the
first forward of fresh ``QuantizedLinear`` modules), and streams expanded back to fp16.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call, on the GPU and from the seed
alone; ``run`` is one pass through the public entry points; ``work`` is what a pass cannot do without.
"""
from __future__ import annotations

import math

import torch

import atlasinfer_b200 as ab

DEVICE = "cuda"
# entries that the z > 3 rule takes out of a 128-block of the weights below (normal tails and the injected ones)
OUTLIERS = 0.003


def listed():
    return [
        # One projection of a small model for one token: the smallest call there is, all latency.
        dict(name="linear_1tok", kind="linear", n=2048, k=2048, m=1, dtype="fp16", bias=True, block=128),
        # A small model's decoder layer (OPT-1.3B shapes, biases, fp16) generating one token.
        dict(name="small_layer_1tok", kind="layer", hidden=2048, kv=2048, inter=8192, gated=False, m=1, dtype="fp16",
             bias=True, fused=True, block=128),
        # A Llama-2-7B-shaped layer generating one token for one user: the headline decode.
        dict(name="mid_layer_1tok", kind="layer", hidden=4096, kv=4096, inter=11008, gated=True, m=1, dtype="bf16",
             bias=False, fused=True, block=128),
        # The same layer with sixteen users, or one user and a speculative draft.
        dict(name="mid_layer_16tok", kind="layer", hidden=4096, kv=4096, inter=11008, gated=True, m=16, dtype="bf16",
             bias=False, fused=True, block=128),
        # A Llama-3-70B-shaped layer with a serving batch of 32: the largest weights.
        dict(name="large_layer_32tok", kind="layer", hidden=8192, kv=1024, inter=28672, gated=True, m=32, dtype="bf16",
             bias=False, fused=True, block=128),
        # A small model's prompt of 128 tokens.
        dict(name="small_layer_128tok", kind="layer", hidden=2048, kv=2048, inter=8192, gated=False, m=128,
             dtype="fp16", bias=True, fused=True, block=128),
        # An ordinary chat prompt: a few hundred tokens, not a round number, siblings not fused.
        dict(name="mid_layer_301tok", kind="layer", hidden=4096, kv=4096, inter=11008, gated=True, m=301,
             dtype="bf16", bias=False, fused=False, block=128),
        # A long prompt: the most arithmetic.
        dict(name="mid_layer_2048tok", kind="layer", hidden=4096, kv=4096, inter=11008, gated=True, m=2048,
             dtype="bf16", bias=False, fused=True, block=128),
        # A whole layer's weights quantized in one batch, as when a model is converted.
        dict(name="quantize_layer", kind="quantize", hidden=4096, kv=4096, inter=11008, gated=True, block=128, z=3.0),
        # One odd-sized tensor on its own, short blocks and a high threshold: ends inside a block, on no alignment.
        dict(name="quantize_odd", kind="quantize_one", n=1001, k=1337, block=64, z=3.5),
        # A stored layer taken into use: the kernel layout is built from the streams and the first token goes through.
        dict(name="load_layer", kind="load", hidden=4096, kv=4096, inter=11008, gated=True, m=1, dtype="bf16",
             bias=False, fused=True, block=128),
        # A layer's weights back to fp16, for export or for a check against the unquantized model.
        dict(name="dequantize_layer", kind="dequantize", hidden=4096, kv=4096, inter=11008, gated=True, block=128),
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of ``step`` between ``lo`` and ``hi``, spread evenly over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi // step, max(-(-lo // step), round(v / step)))) * step


def _draw_layer(rng, hidden_max):
    hidden = _log_int(rng, 1024, hidden_max, 128)
    gated = rng.random() < 0.7
    return dict(hidden=hidden, kv=hidden if rng.random() < 0.5 else max(64, hidden // rng.choice((4, 8)) // 64 * 64),
                inter=_log_int(rng, 2 * hidden, 4 * hidden if not gated else 3.5 * hidden, 128), gated=gated)


def draw(rng):
    kind = rng.choices(("linear", "decode", "prefill", "quantize", "quantize_one", "load", "dequantize"),
                       (2, 6, 5, 2, 2, 2, 1))[0]
    dtype = rng.choice(("fp16", "bf16"))
    block = rng.choice((64, 128, 128, 128))
    if kind == "linear":
        # output features need no round number, input features are whole 128-column blocks
        return dict(kind="linear", n=_log_int(rng, 512, 16384), k=_log_int(rng, 512, 16384, 128),
                    m=_log_int(rng, 1, 512), dtype=dtype, bias=rng.random() < 0.5, block=block)
    if kind == "decode":
        return dict(kind="layer", **_draw_layer(rng, 8192), m=_log_int(rng, 1, 64), dtype=dtype,
                    bias=rng.random() < 0.3, fused=rng.random() < 0.7, block=block)
    if kind == "prefill":
        return dict(kind="layer", **_draw_layer(rng, 4096), m=_log_int(rng, 65, 2048), dtype=dtype,
                    bias=rng.random() < 0.3, fused=rng.random() < 0.7, block=block)
    if kind == "quantize":
        return dict(kind="quantize", **_draw_layer(rng, 4096), block=rng.choice((32, 64, 128, 128, 128, 256)),
                    z=rng.choice((2.5, 3.0, 3.0, 3.5)))
    if kind == "quantize_one":
        return dict(kind="quantize_one", n=_log_int(rng, 100, 8192), k=_log_int(rng, 100, 8192),
                    block=rng.choice((32, 64, 128, 128, 128, 256)), z=rng.choice((2.5, 3.0, 3.0, 3.5)))
    if kind == "load":
        return dict(kind="load", **_draw_layer(rng, 4096), m=_log_int(rng, 1, 64), dtype=dtype, bias=rng.random() < 0.3,
                    fused=rng.random() < 0.7, block=block)
    return dict(kind="dequantize", **_draw_layer(rng, 4096), block=block)


def _shapes(case):
    """(out_features, in_features) of the case's weights, in the order a decoder layer calls them."""
    if case["kind"] in ("linear", "quantize_one"):
        return [(case["n"], case["k"])]
    h, kv, inter = case["hidden"], case["kv"], case["inter"]
    ups = [(inter, h)] * (2 if case["gated"] else 1)
    return [(h, h), (kv, h), (kv, h), (h, h)] + ups + [(h, inter)]


def _weight(n, k, gen):
    """fp16 N(0, 0.02), one entry of every thousand (at a random place among them) replaced by +-U(0.1, 0.5)."""
    w = (torch.randn(n, k, generator=gen, device=DEVICE) * 0.02).to(torch.float16)
    count = n * k // 1000
    at = torch.arange(count, device=DEVICE) * 1000 + torch.randint(0, 1000, (count,), generator=gen, device=DEVICE)
    big = torch.rand(count, generator=gen, device=DEVICE) * 0.4 + 0.1
    sign = torch.where(torch.rand(count, generator=gen, device=DEVICE) < 0.5, -1.0, 1.0)
    w.view(-1)[at] = (big * sign).to(torch.float16)
    return w


def _shuffled(w, block, gen):
    """``w`` with its whole blocks in another order: other inputs, but as many outliers, so that the lengths of the
    quantized streams, which depend on the data, are the same for every seed."""
    flat = w.view(-1)
    whole = flat.numel() // block * block
    order = torch.randperm(whole // block, generator=gen, device=DEVICE)
    flat[:whole] = flat[:whole].view(-1, block)[order].view(-1)
    return w


def _activations(m, k, dtype, gen):
    """N(0, 1); prompts have 0.5 % of their channels twenty times as large."""
    x = torch.randn(m, k, generator=gen, device=DEVICE)
    if m > 64:
        x[:, torch.randperm(k, generator=gen, device=DEVICE)[:max(1, k // 200)]] *= 20
    return x.to(torch.float16 if dtype == "fp16" else torch.bfloat16)


def _modules(case, streams, biases):
    """The case's weights as ``QuantizedLinear`` modules; a layer's siblings joined where the case says so."""
    mods = [ab.QuantizedLinear(q, b) for q, b in zip(streams, biases)]
    groups = []
    if case.get("fused"):
        groups.append(ab.fuse_linears(mods[0:3]))
        if case["gated"]:
            groups.append(ab.fuse_linears(mods[4:6]))
    return mods, groups


def _forward(mods, xs):
    """Every linear called with its input; those that share an input get the very same tensor."""
    return [mod(xs[mod.original_shape[1]]) for mod in mods]


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    shapes = _shapes(case)
    if case["kind"] in ("quantize", "quantize_one"):
        values = torch.Generator(device=DEVICE).manual_seed(1)
        return dict(case=case, weights=[_shuffled(_weight(n, k, values), case["block"], gen) for n, k in shapes])
    weights = [_weight(n, k, gen) for n, k in shapes]
    streams = ab.quantize_tensors(weights, block_size=case["block"])
    del weights
    if case["kind"] == "dequantize":
        return dict(case=case, streams=streams)
    biases = [(torch.randn(n, generator=gen, device=DEVICE) * 0.02).half() if case["bias"] else None for n, _ in shapes]
    xs = {k: _activations(case["m"], k, case["dtype"], gen) for k in sorted({k for _, k in shapes})}
    state = dict(case=case, xs=xs, streams=streams, biases=biases)
    if case["kind"] != "load":
        state["mods"], groups = _modules(case, streams, biases)
        # a program's first forward lays the weights out; every later pass finds them so
        with torch.no_grad():
            _forward(state["mods"], {k: x[:1] for k, x in xs.items()})
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "quantize":
        return [tuple(q[:4]) for q in ab.quantize_tensors(state["weights"], block_size=case["block"], z_threshold=case["z"])]
    if kind == "quantize_one":
        return tuple(ab.quantize_tensor(state["weights"][0], block_size=case["block"], z_threshold=case["z"])[:4])
    if kind == "dequantize":
        device = torch.device(DEVICE, torch.cuda.current_device())
        out = [ab.dequantize_tensor(q, device) for q in state["streams"]]
        ab.clear_dequantized_cache()   # the caller keeps the tensors, not the package
        return out
    with torch.no_grad():
        if kind == "load":
            mods, _ = _modules(case, state["streams"], state["biases"])
            return _forward(mods, state["xs"])
        return _forward(state["mods"], state["xs"])


def work(case):
    """Bytes: every stream, weight and activation once.  Operations: the products of the linears."""
    kind, bs = case["kind"], case["block"]
    nbytes = flops = 0.0
    for n, k in _shapes(case):
        dense = n * k
        out = OUTLIERS * dense
        codes = dense - out + 2.0 * dense / bs          # one byte a code, one fp16 scale a block
        if kind in ("quantize", "quantize_one"):
            nbytes += 2.0 * dense + codes + 10.0 * out  # an outlier is an fp16 value and an int64 position
        elif kind == "dequantize":
            nbytes += codes + 10.0 * out + 2.0 * dense
        else:
            m = case["m"]
            nbytes += codes + 6.0 * out + 2.0 * m * (n + k)
            flops += 2.0 * m * dense
            if kind == "load":
                nbytes += codes + 10.0 * out            # the streams in, the layout out, and the layout read once
                nbytes += codes + 6.0 * out
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """Streams and fp16 reconstructions are the same bits.  Outputs of the linears: the distance of the path from the
    same product in 64 bits is the rounding of the output type, 2-norm 2.1e-4 (fp16) and 1.7e-3 (bf16); four times
    that."""
    if case["kind"] in ("quantize", "quantize_one", "dequantize"):
        return "exact"
    return dict(rel=8e-4) if case["dtype"] == "fp16" else dict(rel=6.6e-3)
