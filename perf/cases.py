"""The calls whose speed matters to a program that uses this package, over the range of sizes it makes them at.

A case is a dict of plain values; its "kind" says which public entry point it goes through:

  linear     nn::Linear on f32 / f16 / bf16 weights: one token per step up to a whole prompt
  matmul     `matmul` against a row-major [k, n] right-hand side
  block      int4 / int8 block-quantized linear, activations quantized to int8 on the way in
  fp8        e4m3 linear with one scale per output channel, bf16 in and out
  grouped    one weight per codebook, all groups in one call
  attention  matmul_t -> softmax -> matmul over a [batch, heads, context, 128] cache, as the models write it
  conv       conv1d / conv_transpose1d of an audio codec, one streaming step up to whole clips
  decode     one token per stream through a stack of decoder layers
  prefill    the prompt of one stream through the same stack
"""
from __future__ import annotations

import math

import torch

import xn_b200 as xn
from xn_b200.decoder import DecoderStack
from xn_b200.prefill import PrefillStack

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
BYTES = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # the attention output projection of one stream's next token: the smallest call, made once per layer and token
        {"name": "linear_bf16_one_token", "kind": "linear", "dtype": "bf16", "m": 1, "n": 4096, "k": 4096, "bias": False},
        # f32 weights, 16 streams: the benchmark's first configuration, the only one the reference's CPU runs as it is
        {"name": "linear_f32_16_streams", "kind": "linear", "dtype": "f32", "m": 16, "n": 11264, "k": 4096, "bias": False},
        # a long prompt of no round length through a 16-bit layer with a bias
        {"name": "linear_f16_prompt", "kind": "linear", "dtype": "f16", "m": 3001, "n": 4096, "k": 11264, "bias": True},
        # 32 one-row products against one row-major weight: the reference's own GPU example
        {"name": "matmul_bf16_32_rows", "kind": "matmul", "dtype": "bf16", "batch": 32, "m": 1, "n": 11264, "k": 2048},
        # int4 weights, a few streams: where quantized decoding lives
        {"name": "int4_4_streams", "kind": "block", "bits": 4, "dtype": "f32", "m": 4, "n": 11264, "k": 4096},
        # fp8 weights with a short prompt, or the rows of a few prompts: between decode and prefill
        {"name": "fp8_short_prompt", "kind": "fp8", "m": 250, "n": 12288, "k": 4096, "variant": 0},
        # the per-codebook feed-forward up projection for 64 streams
        {"name": "grouped_64_streams", "kind": "grouped", "dtype": "bf16", "groups": 16, "m": 64, "n": 4096, "k": 1024},
        # decode attention written as three operations; a context has whatever length the conversation has
        {"name": "attention_8_streams", "kind": "attention", "dtype": "bf16", "batch": 8, "heads": 32, "rows": 1, "context": 1501},
        # one step of a streaming codec: a short window, many channels, one stream
        {"name": "conv1d_f32_stream", "kind": "conv", "dtype": "f32", "transposed": False, "batch": 1, "c_in": 512, "c_out": 512,
         "length": 64, "kernel": 7, "stride": 1, "padding": 3, "groups": 1, "bias": True},
        # one stream's next token through a few layers: everything is latency and launches
        {"name": "decode_one_stream", "kind": "decode", "layers": 4, "heads": 32, "hidden": 11264, "streams": 1, "context": 1000,
         "variant": 0},
        # a full batch of long conversations: the cache is what is read
        {"name": "decode_32_streams", "kind": "decode", "layers": 4, "heads": 32, "hidden": 11264, "streams": 32, "context": 3000,
         "variant": 0},
        # a long prompt through two layers of the same stack
        {"name": "prefill_4096_tokens", "kind": "prefill", "layers": 2, "heads": 32, "hidden": 11264, "tokens": 4096, "variant": 0},
    ]


def _spread(rng, lo: int, hi: int, multiple: int = 1) -> int:
    """A size between lo and hi, evenly over its logarithm, rounded to a multiple."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, multiple * round(v / multiple)))


def _width(rng, lo: int, hi: int) -> int:
    """A layer's width: mostly multiples of 128, now and then only of 16."""
    return _spread(rng, lo, hi, 128 if rng.random() < 0.75 else 16)


def _draw(rng):
    kind = rng.choice(["linear", "matmul", "block", "fp8", "grouped", "attention", "conv", "decode", "prefill"])
    if kind == "linear":
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        n = _width(rng, 1024, 22528)
        # an output width need not be round: a vocabulary with one extra entry
        n += 1 if rng.random() < 0.1 else 0
        return {"kind": kind, "dtype": dtype, "m": _spread(rng, 1, 512 if dtype == "f32" else 4096), "n": n,
                "k": _width(rng, 1024, 11264), "bias": rng.random() < 0.4}
    if kind == "matmul":
        rows = _spread(rng, 1, 512)
        flat = rng.random() < 0.5
        return {"kind": kind, "dtype": rng.choice(["bf16", "bf16", "f16", "f32"]), "batch": 1 if flat else rows,
                "m": rows if flat else 1, "n": _width(rng, 1024, 11264), "k": _width(rng, 1024, 4096)}
    if kind == "block":
        return {"kind": kind, "bits": rng.choice([4, 4, 8]), "dtype": rng.choice(["f32", "bf16"]), "m": _spread(rng, 1, 1024),
                "n": _width(rng, 1024, 22528), "k": _spread(rng, 1024, 11264, 128)}
    if kind == "fp8":
        return {"kind": kind, "m": _spread(rng, 1, 4096), "n": _width(rng, 1024, 22528), "k": _width(rng, 1024, 11264),
                "variant": rng.choice([0, 1])}
    if kind == "grouped":
        return {"kind": kind, "dtype": rng.choice(["bf16", "bf16", "f16"]), "groups": rng.choice([8, 16, 32]), "m": _spread(rng, 1, 128),
                "n": _width(rng, 512, 4096), "k": _width(rng, 512, 2048)}
    if kind == "attention":
        one = rng.random() < 0.6  # one new token per stream, or the rows of a prompt's chunk
        return {"kind": kind, "dtype": rng.choice(["bf16", "bf16", "f16"]), "batch": _spread(rng, 1, 32) if one else 1,
                "heads": rng.choice([8, 16, 32]), "rows": 1 if one else _spread(rng, 2, 256), "context": _spread(rng, 256, 3000)}
    if kind == "conv":
        stride = rng.choice([1, 1, 2, 4, 5, 8])
        channels, transposed = rng.choice([64, 128, 256, 512]), stride > 1 and rng.random() < 0.6
        if transposed:
            c_in, c_out = 2 * channels, channels
        elif stride > 1:
            c_in, c_out = channels, 2 * channels
        else:
            c_in, c_out = channels, channels
        kernel = 2 * stride if stride > 1 else rng.choice([1, 3, 7])
        depthwise = transposed and rng.random() < 0.2  # a learned upsampling of the frames, one filter per channel
        if depthwise:
            c_out = c_in
        return {"kind": kind, "dtype": rng.choice(["f32", "f32", "bf16", "f16"]), "transposed": transposed, "batch": rng.choice([1, 1, 2, 4, 8]),
                "c_in": c_in, "c_out": c_out, "length": _spread(rng, 2 * stride if transposed else 2 * kernel, 512 if transposed else 4096),
                "kernel": kernel, "stride": stride, "padding": (kernel - 1) // 2 if stride == 1 else 0, "groups": c_in if depthwise else 1,
                "bias": rng.random() < 0.8}
    heads = rng.choice([8, 16, 32])
    hidden = _width(rng, 256 * heads, 352 * heads)
    if kind == "decode":
        return {"kind": kind, "layers": rng.choice([2, 3, 4]), "heads": heads, "hidden": hidden, "streams": _spread(rng, 1, 32),
                "context": _spread(rng, 128, 3000), "variant": rng.choice([0, 0, 1])}
    return {"kind": kind, "layers": rng.choice([1, 2]), "heads": heads, "hidden": hidden, "tokens": _spread(rng, 64, 4096),
            "variant": rng.choice([0, 0, 1])}


def draw(rng):
    while True:  # nothing that costs more than the largest listed case
        c = _draw(rng)
        w = work(c)
        if w["bytes"] <= 8e9 and w["flops"] <= (1.2e11 if c.get("dtype") == "f32" else 4e12):
            return c


def _conv_out_length(c) -> int:
    if c["transposed"]:
        return (c["length"] - 1) * c["stride"] + c["kernel"] - 2 * c["padding"]
    return (c["length"] + 2 * c["padding"] - c["kernel"]) // c["stride"] + 1


def prepare(c, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(int(seed))
    kind = c["kind"]

    def normal(*shape, scale=1.0, dtype=None):
        t = torch.randn(*shape, generator=g, device=dev)
        return (t * scale if scale != 1.0 else t).to(dtype or DTYPES[c["dtype"]])

    if kind == "linear":
        w = normal(c["n"], c["k"], scale=0.02)
        return {"kind": kind, "layer": xn.Linear(w, normal(c["n"]) if c["bias"] else None), "x": normal(c["m"], c["k"])}
    if kind == "matmul":
        return {"kind": kind, "lhs": normal(c["batch"], c["m"], c["k"]), "rhs": normal(c["k"], c["n"], scale=0.02)}
    if kind == "block":
        w, x = normal(c["n"], c["k"], scale=0.02, dtype=torch.float32), normal(c["m"], c["k"])
        if c["bits"] == 4:
            return {"kind": "int4", "layer": xn.LinearQ4.from_weight(w), "x": x}
        return {"kind": "int8", "w": xn.quantize_weights_q8(w), "n": c["n"], "x": x}
    if kind == "fp8":
        w = normal(c["n"], c["k"], scale=0.02, dtype=torch.float32)
        return {"kind": kind, "layer": xn.LinearFp8.from_weight(w, c["variant"]), "x": normal(c["m"], c["k"], dtype=torch.bfloat16)}
    if kind == "grouped":
        # [streams, groups, k]: slice g of every stream meets weight g
        x = normal(c["m"], c["groups"], c["k"])
        return {"kind": kind, "x": x.transpose(0, 1), "w": normal(c["groups"], c["n"], c["k"], scale=0.03)}
    if kind == "attention":
        q = normal(c["batch"], c["heads"], c["rows"], 128, scale=1.0 / math.sqrt(128.0))
        return {"kind": kind, "q": q, "k": normal(c["batch"], c["heads"], c["context"], 128),
                "v": normal(c["batch"], c["heads"], c["context"], 128)}
    if kind == "conv":
        fan = (c["c_in"] // c["groups"]) * (c["kernel"] // c["stride"] if c["transposed"] else c["kernel"])
        wshape = (c["c_in"], c["c_out"] // c["groups"], c["kernel"]) if c["transposed"] else (c["c_out"], c["c_in"] // c["groups"], c["kernel"])
        return {"kind": "conv_transpose1d" if c["transposed"] else "conv1d", "x": normal(c["batch"], c["c_in"], c["length"]),
                "w": normal(*wshape, scale=1.0 / math.sqrt(fan)), "bias": normal(c["c_out"]) if c["bias"] else None,
                "stride": c["stride"], "padding": c["padding"], "groups": c["groups"]}
    d = 128 * c["heads"]
    if kind == "decode":
        stack = DecoderStack(c["layers"], d, c["heads"], c["hidden"], c["streams"], c["context"], dev, seed=int(seed), variant=c["variant"])
        return {"kind": kind, "stack": stack, "x": normal(c["streams"], d, dtype=torch.bfloat16)}
    stack = PrefillStack(c["layers"], d, c["heads"], c["hidden"], c["tokens"], dev, seed=int(seed), variant=c["variant"])
    return {"kind": kind, "stack": stack, "x": normal(c["tokens"], d, dtype=torch.bfloat16)}


def run(s):
    kind = s["kind"]
    if kind in ("linear", "int4", "fp8"):
        return s["layer"](s["x"])
    if kind == "matmul":
        return xn.matmul(s["lhs"], s["rhs"])
    if kind == "int8":
        xq, xs = xn.quantize_rows_i8(s["x"])
        return xn.linear_q8(xq, xs, s["w"], s["n"])
    if kind == "grouped":
        return xn.matmul_t(s["x"], s["w"])
    if kind == "attention":
        scores = xn.matmul_t(s["q"], s["k"])
        probs = xn.ops.softmax(scores)
        return {"scores": scores, "probs": probs, "out": xn.matmul(probs, s["v"])}
    if kind == "conv1d":
        return xn.ops.conv1d(s["x"], s["w"], s["bias"], s["stride"], s["padding"], 1, s["groups"])
    if kind == "conv_transpose1d":
        return xn.ops.conv_transpose1d(s["x"], s["w"], s["bias"], s["stride"], s["padding"], 0, s["groups"])
    if kind == "decode":
        stack = s["stack"]
        y = stack.step(s["x"])
        return {"out": y, "k": [lay["k"] for lay in stack.layers], "v": [lay["v"] for lay in stack.layers]}
    return s["stack"].forward(s["x"])


def work(c):
    kind = c["kind"]
    if kind == "linear":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": BYTES[c["dtype"]] * (m * k + n * k + m * n + (n if c["bias"] else 0)), "flops": 2 * m * n * k}
    if kind == "matmul":
        m, n, k = c["batch"] * c["m"], c["n"], c["k"]
        return {"bytes": BYTES[c["dtype"]] * (m * k + n * k + m * n), "flops": 2 * m * n * k}
    if kind == "block":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": BYTES[c["dtype"]] * m * k + n * k * c["bits"] // 8 + n * (k // 32) * 4 + 4 * m * n, "flops": 2 * m * n * k}
    if kind == "fp8":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2 * m * k + n * k + 4 * n + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "grouped":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": BYTES[c["dtype"]] * c["groups"] * (m * k + n * k + m * n), "flops": 2 * c["groups"] * m * n * k}
    if kind == "attention":
        slabs, t, ctx = c["batch"] * c["heads"], c["rows"], c["context"]
        # queries, keys and values in; scores, probabilities and rows out
        return {"bytes": BYTES[c["dtype"]] * slabs * (2 * t * 128 + 2 * ctx * 128 + 2 * t * ctx), "flops": 4 * slabs * t * ctx * 128}
    if kind == "conv":
        b, taps, lo = c["batch"], (c["c_in"] // c["groups"]) * c["c_out"] * c["kernel"], _conv_out_length(c)
        elements = b * c["c_in"] * c["length"] + taps + b * c["c_out"] * lo + (c["c_out"] if c["bias"] else 0)
        return {"bytes": BYTES[c["dtype"]] * elements, "flops": 2 * b * taps * (c["length"] if c["transposed"] else lo)}
    d, hid, layers = 128 * c["heads"], c["hidden"], c["layers"]
    weights = 4 * d * d + 3 * hid * d
    if kind == "decode":
        b, ctx = c["streams"], c["context"]
        # weights and caches read, one row of each cache written, the tokens in and out
        return {"bytes": layers * (weights + 4 * (5 * d + 2 * hid) + 4 * b * d * (ctx + 1)) + 4 * b * d,
                "flops": layers * (2 * b * weights + 4 * b * d * ctx)}
    t = c["tokens"]
    return {"bytes": layers * (weights + 4 * (5 * d + 2 * hid)) + 4 * t * d, "flops": layers * (2 * t * weights + 2 * t * t * d)}


def tolerance(c):
    kind = c["kind"]
    if kind in ("decode", "prefill", "attention"):
        return {"rel": 1e-2}  # bf16 values handed from one step to the next: a rounding that falls the other way is carried on
    if kind == "block":
        return {"rel": 1e-5}  # exact integer block sums, added up in f32
    if kind == "fp8":
        return {"rel": 4e-3}  # one rounding to bf16
    return {"rel": {"f32": 1e-5, "f16": 1e-3, "bf16": 4e-3}[c["dtype"]]}
