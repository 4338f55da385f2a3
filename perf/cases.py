"""Performance cases of the MoE feed-forward operator.

What a serving process asks of it, through the public calls of lumen_b200.moe: one token at a time
through a stack of layers, decode batches of a few requests, prompts of a few dozen to several
thousand tokens, with and without the always-on shared expert, over the three weight formats, the
two gating functions and both activation types. Layer shapes are those of the repository's
configurations, benchmark and tests, and generic ones.

A case is a dict of plain values:
  op        "decode": decode (1..16 tokens) | "decode_norm": the form with the RMSNorm fused in |
            "prefill": any number of tokens. With layers > 1 the stack form of the call
  tokens    rows of the activation
  layers    distinct layers of the stack (x <- x + FFN(rmsnorm(x)) per layer), 1 = a single layer call
  hidden, inter, experts, top_k, quant ("q4_0" | "q8_0" | "bf16"), gating ("softmax" | "sigmoid")
  act       activation type of a prefill call ("f32" | "bf16")
  shared    inter size of the shared expert applied after the routed ones, 0 = none
  skew      exponent of the experts' popularity (0 = near-uniform loads, 1.1 = Zipf)
"""
from __future__ import annotations

import math

import torch

from lumen_b200 import moe, synth

QUANT = {"q4_0": moe.Q4_0, "q8_0": moe.Q8_0, "bf16": moe.BF16}
BYTES = {"q4_0": 18 / 32, "q8_0": 34 / 32, "bf16": 2.0}  # per weight
GATING = {"softmax": moe.SOFTMAX_RENORM, "sigmoid": moe.SIGMOID_RENORM}
EPS = 1e-6

# hidden, inter, experts, top_k
BENCH = (2048, 768, 128, 8)   # the benchmark's layer
MANY = (2048, 512, 256, 8)    # the shape of the end-to-end fixture of the tests: many narrow experts
SMALL = (512, 256, 16, 4)     # the stack tests' layer
WIDE = (4096, 1536, 64, 6)    # generic: a wide model with fewer, larger experts


def _case(op, tokens, shape, quant, *, layers=1, gating="softmax", act="f32", shared=0, skew=0.0):
    h, i, e, k = shape
    return {"op": op, "tokens": tokens, "layers": layers, "hidden": h, "inter": i, "experts": e, "top_k": k,
            "quant": quant, "gating": gating, "act": act, "shared": shared, "skew": skew}


def listed():
    cases = {
        # interactive decoding, one request: the token's way through (a part of) the model
        "token": _case("decode_norm", 1, BENCH, "q4_0", layers=8),
        # the same in the 8-bit format, one layer call at a time
        "token-q8": _case("decode", 1, BENCH, "q8_0"),
        # the smallest call: a small layer, one token; latency and launches are all there is
        "token-small": _case("decode", 1, SMALL, "q8_0"),
        # a few requests decoded together, layer with its shared expert
        "batch-3-shared": _case("decode", 3, MANY, "q4_0", gating="sigmoid", shared=512),
        # an odd batch on unquantised weights
        "batch-5-bf16": _case("decode_norm", 5, MANY, "bf16", gating="sigmoid"),
        # a wide model, 8-bit weights, an odd batch
        "batch-13-wide": _case("decode", 13, WIDE, "q8_0"),
        # the largest decode batch
        "batch-16": _case("decode_norm", 16, BENCH, "q4_0"),
        # a short prompt
        "prompt-77": _case("prefill", 77, BENCH, "q4_0"),
        # an ordinary prompt (or a chunk of a long one), layer with its shared expert
        "prompt-300-shared": _case("prefill", 300, MANY, "q8_0", act="bf16", shared=512),
        # a long prompt of odd length on unquantised weights
        "prompt-1777-bf16": _case("prefill", 1777, BENCH, "bf16", act="bf16"),
        # a full prefill chunk with skewed expert loads
        "prompt-4096-zipf": _case("prefill", 4096, BENCH, "q4_0", act="bf16", skew=1.1),
        # several prompts together through a stack of layers
        "prompts-8192": _case("prefill", 8192, BENCH, "q4_0", layers=2),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def draw(rng):
    tokens = round(math.exp(rng.uniform(0.0, math.log(8192))))
    if rng.random() < 0.4:
        h, i, e, k = rng.choice([BENCH, BENCH, MANY, WIDE])
    else:
        h = 256 * round(math.exp(rng.uniform(math.log(2), math.log(16))))
        i = 128 * round(math.exp(rng.uniform(math.log(2), math.log(12))))
        e = rng.choice([16, 32, 64, 64, 128, 128, 256])
        while e > 16 and 3 * e * h * i > 1.25e9:  # device memory of a layer
            e //= 2
        k = rng.choice([2, 4, 6, 8, 8])
    op = "prefill"
    if tokens <= 16 and rng.random() < 0.85:  # very short prompts take the prefill call as well
        op = rng.choice(["decode", "decode_norm"])
    layers = 1
    if op == "decode_norm" and tokens <= 4:
        layers = rng.choice([1, 2, 4])
    elif op == "prefill" and rng.random() < 0.2:
        layers = 2
    while layers * tokens * k * 6 * h * i > 1.2e12:  # no more than the largest listed case
        tokens = tokens * 3 // 4
    stack = layers > 1
    return _case(op, tokens, (h, i, e, k), rng.choice(["q4_0", "q4_0", "q4_0", "q8_0", "q8_0", "bf16"]), layers=layers,
                 gating=rng.choice(["softmax", "sigmoid"]),
                 act=rng.choice(["f32", "bf16"]) if op == "prefill" and not stack else "f32",
                 shared=rng.choice([0, 0, 0, 512]) if not stack and op != "decode_norm" else 0,
                 skew=rng.choice([0.0, 0.0, 1.1]) if op == "prefill" and not stack else 0.0)


class _State:
    pass


def prepare(case, seed):
    h, t, e = case["hidden"], case["tokens"], case["experts"]
    quant, gating = QUANT[case["quant"]], GATING[case["gating"]]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s = _State()
    s.case = case
    lay = synth.LayerLayout(h, case["inter"], e, quant)
    s.scratch = moe.allocate_moe_scratch(h, case["inter"], e, case["top_k"], max(t, 16), gating)
    s.x = torch.randn((t, h), generator=g, device="cuda")
    common = None
    if case["skew"]:
        # expert popularity ~ rank^-skew: activations of a real model share a component, and a
        # router row's product with it is the expert's standing advantage in the logits
        common = torch.randn(h, generator=g, device="cuda")
        common /= common.norm()
        s.x += 8.0 * common
        rank = torch.randperm(e, generator=g, device="cuda") + 1
        bias = -case["skew"] * torch.log(rank.float())
    s.layers, s.gammas = [], []
    for l in range(case["layers"]):
        blob = synth.make_layer_blob(lay, seed * 64 + l)
        if common is not None:
            router = blob[:lay.router_bytes].view(torch.float32).view(e, h)
            router += (bias / 8.0)[:, None] * common[None, :]
        s.layers.append(s.scratch.prepare_layer(blob, lay.meta()))
        s.gammas.append(1.0 + 0.1 * torch.randn(h, generator=g, device="cuda"))
    s.residual = torch.randn((t, h), generator=g, device="cuda")
    s.out = torch.empty_like(s.residual)
    s.normed = torch.empty_like(s.residual)
    if case["op"] == "prefill" and case["act"] == "bf16":
        s.x = s.x.to(torch.bfloat16)
    s.shared = None
    if case["shared"]:
        sl = synth.LayerLayout(h, case["shared"], 1, quant)
        s.shared = moe.allocate_moe_scratch(h, case["shared"], 1, 1, max(t, 16), moe.SIGMOID_GATE)
        s.shared_layer = s.shared.prepare_layer(synth.make_layer_blob(sl, seed * 64 + 63), sl.meta())
    return s


def run(s):
    op, sc = s.case["op"], s.scratch
    if s.case["layers"] > 1:
        s.out.copy_(s.x)  # the stack works in place on the residual stream
        if op == "prefill":
            return sc.stack_prefill(s.layers, s.gammas, s.out, EPS, s.normed)
        return sc.stack_decode(s.layers, s.gammas, s.out, EPS)
    layer = s.layers[0]
    if op == "prefill":
        out = moe.encode_moe_ffn_prefill_grouped(sc, layer, s.x, s.residual, s.out)
        return out if s.shared is None else s.shared.shared_expert_prefill(s.shared_layer, s.x, out)
    if op == "decode_norm":
        out = moe.encode_moe_ffn_decode_fused_norm(sc, layer, s.x, s.gammas[0], s.normed, s.out, EPS)
        return {"out": out, "normed": s.normed}
    out = moe.encode_moe_ffn_decode(sc, layer, s.x, s.residual, s.out)
    return out if s.shared is None else s.shared.shared_expert_decode(s.shared_layer, s.x, out)


def work(case):
    """Router weight, the matrices of the experts that some token selects (their expected number
    under uniform selection), activations in, residual in, output out."""
    h, i, e, k, t = (case[n] for n in ("hidden", "inter", "experts", "top_k", "tokens"))
    hit = e * (1.0 - (1.0 - k / e) ** t)
    act = 2 if case["act"] == "bf16" else 4
    per_layer = 4 * e * h + hit * 3 * i * h * BYTES[case["quant"]]
    flops = t * (2 * e * h + k * 6 * i * h)
    if case["shared"]:
        per_layer += 4 * h + 3 * case["shared"] * h * BYTES[case["quant"]]
        flops += t * (2 * h + 6 * case["shared"] * h)
    if case["layers"] > 1 or case["op"] == "decode_norm":
        per_layer += 4 * h  # the norm's weight
        rows = t * h * (8 if case["layers"] > 1 else 12)  # x in, out (and normed) out
    else:
        rows = t * h * (act + 8)
    return {"bytes": case["layers"] * per_layer + rows, "flops": case["layers"] * flops}


def tolerance(case):
    """Decode keeps f32-grade activations (two-term int8 against 4-bit weights, two-term f16 or bf16
    otherwise) and sums in f32; a prefill rounds its operands to f16 (2^-11) and sums in f32, and
    among thousands of tokens a few have two experts whose logits agree to rounding at the edge of
    the top-k: either is right, and the token's row then differs by that expert's small share."""
    if case["op"] == "prefill":
        return {"rel": 1e-3, "max": 0.15}
    return {"rel": 5e-5 if case["quant"] == "q4_0" else 1e-5, "max": 2e-3}
