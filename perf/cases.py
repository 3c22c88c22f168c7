"""The work that a user of this package has it do, as cases that can be timed and compared.

Kinds of cases:
  decode       one decode step of a stack of MoE layers (W4A16, 1..16 tokens): `Weights.forward` once per layer, each layer with
               its own weights, as a model's layers have (the weights of a step do not stay in L2 from one step to the next)
  decode_host  the same for a program that holds its tensors in page-locked host memory: `Weights.forward_host`
  mid          one W4A16 layer call for 17..256 tokens (small prefill chunks, large decode batches) after `enable_mid`
  prefill      one W4A4 layer call for 17..8192 tokens after `enable_prefill`
  quantize     a batch of activations to NVFP4: `quantize_nvfp4` (own global scale, row-major block scales) or
               `quantize_nvfp4_128x4` (calibrated global scale, swizzled block scales)
  quantize_experts  the expert matrices of one projection to NVFP4 at load time: `quantize_nvfp4_experts`

Layer inputs: weights N(0, 0.02) in bf16, quantised per expert; hidden states N(0, 1) in bf16 (what a layer sees after its
norm); router logits N(0, 1) -> softmax -> top-k -> renormalised. routing "random": that; "skewed": with a bias per expert of
standard deviation 1.5 (some experts are hot, some are cold); "same": every token on the same evenly spaced top_k experts."""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

import sm120fp4_b200 as fp4
from sm120fp4_b200.vllm_backend import Weights

QWEN = dict(experts=128, hidden=2048, inter=768, top_k=8)
GEMMA = dict(experts=128, hidden=2816, inter=704, top_k=8)
WIDE = dict(experts=128, hidden=4096, inter=1536, top_k=8)     # a larger model's layer: hidden size above 3072

MOST_WEIGHTS = WIDE["experts"] * WIDE["hidden"] * WIDE["inter"]


def listed():
    return [
        # one user typing: the smallest step, latency and launches
        dict(name="decode_m1", kind="decode", **QWEN, tokens=1, layers=4, routing="random"),
        # a few users, a shape that is no power of two
        dict(name="decode_m4_gemma", kind="decode", **GEMMA, tokens=4, layers=4, routing="random"),
        # a served batch: the largest decode step of one launch
        dict(name="decode_m16", kind="decode", **QWEN, tokens=16, layers=4, routing="random"),
        # a larger model's layers, medium batch
        dict(name="decode_m8_wide", kind="decode", **WIDE, tokens=8, layers=2, routing="random"),
        # an engine whose tensors live in host memory (speculative drafts of two tokens)
        dict(name="host_m2", kind="decode_host", **QWEN, tokens=2, layers=4, routing="random"),
        # a large decode batch, or a short prompt, on a checkpoint without activation scales
        dict(name="mid_m96", kind="mid", **QWEN, tokens=96, routing="random"),
        # one prompt of odd length, hot and cold experts
        dict(name="prefill_m333_gemma", kind="prefill", **GEMMA, tokens=333, routing="skewed"),
        # a prefill chunk
        dict(name="prefill_m1024", kind="prefill", **QWEN, tokens=1024, routing="random"),
        # the largest prefill chunk
        dict(name="prefill_m8192", kind="prefill", **QWEN, tokens=8192, routing="random"),
        # a ragged chunk of a larger model
        dict(name="prefill_m2050_wide", kind="prefill", **WIDE, tokens=2050, routing="random"),
        # a decode-sized batch of activations quantised by itself
        dict(name="quantize_m16", kind="quantize", rows=16, hidden=2048, dtype="bf16", layout="linear"),
        # a layer's gate and up weights quantised at load time
        dict(name="quantize_experts", kind="quantize_experts", experts=128, rows=1536, hidden=2048, dtype="bf16", swizzle=True),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def _draw_shape(rng):
    if rng.random() < 0.5:
        return dict(rng.choice([QWEN, QWEN, GEMMA, WIDE]))
    while True:
        s = dict(experts=rng.choice([16, 32, 60, 64, 96, 128, 256]), hidden=128 * _log_int(rng, 8, 32), inter=64 * _log_int(rng, 6, 24),
                 top_k=rng.choice([2, 4, 6, 8]))
        if s["experts"] * s["hidden"] * s["inter"] <= MOST_WEIGHTS:
            return s


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "decode_host", "mid", "prefill", "prefill", "prefill", "quantize", "quantize_experts"])
    routing = rng.choice(["random", "random", "random", "skewed", "skewed", "same"])
    if kind in ("decode", "decode_host"):
        s = _draw_shape(rng)
        most = max(1, min(4, 2 * MOST_WEIGHTS // (s["experts"] * s["hidden"] * s["inter"])))
        return dict(kind=kind, **s, tokens=_log_int(rng, 1, 16), layers=rng.randint(1, most), routing=routing)
    if kind == "mid":
        s = _draw_shape(rng)
        s["hidden"] = min(s["hidden"], 3072)   # the one-call path takes hidden and intermediate sizes up to 3072
        return dict(kind=kind, **s, tokens=_log_int(rng, 17, 256), routing=routing)
    if kind == "prefill":
        s = _draw_shape(rng)
        most = min(8192, int(8192 * 8 * QWEN["hidden"] * QWEN["inter"] / (s["top_k"] * s["hidden"] * s["inter"])))   # no dearer than the largest listed case
        return dict(kind=kind, **s, tokens=_log_int(rng, 17, most), routing=routing)
    if kind == "quantize":
        return dict(kind=kind, rows=_log_int(rng, 1, 8192), hidden=64 * _log_int(rng, 8, 64), dtype=rng.choice(["bf16", "bf16", "f32"]),
                    layout=rng.choice(["linear", "128x4"]))
    return dict(kind=kind, experts=rng.choice([8, 16, 60, 64, 128]), rows=64 * _log_int(rng, 6, 24), hidden=64 * _log_int(rng, 12, 32),
                dtype=rng.choice(["bf16", "bf16", "f32"]), swizzle=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------------------ inputs
def _generator(seed, part):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + part)


def _normal(g, shape, std, dtype):
    t = torch.empty(shape, dtype=dtype, device="cuda")
    return t.normal_(0.0, std, generator=g)


def _route(g, tokens, experts, top_k, routing):
    if routing == "same":
        ids = (torch.arange(top_k, dtype=torch.int32, device="cuda") * (experts // top_k)).repeat(tokens, 1).contiguous()
        return ids, torch.full((tokens, top_k), 1.0 / top_k, dtype=torch.float32, device="cuda")
    logits = torch.randn(tokens, experts, generator=g, device="cuda")
    if routing == "skewed":
        logits += 1.5 * torch.randn(experts, generator=g, device="cuda")
    wts, ids = torch.topk(torch.softmax(logits, dim=-1), top_k, dim=-1)
    return ids.to(torch.int32).contiguous(), (wts / wts.sum(-1, keepdim=True)).float().contiguous()


def _layer(case, g):
    e, h, i = case["experts"], case["hidden"], case["inter"]
    q1, s1, g1 = fp4.quantize_nvfp4_experts(_normal(g, (e, 2 * i, h), 0.02, torch.bfloat16))
    q2, s2, g2 = fp4.quantize_nvfp4_experts(_normal(g, (e, h, i), 0.02, torch.bfloat16))
    w = Weights(q1, s1, 1.0 / g1, q2, s2, 1.0 / g2, case["top_k"])
    if case["kind"] == "prefill":
        w.enable_prefill()
    if case["kind"] == "mid":
        w.enable_mid()
    return w


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("quantize", "quantize_experts"):
        g = _generator(seed, 0)
        dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        if kind == "quantize":
            x = _normal(g, (case["rows"], case["hidden"]), 1.0, dtype)
            return SimpleNamespace(case=case, x=x, gs=fp4.global_scale_for(x) if case["layout"] == "128x4" else None)
        return SimpleNamespace(case=case, w=_normal(g, (case["experts"], case["rows"], case["hidden"]), 0.02, dtype))
    calls = []
    for n in range(case.get("layers", 1)):
        g = _generator(seed, n)
        w = _layer(case, g)
        x = _normal(g, (case["tokens"], case["hidden"]), 1.0, torch.bfloat16)
        ids, wts = _route(g, case["tokens"], case["experts"], case["top_k"], case["routing"])
        if kind == "decode_host":
            host = [t.cpu().pin_memory() for t in (x, ids, wts)]
            calls.append((w, *host, torch.empty_like(host[0]).pin_memory()))
        else:
            calls.append((w, x, ids, wts))
    return SimpleNamespace(case=case, calls=calls)


def run(state):
    kind = state.case["kind"]
    if kind == "decode_host":
        return [w.forward_host(x, ids, wts, out) for w, x, ids, wts, out in state.calls]
    if kind == "quantize":
        return fp4.quantize_nvfp4(state.x) if state.case["layout"] == "linear" else fp4.quantize_nvfp4_128x4(state.x, state.gs)
    if kind == "quantize_experts":
        return fp4.quantize_nvfp4_experts(state.w, swizzle=state.case["swizzle"])
    return [w.forward(x, ids, wts) for w, x, ids, wts in state.calls]


# ------------------------------------------------------------------------------------------------------------ what a pass needs
def _touched(case):
    """Experts that a batch of this case reaches: the mean over three batches."""
    if case["routing"] == "same":
        return case["top_k"]
    n = 0.0
    for seed in range(3):
        g = torch.Generator().manual_seed(seed)
        logits = torch.randn(case["tokens"], case["experts"], generator=g)
        if case["routing"] == "skewed":
            logits += 1.5 * torch.randn(case["experts"], generator=g)
        n += torch.topk(logits, case["top_k"], dim=-1).indices.unique().numel() / 3.0
    return n


def work(case):
    kind = case["kind"]
    if kind in ("quantize", "quantize_experts"):
        n = case.get("experts", 1) * case["rows"] * case["hidden"]
        return {"bytes": n * ((2 if case["dtype"] == "bf16" else 4) + 0.5 + 1 / 16), "flops": 0}
    h, i, m, k = case["hidden"], case["inter"], case["tokens"], case["top_k"]
    layers = case.get("layers", 1)
    weights = _touched(case) * 3 * h * i * (1 / 2 + 1 / 16)
    return {"bytes": layers * (weights + m * h * 4 + m * k * 8), "flops": layers * 6.0 * m * k * h * i}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "quantize_experts"):
        return "exact"                            # codes, scales and global scales follow one fixed order of operations
    if kind == "prefill":
        return {"rel": 1e-2, "max": 1e-1}         # bf16 results; an activation on the edge of two FP4 codes may take either
    return {"rel": 5e-3, "max": 5e-2}             # bf16 results, 16-bit activations, 32-bit sums
