"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is a dict of plain values.  `kind` says which public entry point it goes through:

  linear     ops.int4_linear                        one INT4 weight-only linear layer
  attention  ops.flash_attn / flash_attn_kv_view    prefill: several query positions per sequence
  decode     ops.flash_attn_decode                  one query position against a static KV cache
  quantize   quantize.quantize_weight               a linear's weight to INT4, once per layer at model load
  generate   LlamaInt4Decoder.prefill + .decode     a prompt and a greedy continuation of a whole model
"""

import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("kernel-forge_b200"))

from kernelforge import ops, quantize  # noqa: E402
from kernelforge.llama_decode import LlamaInt4Decoder, LlamaShape  # noqa: E402

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
BYTES = {"fp16": 2, "bf16": 2, "fp32": 4}


def listed():
    return [
        # One token of one user through the gate projection of a 2048-wide model: the smallest call there is, and the
        # one that a decode loop written against the operators makes more often than any other.
        dict(name="linear_token", kind="linear", m=1, n=5632, k=2048, group=128, dtype="fp16", bias=False),
        # A decode batch of 16 users through a down projection: few rows, a long reduction.
        dict(name="linear_batch", kind="linear", m=16, n=1536, k=8960, group=128, dtype="fp16", bias=False),
        # A short prompt (an odd number of tokens) through a query projection with a bias, in the finer group size.
        dict(name="linear_prompt", kind="linear", m=131, n=1536, k=1536, group=64, dtype="fp16", bias=True),
        # A chunk of a prompt through a gate projection with bf16 activations.
        dict(name="linear_chunk_bf16", kind="linear", m=1000, n=8960, k=1536, group=128, dtype="bf16", bias=False),
        # The prompts of a whole batch through a fused gate / up projection: compute-bound prefill.
        dict(name="linear_prefill", kind="linear", m=4096, n=11264, k=2048, group=128, dtype="fp16", bias=False),
        # Full (non-causal) attention over two sequences, as in an encoder.
        dict(name="attention_full", kind="attention", b=2, h=16, hk=16, nq=2048, nk=2048, d=64, dtype="fp16", causal=False,
             capacity=0),
        # Chunked prefill: the next 509 tokens of one sequence against the 4093 that its cache holds then, grouped
        # queries, K and V read in place from a static cache.
        dict(name="attention_chunk", kind="attention", b=1, h=12, hk=2, nq=509, nk=4093, d=128, dtype="bf16", causal=True,
             capacity=8192),
        # Causal prefill of two long prompts.
        dict(name="attention_long", kind="attention", b=2, h=16, hk=16, nq=8192, nk=8192, d=128, dtype="fp16", causal=True,
             capacity=0),
        # One decode step of a serving batch: eight sequences of different lengths in one static cache.
        dict(name="decode_batch", kind="decode", b=8, h=32, hk=4, d=64, shortest=1000, longest=4096, capacity=4608, dtype="fp16"),
        # Loading a model: a fused gate / up weight to INT4.
        dict(name="quantize_layer", kind="quantize", n=11264, k=2048, group=128, dtype="fp16"),
        # One user's request: a 512-token prompt, then 32 greedy tokens.
        dict(name="generate_one", kind="generate", b=1, prompt=512, steps=32, layers=22),
        # A batch of requests: 32 prompts of 200 tokens, then 24 greedy tokens each.
        dict(name="generate_batch", kind="generate", b=32, prompt=200, steps=24, layers=22),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choices(("linear", "attention", "decode", "quantize", "generate"), (5, 4, 2, 1, 1))[0]
    if kind == "linear":
        group = rng.choice((64, 128, 128))
        while True:
            m, n, k = _log(rng, 1, 4096), _log(rng, 256, 16384), group * _log(rng, 1024 // group, 12288 // group)
            if m * n * k <= 4096 * 11264 * 2048:
                break
        n = n if rng.random() < 0.15 else -(-n // 64) * 64    # nearly every linear's width is a round number
        return dict(kind=kind, m=m, n=n, k=k, group=group, dtype=rng.choice(("fp16", "fp16", "bf16")), bias=rng.random() < 0.4)
    if kind == "attention":
        while True:
            hk, g, d, causal = rng.choice((1, 2, 4, 8, 16)), rng.choice((1, 1, 4, 6, 8)), rng.choice((64, 128)), rng.random() < 0.7
            b, nq = _log(rng, 1, 16), _log(rng, 2, 8192)
            nk = nq if rng.random() < 0.6 else min(16384, nq + _log(rng, 1, 8192))    # a prompt, or a chunk behind a cache
            if hk * g <= 32 and 4 * b * hk * g * nq * nk * d * (0.5 if causal else 1) <= 4 * 2 * 16 * 8192 * 8192 * 128 * 0.5:
                break
        capacity = 64 * -(-(nk + rng.randrange(2048)) // 64) if rng.random() < 0.4 else 0
        return dict(kind=kind, b=b, h=hk * g, hk=hk, nq=nq, nk=nk, d=d, dtype=rng.choice(("fp16", "bf16")), causal=causal,
                    capacity=capacity)
    if kind == "decode":
        b, longest = _log(rng, 1, 64), _log(rng, 64, 16384)
        longest = min(longest, 64 * 4096 // b)
        hk = rng.choice((2, 4, 8))
        return dict(kind=kind, b=b, h=hk * rng.choice((1, 4, 6, 8)), hk=hk, d=rng.choice((64, 128)),
                    shortest=max(1, round(longest * rng.uniform(0.2, 1.0))), longest=longest,
                    capacity=64 * -(-(longest + rng.randrange(1, 1024)) // 64), dtype=rng.choice(("fp16", "bf16")))
    if kind == "quantize":
        group = rng.choice((64, 128))
        return dict(kind=kind, n=_log(rng, 256, 11264), k=group * _log(rng, 512 // group, 2048 // group), group=group,
                    dtype=rng.choice(("fp16", "bf16", "fp32")))
    b = _log(rng, 1, 32)
    return dict(kind=kind, b=b, prompt=_log(rng, 16, min(768, 32 * 200 // b)), steps=rng.randint(8, 24), layers=rng.choice((11, 22)))


def _lengths(case):
    """The valid cache rows of each sequence: spread evenly from the shortest to the longest."""
    b = case["b"]
    return [case["shortest"] + (case["longest"] - case["shortest"]) * i // max(1, b - 1) for i in range(b - 1)] + [case["longest"]]


def _model(shape, seed):
    """Random weights of a Llama-architecture model.  Layers as initialised; the output rows are the input embeddings
    in another order, so that the model is sure of its next token, as a trained one mostly is, and greedy decoding
    does not hang on the last bit of a logit."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rn(rows, cols, std=0.02):
        return torch.randn(rows, cols, generator=g, device="cuda", dtype=torch.float16) * std

    s, ones = shape, torch.ones(shape.hidden, device="cuda")
    qd, kd = s.heads * s.head_dim, s.kv_heads * s.head_dim
    embed = rn(s.vocab, s.hidden, 1.0)
    order = torch.randperm(s.vocab, generator=g, device="cuda")
    layers = [{"in_norm": ones, "post_norm": ones, "q": rn(qd, s.hidden), "k": rn(kd, s.hidden), "v": rn(kd, s.hidden),
               "o": rn(s.hidden, qd), "gate": rn(s.intermediate, s.hidden), "up": rn(s.intermediate, s.hidden),
               "down": rn(s.hidden, s.intermediate)} for _ in range(s.layers)]
    return {"embed": embed, "lm_head": embed[order] * 0.02, "final_norm": ones, "layers": layers}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case.get("dtype", "fp16")]

    def rn(*size):
        return torch.randn(*size, generator=g, device="cuda", dtype=dtype)

    kind = case["kind"]
    if kind == "linear":
        qw = quantize.quantize_weight(rn(case["n"], case["k"]).half() * 0.02, case["group"])
        bias = rn(case["n"]) * 0.1 if case["bias"] else None
        return dict(kind=kind, x=rn(case["m"], case["k"]), packed=qw.packed, scales=qw.scales, group=case["group"], bias=bias)
    if kind == "attention":
        b, h, hk, nq, nk, d = (case[n] for n in ("b", "h", "hk", "nq", "nk", "d"))
        k, v = rn(b, hk, case["capacity"] or nk, d), rn(b, hk, case["capacity"] or nk, d)
        return dict(kind=kind, q=rn(b, h, nq, d), k=k, v=v, nk=nk, causal=case["causal"], cached=case["capacity"] > 0)
    if kind == "decode":
        b, h, hk, d = (case[n] for n in ("b", "h", "hk", "d"))
        lengths = torch.tensor(_lengths(case), dtype=torch.int32, device="cuda")
        return dict(kind=kind, q=rn(b, h, 1, d), k=rn(b, hk, case["capacity"], d), v=rn(b, hk, case["capacity"], d), lengths=lengths)
    if kind == "quantize":
        return dict(kind=kind, weight=rn(case["n"], case["k"]) * 0.02, group=case["group"])
    shape = LlamaShape(layers=case["layers"])
    model = LlamaInt4Decoder(shape, _model(shape, seed), "cuda", batch=case["b"], max_len=case["prompt"] + case["steps"] + 1)
    model.capture()
    ids = torch.randint(0, shape.vocab, (case["b"], case["prompt"]), generator=g, device="cuda")
    return dict(kind=kind, model=model, ids=ids, steps=case["steps"])


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return ops.int4_linear(state["x"], state["packed"], state["scales"], state["group"], state["bias"])
    if kind == "attention":
        if state["cached"]:
            nk = state["nk"]
            return ops.flash_attn_kv_view(state["q"], state["k"][:, :, :nk], state["v"][:, :, :nk], causal=state["causal"])
        return ops.flash_attn(state["q"], state["k"], state["v"], causal=state["causal"])
    if kind == "decode":
        return ops.flash_attn_decode(state["q"], state["k"], state["v"], state["lengths"])
    if kind == "quantize":
        qw = quantize.quantize_weight(state["weight"], state["group"])
        return qw.packed, qw.scales
    model = state["model"]
    prompt_logits = model.prefill(state["ids"])
    tokens, _ = model.decode(state["steps"])
    return {"tokens": tokens, "prompt_logits": prompt_logits, "last_logits": model.step_logits, "k_cache": model.k_cache,
            "v_cache": model.v_cache}


def work(case):
    kind, size = case["kind"], BYTES[case.get("dtype", "fp16")]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        weight = n * k // 2 + n * (k // case["group"]) * 2
        return {"bytes": weight + size * (m * k + m * n + (n if case["bias"] else 0)), "flops": 2 * m * n * k}
    if kind == "attention":
        b, h, hk, nq, nk, d = (case[n] for n in ("b", "h", "hk", "nq", "nk", "d"))
        seen = nq * (nk - nq) + nq * (nq + 1) // 2 if case["causal"] else nq * nk
        return {"bytes": size * (2 * b * h * nq * d + 2 * b * hk * nk * d), "flops": 4 * b * h * seen * d}
    if kind == "decode":
        rows = sum(_lengths(case))
        return {"bytes": size * (2 * case["hk"] * rows * case["d"] + 2 * case["b"] * case["h"] * case["d"]),
                "flops": 4 * case["h"] * rows * case["d"]}
    if kind == "quantize":
        n, k = case["n"], case["k"]
        return {"bytes": size * n * k + n * k // 2 + 2 * n * (k // case["group"]), "flops": 2 * n * k}
    s, b, t, steps = LlamaShape(layers=case["layers"]), case["b"], case["prompt"], case["steps"]
    qd, kd = s.heads * s.head_dim, s.kv_heads * s.head_dim
    linear = s.layers * (s.hidden * (qd + 2 * kd) + qd * s.hidden + 3 * s.hidden * s.intermediate)
    head = s.vocab * s.hidden
    weights = linear // 2 + linear // 128 * 2 + 2 * head
    row = 2 * 2 * s.layers * kd     # K and V of one position
    cached = sum(t + i + 1 for i in range(steps))
    read = weights * (1 + steps) + row * b * cached
    written = row * b * (t + steps) + 2 * b * t * s.vocab + 2 * b * steps * s.vocab
    attention = 4 * s.layers * b * qd * (t * (t + 1) // 2 + cached)
    return {"bytes": read + written, "flops": 2 * (linear + head) * b * (t + steps) + attention}


def tolerance(case):
    kind = case["kind"]
    if kind == "quantize":
        return "exact"
    if kind == "generate":      # fp16 activations through all layers; the tokens themselves have to agree
        return {"rel": 1e-2, "max": 0.2, "differ": 0.0}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
