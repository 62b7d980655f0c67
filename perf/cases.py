"""What this framework is measured on: the prompt pass, the decode step, the multi-token
verification step and the stand-alone operators, through their public entry points.

The architecture is the one of the repository's benchmark (hidden 2560, FFN 9728, 32 query / 8 kv
heads of 128, vocabulary 151936, bf16, random-init N(0, 0.02) weights with norm gains 1). A
program keeps one model for all its requests, so the weights are made once per process; what a
seed changes are the token ids, the keys and values already in the cache and the activations.

Depth: 12 layers of the benchmark's 36. A layer costs the same at any depth, and at 12 the
outputs (logits and every layer's key / value pages) can be compared: with random weights the
logits of two correct evaluations that add their products in another order drift apart by one
bf16 rounding per layer, 0.04 in the 2-norm after 36 layers and 0.02 after 12.
"""
from __future__ import annotations

import math

import torch

from starter_b200 import ops, weights
from starter_b200.decode import DecodeState

HIDDEN, INTER, VOCAB, N_Q, N_KV, HEAD = 2560, 9728, 151936, 32, 8, 128
LAYERS = 12
STEPS = 4                  # decode steps of one pass
DEVICE = "cuda"

_CONFIG = weights.ModelConfig(
    vocab=VOCAB, hidden=HIDDEN, inter=INTER, n_layers=LAYERS, n_q_heads=N_Q, n_kv_heads=N_KV,
    head_dim=HEAD, rms_eps=1e-6, rope_theta=1_000_000.0, tied=True, max_position=40960)
_model = None


def listed():
    return [
        # One token through one gate|up projection + SwiGLU: the smallest operator call, where the
        # host's share of a call counts.
        {"name": "linear_silu_mul_1", "kind": "linear_silu_mul", "rows": 1},
        # A chat turn of one user: the benchmark's default decode workload.
        {"name": "decode_1x1024", "kind": "decode", "batch": 1, "context": 1024},
        # A few users with an odd context (1-8 rows take the same kernels as one row).
        {"name": "decode_5x701", "kind": "decode", "batch": 5, "context": 701},
        # A served batch: the benchmark's second decode workload.
        {"name": "decode_32x2048", "kind": "decode", "batch": 32, "context": 2048},
        # The largest batch the step takes, contexts short and ragged.
        {"name": "decode_64x333", "kind": "decode", "batch": 64, "context": 333},
        # Time to first token of a short prompt: launches and the weight stream.
        {"name": "prompt_1x64", "kind": "prompt", "batch": 1, "context": 64},
        # ... of the benchmark's default prompt.
        {"name": "prompt_1x1024", "kind": "prompt", "batch": 1, "context": 1024},
        # Three requests of odd length admitted together.
        {"name": "prompt_3x701", "kind": "prompt", "batch": 3, "context": 701},
        # One long document: attention weighs as much as the projections.
        {"name": "prompt_1x7000", "kind": "prompt", "batch": 1, "context": 7000},
        # A batch of prompts as a server admits them: the largest piece of work.
        {"name": "prompt_12x2048", "kind": "prompt", "batch": 12, "context": 2048},
        # Speculative decoding for one user: four candidate tokens verified in one step.
        {"name": "verify_1x4x1024", "kind": "verify", "batch": 1, "tokens": 4, "context": 1024},
        # Verification attention over a long cache (the operator sweep's middle size).
        {"name": "attention_8x4x16384", "kind": "attention", "batch": 8, "tokens": 4, "context": 16384},
    ]


def _spread(rng, low, high):
    """A whole number in [low, high], spread evenly over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "prompt", "verify", "attention",
                       "linear_silu_mul"])
    if kind == "linear_silu_mul":
        return {"kind": kind, "rows": _spread(rng, 1, 64)}
    if kind == "decode":
        batch = _spread(rng, 1, 64)
        return {"kind": kind, "batch": batch, "context": _spread(rng, 64, min(16384, 65536 // batch))}
    if kind == "prompt":
        context = _spread(rng, 16, 8192)
        return {"kind": kind, "batch": _spread(rng, 1, max(1, min(32, 12 * 2048 // context // 2))), "context": context}
    if kind == "verify":
        tokens = rng.randint(2, 8)
        batch = _spread(rng, 1, 64 // tokens)
        return {"kind": kind, "batch": batch, "tokens": tokens,
                "context": _spread(rng, 64, min(16384, 65536 // batch))}
    return {"kind": kind, "batch": _spread(rng, 1, 8), "tokens": rng.randint(1, 8),
            "context": _spread(rng, 512, 32768)}


def _weights():
    """The process's one model."""
    global _model
    if _model is None:
        gen = torch.Generator(device=DEVICE).manual_seed(0)
        q, kv = N_Q * HEAD, N_KV * HEAD
        shape = {"q_proj": (q, HIDDEN), "k_proj": (kv, HIDDEN), "v_proj": (kv, HIDDEN), "o_proj": (HIDDEN, q),
                 "gate_proj": (INTER, HIDDEN), "up_proj": (INTER, HIDDEN), "down_proj": (HIDDEN, INTER),
                 "embed_tokens": (VOCAB, HIDDEN)}

        def get(name):
            part = name.split(".")[-2]
            if part in shape:
                w = torch.empty(shape[part], dtype=torch.bfloat16, device=DEVICE)
                return w.normal_(0.0, 0.02, generator=gen)
            return torch.ones(HEAD if part in ("q_norm", "k_norm") else HIDDEN, dtype=torch.bfloat16, device=DEVICE)

        _model = weights.pack(_CONFIG, get, lambda name: False, torch.device(DEVICE, torch.cuda.current_device()))
    return _model


def _normal(shape, gen):
    return torch.empty(shape, dtype=torch.bfloat16, device=DEVICE).normal_(generator=gen)


def _ids(shape, gen):
    return torch.randint(0, VOCAB, shape, generator=gen, device=DEVICE)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]
    if kind == "linear_silu_mul":
        w = torch.empty((2 * INTER, HIDDEN), dtype=torch.bfloat16, device=DEVICE).normal_(0.0, 0.02, generator=gen)
        return {"kind": kind, "x": _normal((case["rows"], HIDDEN), gen),
                "weight": weights.TiledWeight.pack(w, interleave8=True)}
    if kind == "attention":
        B, T, L = case["batch"], case["tokens"], case["context"]
        cache = ops.PagedKV(B, N_KV, L, DEVICE)
        cache.k.normal_(generator=gen)
        cache.v.normal_(generator=gen)
        return {"kind": kind, "cache": cache, "q": _normal((B * T, N_Q, HEAD), gen),
                "attn": ops.SmallQueryAttention(B, N_Q, N_KV, L, DEVICE, tokens_per_seq=T),
                "position": torch.full((1,), L - T, dtype=torch.int32, device=DEVICE)}
    B, L = case["batch"], case["context"]
    if kind == "prompt":
        state = DecodeState(_weights(), B, L, 1)
        return {"kind": kind, "state": state, "ids": _ids((B, L), gen)}
    # A sequence in the middle of its life: L tokens in the cache. After the key norm a key's
    # elements have variance 1, and so have the values with N(0, 0.02) weights at this width.
    T = case.get("tokens", 1)
    state = DecodeState(_weights(), B, L, STEPS, keep_logits=True, q_tokens=T)
    for pool in state.kpools + state.vpools:
        pool.normal_(generator=gen)
    state.position.fill_(L)
    if kind == "decode":
        state.tokens.copy_(_ids((B,), gen))
        state.capture()
        return {"kind": kind, "state": state, "tokens": _ids((STEPS, B), gen), "context": L}
    return {"kind": kind, "state": state, "candidates": _ids((B, T), gen)}


def run(state):
    kind, s = state["kind"], state.get("state")
    if kind == "linear_silu_mul":
        return ops.linear_silu_mul(state["x"], state["weight"])
    if kind == "attention":
        return state["attn"].run(state["q"], state["cache"], state["position"], HEAD ** -0.5)
    logits = s.logits
    if kind == "prompt":
        logits = s.prefill(state["ids"])
    elif kind == "verify":
        s.verify(state["candidates"])
    else:
        # a program that picks each token from the logits by itself and writes it into the state
        s.position.fill_(state["context"])
        for tokens in state["tokens"]:
            s.tokens.copy_(tokens)
            s.advance()
    # (the picked tokens follow from the logits, and differ where two of them tie)
    return {"logits": logits, "keys": s.kpools, "values": s.vpools}


def work(case):
    kind = case["kind"]
    if kind == "linear_silu_mul":
        M, N, K = case["rows"], 2 * INTER, HIDDEN
        return {"bytes": 2.0 * (N * K + M * K + M * N // 2), "flops": 2.0 * M * N * K}
    B, L, T = case["batch"], case["context"], case.get("tokens", 1)
    if kind == "attention":
        keys = sum(L - T + t + 1 for t in range(T))
        return {"bytes": 4.0 * B * N_KV * HEAD * L + 4.0 * B * T * N_Q * HEAD, "flops": 4.0 * B * N_Q * HEAD * keys}
    layer = (N_Q + 2 * N_KV) * HEAD * HIDDEN + HIDDEN * N_Q * HEAD + 3 * INTER * HIDDEN
    kv_row = 2 * N_KV * HEAD * 2                               # bytes of one token's keys and values in a layer
    head = VOCAB * HIDDEN
    if kind == "prompt":
        pairs = B * L * (L + 1) / 2
        return {"bytes": 2.0 * (LAYERS * layer + head + B * L * HIDDEN + B * VOCAB) + LAYERS * kv_row * B * L,
                "flops": 2.0 * LAYERS * layer * B * L + 4.0 * LAYERS * N_Q * HEAD * pairs + 2.0 * head * B}
    passes = STEPS if kind == "decode" else 1
    total = {"bytes": 0.0, "flops": 0.0}
    for step in range(passes):
        first = L + step                                       # position of the pass's first token
        total["bytes"] += (2.0 * (LAYERS * layer + head + B * T * VOCAB)
                           + LAYERS * kv_row * B * (first + T))
        total["flops"] += (2.0 * B * T * (LAYERS * layer + head)
                           + 4.0 * LAYERS * N_Q * HEAD * B * sum(first + t + 1 for t in range(T)))
    return total


def tolerance(case):
    if case["kind"] in ("linear_silu_mul", "attention"):
        # one rounding of the sums to bf16 (and of the probabilities or of silu before it): 2^-9
        return {"rel": 6e-3, "max": 2e-2}
    return {"rel": 3e-2, "max": 4e-1}
