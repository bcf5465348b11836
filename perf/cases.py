"""What programs have this package do, as cases that can be timed: single quantized layers, one expert, one MoE block,
and a decoder's steps through its model classes.

Shapes are the ones the package is built around (hidden 4096, experts of 14336, 32 query and 8 key/value heads of 128,
8 experts of which 2 are routed to; experts 2-bit in groups of 16, attention 4-bit in groups of 64, 3-bit layers in
groups of 64); drawn layers take other multiples of 1024.  A decoder has a few layers instead of 32: they are all alike.
Weights are N(0, 0.02^2), as everywhere in this repository, quantized through the package's own constructors; the two
projections that add to the residual stream (o and w2) are scaled down by sqrt(2 * 32), the usual initialisation of a
32-layer decoder, so that the stream stays in the range a trained model keeps it in.  A token carries a component of
the two experts it is routed to, so that routing is as decided as a trained router's.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch
from torch import nn

from mixtral_offloading_b200 import (AttentionDecode, BaseQuantizeConfig, BatchDecode, DecoderLayerDecode, ExpertCache,
                                     HQQLinearTritonSavable, MixtralDecodeModel, MixtralExpertWrapper,
                                     MixtralOffloadModel, QuantConfig, ResidentMoe, SparseMoeWrapper, make_empty_expert)

HIDDEN, FFN, EXPERTS, VOCAB = 4096, 14336, 8, 32000
HEADS, KV_HEADS, HEAD_DIM = 32, 8, 128
GROUP = {2: 16, 3: 64, 4: 64}
STD, RESIDUAL_STD = 0.02, 0.02 / math.sqrt(2 * 32)
DEVICE = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
CONFIG = SimpleNamespace(hidden_size=HIDDEN, intermediate_size=FFN, num_local_experts=EXPERTS, num_experts_per_tok=2,
                         hidden_act="silu")


def listed():
    return [
        # The smallest call: one row through a key (or value) projection, as a decoder that calls layer by layer does.
        {"name": "linear_4bit_1_row", "kind": "linear", "nbits": 4, "n": 1024, "k": 4096, "rows": 1, "dtype": "bf16"},
        # A query or output projection for a small batch of sequences.
        {"name": "linear_4bit_16_rows", "kind": "linear", "nbits": 4, "n": 4096, "k": 4096, "rows": 16, "dtype": "bf16"},
        # The 3-bit format at decode.
        {"name": "linear_3bit_1_row", "kind": "linear", "nbits": 3, "n": 14336, "k": 4096, "rows": 1, "dtype": "bf16"},
        # The 3-bit format for a short prompt, from a half-precision host (what the package replaces is fp16 throughout).
        {"name": "linear_3bit_100_rows", "kind": "linear", "nbits": 3, "n": 14336, "k": 4096, "rows": 100, "dtype": "fp16"},
        # One expert on the few rows that a batch of sequences routes to it.
        {"name": "expert_3_rows", "kind": "expert", "rows": 3, "dtype": "bf16"},
        # One expert on the rows of a long prompt: the most a single expert is given at once.
        {"name": "expert_512_rows", "kind": "expert", "rows": 512, "dtype": "bf16"},
        # A whole MoE block with resident experts for a short prompt of a length that fits nothing.
        {"name": "moe_block_33_tokens", "kind": "moe", "tokens": 33, "dtype": "bf16"},
        # One greedy decode step at batch 1 behind 512 cached positions: the case the framework exists for.
        {"name": "decode_1_sequence", "kind": "decode", "layers": 8, "context": 512},
        # One decode step of eight sequences.
        {"name": "decode_8_sequences", "kind": "batch", "layers": 4, "sequences": 8, "context": 512},
        # A prompt in one pass.
        {"name": "prompt_500_tokens", "kind": "prompt", "layers": 4, "tokens": 500},
        # Decoding with half of every layer's experts in host memory (least-recently-used swaps).
        {"name": "offloaded_6_tokens", "kind": "offload", "layers": 2, "tokens": 6, "context": 64},
        # The full weight, for a host that multiplies with its own kernels.
        {"name": "dequantize_2bit", "kind": "dequantize", "nbits": 2, "n": 14336, "k": 4096, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "expert", "moe", "decode", "batch", "prompt", "offload", "dequantize"))
    dtype = rng.choice(("bf16", "bf16", "bf16", "fp16"))
    if kind in ("linear", "dequantize"):
        case = {"kind": kind, "nbits": rng.choice((2, 3, 4)), "n": 1024 * _log_int(rng, 1, 14), "k": 1024 * _log_int(rng, 1, 14)}
        if kind == "linear":
            return dict(case, rows=_log_int(rng, 1, 512), dtype=dtype)
        return dict(case, dtype=rng.choice(("bf16", "fp16", "fp32")))
    if kind == "expert":
        return {"kind": kind, "rows": _log_int(rng, 1, 512), "dtype": dtype}
    if kind == "moe":
        return {"kind": kind, "tokens": _log_int(rng, 1, 512), "dtype": dtype}
    if kind == "decode":
        return {"kind": kind, "layers": rng.randint(2, 8), "context": _log_int(rng, 1, 4000)}
    if kind == "batch":
        return {"kind": kind, "layers": rng.randint(1, 4), "sequences": rng.randint(2, 16), "context": _log_int(rng, 1, 2000)}
    if kind == "prompt":
        return {"kind": kind, "layers": rng.randint(1, 4), "tokens": _log_int(rng, 17, 511)}
    return {"kind": kind, "layers": rng.randint(1, 2), "tokens": rng.randint(2, 8), "context": _log_int(rng, 1, 500)}


# ---- building blocks, through the package's constructors -------------------------------------------------------------
def _quant(nbits):
    return BaseQuantizeConfig(nbits=nbits, group_size=GROUP[nbits], quant_zero=True, quant_scale=True)


QUANT = QuantConfig(ffn_config=_quant(2), attn_config=_quant(4))


def _normal(gen, *shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=gen, device=DEVICE, dtype=dtype).mul_(std)


def _fill(layer, gen, std=STD):
    layer.quantize(_normal(gen, *layer.meta["shape"], std=std), **layer.quant_config)
    return layer


def _linear(gen, n, k, nbits, std=STD):
    cfg = _quant(nbits)
    return _fill(HQQLinearTritonSavable(None, cfg, HQQLinearTritonSavable.get_hqq_meta((k, n), cfg)), gen, std)


def _expert(gen):
    expert = make_empty_expert(CONFIG, QUANT)
    _fill(expert.w1, gen), _fill(expert.w2, gen, RESIDUAL_STD), _fill(expert.w3, gen)
    return MixtralExpertWrapper(expert, torch.device(DEVICE, torch.cuda.current_device()))


def _directions(gen):
    """One unit vector of the hidden space per expert."""
    return torch.nn.functional.normalize(_normal(gen, EXPERTS, HIDDEN, dtype=torch.float32), dim=1)


def _gate(gen, directions):
    """A router that answers to the experts' directions, every layer with an assignment of its own."""
    order = torch.randperm(EXPERTS, generator=gen, device=DEVICE)
    gate = nn.Linear(HIDDEN, EXPERTS, bias=False, dtype=torch.bfloat16, device=DEVICE)
    gate.weight.data = (0.25 * directions[order] + _normal(gen, EXPERTS, HIDDEN, std=0.002, dtype=torch.float32)).to(torch.bfloat16)
    return gate


def _tokens(gen, directions, count):
    """(count, hidden): noise plus the directions of two different experts, one about twice as strong as the other."""
    pick = torch.rand(count, EXPERTS, generator=gen, device=DEVICE).topk(2, dim=1).indices
    strength = torch.zeros(count, EXPERTS, device=DEVICE)
    strength.scatter_(1, pick, torch.tensor([[17.0, 9.0]], device=DEVICE).expand(count, 2))
    return (_normal(gen, count, HIDDEN, dtype=torch.float32) + strength @ directions).to(torch.bfloat16)


def _norm_weight(gen):
    return (1.0 + _normal(gen, HIDDEN, std=0.1, dtype=torch.float32)).to(torch.bfloat16)


def _attention(gen, max_len):
    return AttentionDecode(_linear(gen, HEADS * HEAD_DIM, HIDDEN, 4), _linear(gen, KV_HEADS * HEAD_DIM, HIDDEN, 4),
                           _linear(gen, KV_HEADS * HEAD_DIM, HIDDEN, 4), _linear(gen, HIDDEN, HEADS * HEAD_DIM, 4, RESIDUAL_STD),
                           _norm_weight(gen), _norm_weight(gen), HEADS, KV_HEADS, HEAD_DIM, max_len)


def _decoder(gen, layers, max_len):
    directions = _directions(gen)
    attentions = [_attention(gen, max_len) for _ in range(layers)]
    final_ln = _norm_weight(gen)
    blocks = []
    for l, attention in enumerate(attentions):
        moe = ResidentMoe(CONFIG, l, _gate(gen, directions), [_expert(gen) for _ in range(EXPERTS)])
        blocks.append(DecoderLayerDecode(attention, moe, attentions[l + 1].ln_in if l + 1 < layers else final_ln))
    return MixtralDecodeModel(_tokens(gen, directions, VOCAB), blocks, attentions[0].ln_in, _normal(gen, VOCAB, HIDDEN, std=STD))


def _fill_caches(gen, caches, context):
    """Keys and values of `context` earlier positions, nothing behind them."""
    for cache in caches:
        cache.zero_()
        cache[..., :context, :] = _normal(gen, *cache.shape[:-2], context, cache.shape[-1])


def _ids(gen, count):
    return torch.randint(0, VOCAB, (count,), generator=gen, device=DEVICE)


# ---- the cases ---------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        layer = _linear(gen, case["n"], case["k"], case["nbits"])
        return {"case": case, "layer": layer, "x": _normal(gen, case["rows"], case["k"]).to(DTYPES[case["dtype"]])}
    if kind == "dequantize":
        return {"case": case, "layer": _linear(gen, case["n"], case["k"], case["nbits"])}
    if kind == "expert":
        return {"case": case, "expert": _expert(gen), "x": _normal(gen, case["rows"], HIDDEN).to(DTYPES[case["dtype"]])}
    if kind == "moe":
        directions = _directions(gen)
        block = ResidentMoe(CONFIG, 0, _gate(gen, directions), [_expert(gen) for _ in range(EXPERTS)])
        x = _tokens(gen, directions, case["tokens"]).view(1, case["tokens"], HIDDEN).to(DTYPES[case["dtype"]])
        return {"case": case, "block": block, "x": x}
    if kind == "prompt":
        model = _decoder(gen, case["layers"], case["tokens"] + 128)
        return {"case": case, "model": model, "prompt": _ids(gen, case["tokens"]).tolist()}
    if kind == "decode":
        model = _decoder(gen, case["layers"], case["context"] + 128)
        model.position.fill_(case["context"])
        model.capture()
        _fill_caches(gen, [c for l in model.layers for c in (l.attention.k_cache, l.attention.v_cache)], case["context"])
        return {"case": case, "model": model, "token": _ids(gen, 1)}
    if kind == "batch":
        model = _decoder(gen, case["layers"], 8)                    # the sequences' caches are the batch's own
        batch = BatchDecode(model, case["sequences"], case["context"] + 128)
        tokens = _ids(gen, case["sequences"])
        batch.step(tokens, case["context"])
        batch.capture()
        _fill_caches(gen, batch.k_caches + batch.v_caches, case["context"])
        return {"case": case, "batch": batch, "tokens": tokens}
    # "offload": half of every layer's experts on the device, half in host memory
    layers, directions = case["layers"], _directions(gen)
    cache = ExpertCache(lambda: _expert(gen), main_size=layers * EXPERTS // 2, offload_size=layers * EXPERTS // 2, buffer_size=4)
    attentions = [_attention(gen, case["context"] + 128) for _ in range(layers)]
    blocks = [SparseMoeWrapper(CONFIG, l, _gate(gen, directions), cache) for l in range(layers)]
    for l in range(layers):
        for e in range(EXPERTS):
            cache.add_expert((l, e), _expert(gen), eviction_group=l, offload=e < EXPERTS // 2)
    model = MixtralOffloadModel(_tokens(gen, directions, VOCAB), attentions, blocks, _norm_weight(gen), _normal(gen, VOCAB, HIDDEN, std=STD))
    _fill_caches(gen, [c for a in attentions for c in (a.k_cache, a.v_cache)], case["context"])
    return {"case": case, "model": model, "tokens": _ids(gen, case["tokens"])}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "dequantize":
        return state["layer"].dequantize(DTYPES[case["dtype"]])
    if kind == "expert":
        return state["expert"](state["x"])
    if kind == "moe":
        return state["block"](state["x"])
    if kind == "batch":
        batch = state["batch"]
        logits = batch.step(state["tokens"], case["context"])
        return {"logits": logits, "router": batch.router_logits, "keys": batch.k_caches, "values": batch.v_caches}
    model = state["model"]
    if kind == "prompt":
        logits = model.prefill(state["prompt"])
        attentions = [l.attention for l in model.layers]
    elif kind == "decode":
        model.token.copy_(state["token"])
        model.position.fill_(case["context"])
        logits = model.replay()
        attentions = [l.attention for l in model.layers]
    else:                                                          # "offload": a prompt is fed token by token
        model.position.fill_(case["context"])
        logits = []
        for i in range(case["tokens"]):
            model.token.copy_(state["tokens"][i:i + 1])
            logits.append(model.step())
        attentions = model.attentions
    return {"logits": logits, "router": model.router_logits, "keys": [a.k_cache for a in attentions],
            "values": [a.v_cache for a in attentions]}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------
def _layer_bytes(n, k, nbits):
    """Packed codes, 8-bit scale and zero, and the fp16 pairs that decode them."""
    g = n // GROUP[nbits]
    codes = {2: n // 4 * k, 3: (n + 9) // 10 * k * 4, 4: n // 2 * k}[nbits]
    return codes + 2 * g * k + 8 * (g * k // 256)


EXPERT_BYTES = 2 * _layer_bytes(FFN, HIDDEN, 2) + _layer_bytes(HIDDEN, FFN, 2)
ATTENTION_SHAPES = ((HEADS * HEAD_DIM, HIDDEN), (KV_HEADS * HEAD_DIM, HIDDEN), (KV_HEADS * HEAD_DIM, HIDDEN), (HIDDEN, HEADS * HEAD_DIM))
ATTENTION_BYTES = sum(_layer_bytes(n, k, 4) for n, k in ATTENTION_SHAPES)
ATTENTION_FLOPS = sum(2 * n * k for n, k in ATTENTION_SHAPES)
EXPERT_FLOPS = 3 * 2 * HIDDEN * FFN


def _active(tokens):
    """Experts that `tokens` tokens are expected to need."""
    return EXPERTS * (1.0 - (1.0 - 2.0 / EXPERTS) ** tokens)


def work(case):
    kind = case["kind"]
    size = {"bf16": 2, "fp16": 2, "fp32": 4}.get(case.get("dtype"), 2)
    if kind == "linear":
        n, k, rows = case["n"], case["k"], case["rows"]
        return {"bytes": _layer_bytes(n, k, case["nbits"]) + size * rows * (n + k), "flops": 2.0 * rows * n * k}
    if kind == "dequantize":
        n, k = case["n"], case["k"]
        return {"bytes": _layer_bytes(n, k, case["nbits"]) + size * n * k, "flops": 2.0 * n * k}
    if kind == "expert":
        return {"bytes": EXPERT_BYTES + 2 * size * case["rows"] * HIDDEN, "flops": 1.0 * case["rows"] * EXPERT_FLOPS}
    if kind == "moe":
        t = case["tokens"]
        return {"bytes": _active(t) * EXPERT_BYTES + 2 * EXPERTS * HIDDEN + size * t * (2 * HIDDEN + EXPERTS),
                "flops": t * (2.0 * EXPERT_FLOPS + 2 * EXPERTS * HIDDEN)}
    # decoders: `tokens` tokens, `at_once` of them sharing a pass over the weights, `seen` cached positions each attends to
    layers = case["layers"]
    tokens, at_once, seen, heads_of = {
        "decode": lambda: (1, 1, case["context"] + 1, 1),
        "batch": lambda: (case["sequences"], case["sequences"], case["context"] + 1, case["sequences"]),
        "prompt": lambda: (case["tokens"], case["tokens"], case["tokens"] / 2, 1),
        "offload": lambda: (case["tokens"], 1, case["context"] + case["tokens"] / 2, case["tokens"]),
    }[kind]()
    passes, rows_out = tokens / at_once, 1 if kind == "prompt" else tokens
    cached = 2 * 2 * KV_HEADS * HEAD_DIM * (tokens if kind == "prompt" else seen * heads_of)
    per_layer = passes * (_active(at_once) * EXPERT_BYTES + ATTENTION_BYTES + 2 * EXPERTS * HIDDEN) + cached
    flops = tokens * (2.0 * EXPERT_FLOPS + ATTENTION_FLOPS + 2 * EXPERTS * HIDDEN + 4 * HEADS * HEAD_DIM * seen)
    return {"bytes": layers * per_layer + passes * 2 * VOCAB * HIDDEN + 2 * tokens * HIDDEN + 2 * rows_out * VOCAB,
            "flops": layers * flops + rows_out * 2.0 * VOCAB * HIDDEN}


def tolerance(case):
    """A dequantized weight is a fixed sequence of fp32 operations.  Layers compute in 16-bit factors with fp32 sums; through
    a decoder's layers the bf16 residual stream adds its own roundings."""
    kind = case["kind"]
    if kind == "dequantize":
        return "exact"
    return {"rel": 1e-2 if kind in ("linear", "expert", "moe") else 2e-2}
