"""Performance cases of the W4A16 framework: what its users have it do, through its public entry points.

A case is one of
  linear      a ``QuantizedLinear`` call: decode (one row), small and ragged batches, prompts
  dequantize  ``dequantize_cuda``: FP16 weights back from packed codes
  quantize    ``quantize_and_pack_weights`` on CUDA weights: what converting a checkpoint spends its time in
  decode      one token through ``LlamaDecodeRunner``, the whole model captured as the runner does it
Layer sizes are those of TinyLlama-1.1B and Llama-70B, which the benchmark uses, and generic ones around them.
"""
from __future__ import annotations

import math
import types

import torch

import nibble_b200
from nibble_b200.cuda import set_programmatic_launch
from nibble_b200.decode import LlamaDecodeRunner

DEVICE = "cuda"


def _linear(name, m, k, n, group=128, bias=False):
    return {"name": name, "op": "linear", "m": m, "k": k, "n": n, "group": group, "bias": bias}


def listed():
    return [
        # The call a decoding model makes most often: one token through a small attention projection.
        _linear("linear_tl_qo_m1", 1, 2048, 2048),
        # One token through the widest layer of a large model: the weights stream from memory once.
        _linear("linear_70b_gate_up_m1", 1, 8192, 28672),
        # Eight sequences decoded together, on the layer with the longest sums.
        _linear("linear_70b_down_m8", 8, 28672, 8192),
        # A batch and a layer of no round size, with a bias (as query/key/value projections of some models have).
        _linear("linear_ragged_m13_bias", 13, 4864, 5003, bias=True),
        # A serving batch of 48 sequences through a square projection.
        _linear("linear_70b_qo_m48", 48, 8192, 8192),
        # A short prompt, or a large decoding batch, through the widest layer.
        _linear("linear_70b_gate_up_m128", 128, 8192, 28672),
        # A prompt of ordinary, odd length through a narrow layer of a small model.
        _linear("linear_tl_down_m777", 777, 5632, 2048),
        # A long prompt through the widest layer.
        _linear("linear_70b_gate_up_m2048", 2048, 8192, 28672),
        # Finer scales, as many published 4-bit checkpoints have them: a few sequences decoded together.
        _linear("linear_qo_g64_m4", 4, 8192, 8192, group=64),
        # FP16 weights of a whole layer rebuilt, for a caller that goes on with a matrix product of its own.
        {"name": "dequantize_70b_gate_up", "op": "dequantize", "k": 8192, "n": 28672, "group": 128},
        # Converting a large model's layer from its FP16 checkpoint.
        {"name": "quantize_70b_gate_up", "op": "quantize", "k": 8192, "n": 28672, "group": 128, "dtype": "float16"},
        # One token of a small model late in a long answer, as a serving loop steps it.
        {"name": "decode_tl_ctx1500", "op": "decode", "layers": 22, "hidden": 2048, "inter": 5632, "heads": 32, "kv_heads": 4,
         "vocab": 32000, "max_len": 2048, "context": 1500},
    ]


_LARGEST = 8192 * 28672      # weights of the largest listed layer


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _layer_shape(rng, largest=_LARGEST):
    """Layers from 512 x 256 up to the largest; K in whole groups of 128, N as it falls."""
    while True:
        k = 128 * _log_uniform(rng, 4, 224)
        n = _log_uniform(rng, 256, 32000)
        if rng.random() < 0.6:
            n = max(256, n // 128 * 128)      # most layers of real models; the rest are ragged
        if k * n <= largest:
            return k, n


def draw(rng):
    what = rng.random()
    group = rng.choice([128, 128, 128, 128, 64, 32])
    if what < 0.66:
        k, n = _layer_shape(rng, _LARGEST if group == 128 else 8192 * 8192)
        return {"op": "linear", "m": _log_uniform(rng, 1, 2048), "k": k, "n": n, "group": group, "bias": rng.random() < 0.25}
    k, n = _layer_shape(rng)
    if what < 0.76:
        return {"op": "dequantize", "k": k, "n": n, "group": group}
    if what < 0.86:
        dtype = rng.choice(["float16", "float32"])
        return {"op": "quantize", "k": k, "n": n, "group": group, "dtype": dtype}
    head_dim = rng.choice([64, 64, 128])
    heads = rng.choice([8, 16, 32])
    hidden = heads * head_dim
    max_len = rng.choice([512, 1024, 2048])
    return {"op": "decode", "layers": rng.randint(2, 22 if hidden < 2048 else 16 if hidden == 2048 else 6), "hidden": hidden,
            "inter": 128 * rng.randint(hidden * 2 // 128, hidden * 7 // 256), "heads": heads,
            "kv_heads": heads // rng.choice([1, 4, 8]), "vocab": 128 * rng.randint(16, 250), "max_len": max_len,
            "context": _log_uniform(rng, 1, min(max_len - 1, 1500))}


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _half(gen, *shape, std=1.0, mean=0.0):
    return torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float16).mul_(std).add_(mean)


def _layer(gen, k, n, group=128, bias=False):
    packed, scales = nibble_b200.quantize_and_pack_weights(_half(gen, n, k, std=0.02), group)
    return nibble_b200.QuantizedLinear(packed, scales, group, bias=_half(gen, n, std=0.1) if bias else None)


def _llama(gen, case):
    """A LLaMA-shaped module tree with W4A16 linears of random weights: the parts that the decode runner reads."""
    hidden, inter, heads, kv_heads = case["hidden"], case["inter"], case["heads"], case["kv_heads"]
    head_dim = hidden // heads

    def norm():
        module = torch.nn.Module()
        module.weight = torch.nn.Parameter(_half(gen, hidden, std=0.1, mean=1.0), requires_grad=False)
        return module

    model, body = torch.nn.Module(), torch.nn.Module()
    model.config = types.SimpleNamespace(hidden_size=hidden, num_attention_heads=heads, num_key_value_heads=kv_heads,
                                         head_dim=head_dim, rms_norm_eps=1e-5)
    body.embed_tokens = torch.nn.Module()
    body.embed_tokens.weight = torch.nn.Parameter(_half(gen, case["vocab"], hidden), requires_grad=False)
    body.layers = torch.nn.ModuleList()
    for _ in range(case["layers"]):
        layer = torch.nn.Module()
        layer.self_attn, layer.mlp = torch.nn.Module(), torch.nn.Module()
        layer.input_layernorm, layer.post_attention_layernorm = norm(), norm()
        layer.self_attn.q_proj = _layer(gen, hidden, hidden)
        layer.self_attn.k_proj = _layer(gen, hidden, kv_heads * head_dim)
        layer.self_attn.v_proj = _layer(gen, hidden, kv_heads * head_dim)
        layer.self_attn.o_proj = _layer(gen, hidden, hidden)
        layer.mlp.gate_proj = _layer(gen, hidden, inter)
        layer.mlp.up_proj = _layer(gen, hidden, inter)
        layer.mlp.down_proj = _layer(gen, inter, hidden)
        body.layers.append(layer)
    body.norm = norm()
    body.rotary_emb = torch.nn.Module()
    body.rotary_emb.inv_freq = 1.0 / (10000.0 ** (torch.arange(0, head_dim, 2, device=DEVICE).float() / head_dim))
    model.model = body
    model.lm_head = _layer(gen, hidden, case["vocab"])
    return model


def prepare(case, seed):
    gen = _generator(seed)
    if case["op"] == "linear":
        layer = _layer(gen, case["k"], case["n"], case["group"], case["bias"])
        return {"op": "linear", "layer": layer, "x": _half(gen, 1, case["m"], case["k"])}
    if case["op"] == "dequantize":
        layer = _layer(gen, case["k"], case["n"], case["group"])
        return {"op": "dequantize", "packed": layer.packed_weights, "scales": layer.scales, "group": case["group"]}
    if case["op"] == "quantize":
        weights = _half(gen, case["n"], case["k"], std=0.02)
        return {"op": "quantize", "weights": weights.to(getattr(torch, case["dtype"])), "group": case["group"]}
    # A serving program turns programmatic launch on once its weights are in place; the runner captures its step with
    # it, at the first step.
    runner = LlamaDecodeRunner(_llama(gen, case), case["max_len"])
    past = case["context"]
    runner.k_cache[:, :, :past] = _half(gen, *runner.k_cache[:, :, :past].shape)
    runner.v_cache[:, :, :past] = _half(gen, *runner.v_cache[:, :, :past].shape)
    token = torch.randint(case["vocab"], (1,), generator=gen, device=DEVICE)
    state = {"op": "decode", "runner": runner, "token": token,
             "position": torch.full((1,), past, dtype=torch.long, device=DEVICE)}
    set_programmatic_launch(True)
    try:
        run(state)
    finally:
        set_programmatic_launch(False)
    return state


def run(state):
    if state["op"] == "linear":
        return state["layer"](state["x"])
    if state["op"] == "dequantize":
        return nibble_b200.dequantize_cuda(state["packed"], state["scales"], state["group"])
    if state["op"] == "quantize":
        return nibble_b200.quantize_and_pack_weights(state["weights"], state["group"])
    runner = state["runner"]
    runner.token.copy_(state["token"])
    runner.position.copy_(state["position"])
    runner.step()
    # The next token is the largest of these logits; it is left out here because near ties may fall either way.
    return {"logits": runner.logits, "k_cache": runner.k_cache, "v_cache": runner.v_cache, "position": runner.position}


def _packed_bytes(k, n, group):
    return n * k // 2 + n * (k // group) * 2


def work(case):
    if case["op"] == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": _packed_bytes(k, n, case["group"]) + 2 * m * (k + n) + (2 * n if case["bias"] else 0),
                "flops": 2 * m * n * k}
    if case["op"] in ("dequantize", "quantize"):
        k, n = case["k"], case["n"]
        wide = 4 if case.get("dtype") == "float32" else 2
        return {"bytes": _packed_bytes(k, n, case["group"]) + n * k * wide, "flops": n * k}
    hidden, inter, layers, vocab = case["hidden"], case["inter"], case["layers"], case["vocab"]
    kv = case["kv_heads"] * (hidden // case["heads"])
    shapes = [(hidden, hidden + 2 * kv), (hidden, hidden), (hidden, 2 * inter), (inter, hidden)]
    weights = layers * sum(k * n for k, n in shapes) + hidden * vocab
    cache = layers * 2 * kv * (case["context"] + 1)
    packed = layers * sum(_packed_bytes(k, n, 128) for k, n in shapes) + _packed_bytes(hidden, vocab, 128)
    return {"bytes": packed + 2 * cache + 2 * hidden * (2 * layers + 2) + 2 * vocab,
            "flops": 2 * weights + 2 * cache * (case["heads"] // case["kv_heads"])}


def tolerance(case):
    if case["op"] in ("dequantize", "quantize"):
        return "exact"      # codes, scales and FP16 weights are defined bit by bit
    if case["op"] == "linear":
        # One FP16 rounding of the result, and of each weight where the product is formed from FP16 weights.
        return {"rel": 2e-3, "max": 2e-2}
    # FP16 residual stream and activations, rounded some nine times in each of up to 22 layers.
    return {"rel": 1e-2, "max": 0.2}
