"""The work this framework is used for, as timed cases.

A case is one pass of one kind of work (`op`) at one size, through the package's public entry points:

  generate      flash_attention, forward only: one token of generation that recomputes its whole prefix (no key/value cache)
  decode        attention_decode: one new token per sequence against a key/value cache
  decode_layer  qkv_rope_forward + attention_decode + linear_forward: the attention layer of one generation step
  prefill       qkv_rope_forward + attention_gqa + linear_forward: the attention layer over a prompt
  train         flash_attention + attention_backward_recompute: attention in a training step, [batch, heads, seq, head_dim]
  train_gqa     rope_qk + attention_gqa + attention_gqa_backward: the same with rotary embedding, grouped K/V heads and
                [batch, seq, heads, head_dim] tensors
  train_layer   the whole attention layer of a training step, projections included, on the packed q|k|v layout

Everything is causal.  `dtype` is "fp32" (the precision the reference trains and generates in) or "bf16".
"""
import math

import torch

from irontensor_b200 import (Precision, Tensor, attention_backward_recompute, attention_decode, attention_gqa,
                             attention_gqa_backward, attention_packed, attention_packed_backward, flash_attention,
                             linear_backward, linear_forward, qkv_rope_forward, rope_qk)

ROPE_BASE = 10000.0


def _case(name, op, dtype, B, S, H, D, Hkv=None):
    """S: sequence length, or the valid cache positions of a decode step."""
    c = {"op": op, "dtype": dtype, "B": B, "S": S, "H": H, "Hkv": H if Hkv is None else Hkv, "D": D}
    return dict(c, name=name) if name else c


def listed():
    return [
        # One token of greedy generation at batch 1 without a cache: the smallest call there is, all latency.
        _case("generate_fp32", "generate", "fp32", 1, 87, 4, 64),
        # The same model generating from a cache.
        _case("decode_fp32", "decode", "fp32", 1, 100, 4, 64),
        # One generation step of the attention layer of a hidden-2048 model for a handful of users.
        _case("decode_layer_bf16", "decode_layer", "bf16", 4, 1000, 16, 128, 4),
        # A full serving batch against long caches: nothing but reading the cache counts.
        _case("decode_bf16_batch", "decode", "bf16", 32, 8190, 32, 128, 8),
        # A prompt of ragged length through the attention layer, forward only.
        _case("prefill_bf16", "prefill", "bf16", 1, 2999, 16, 128, 4),
        # Attention of a training step in fp32: the reference's own model (hidden 256, batch 16 x 256 tokens) ...
        _case("train_fp32_tiny", "train", "fp32", 16, 256, 4, 64),
        # ... and a GPT-small-width batch, one of the shapes the reference times its attention backward on.
        _case("train_fp32_wide", "train", "fp32", 8, 512, 12, 64),
        # The small model in bf16: a launch-bound training step.
        _case("train_bf16_tiny", "train", "bf16", 16, 256, 4, 64),
        # GPT-small width at its ordinary sequence length.
        _case("train_bf16_1k", "train", "bf16", 32, 1024, 12, 64),
        # Long-context training, the largest case.
        _case("train_bf16_8k", "train", "bf16", 4, 8192, 16, 128),
        # Rotary embedding, grouped K/V heads, an odd sequence length and a head_dim that is no power of two.
        _case("train_gqa_ragged", "train_gqa", "bf16", 2, 1003, 16, 96, 4),
        # The whole attention layer of a training step: 8192 tokens of a hidden-2048 model.
        _case("train_layer_bf16", "train_layer", "bf16", 4, 2048, 16, 128),
    ]


def _log(rng, lo, hi):
    """A whole number in lo..hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_one(rng):
    op = rng.choice(("generate", "decode_fp32", "decode_bf16", "decode_layer", "prefill", "train_fp32", "train_bf16",
                     "train_bf16", "train_gqa", "train_layer"))
    if op == "generate":
        return _case(None, "generate", "fp32", 1, _log(rng, 16, 512), rng.choice((4, 8, 12)), rng.choice((32, 64)))
    if op == "decode_fp32":
        return _case(None, "decode", "fp32", _log(rng, 1, 8), _log(rng, 16, 2048), rng.choice((4, 8, 12)), rng.choice((32, 64)))
    if op == "decode_bf16":
        H = rng.choice((8, 16, 32))
        return _case(None, "decode", "bf16", _log(rng, 1, 64), _log(rng, 128, 16384), H, rng.choice((64, 128)), H // rng.choice((1, 4)))
    if op == "decode_layer":
        H = rng.choice((8, 16, 32))
        return _case(None, "decode_layer", "bf16", _log(rng, 1, 32), _log(rng, 64, 8192), H, rng.choice((64, 128)), H // rng.choice((1, 4)))
    if op == "prefill":
        H = rng.choice((8, 16))
        return _case(None, "prefill", "bf16", _log(rng, 1, 4), _log(rng, 33, 8192), H, rng.choice((64, 128)), H // rng.choice((1, 4)))
    if op == "train_fp32":
        return _case(None, "train", "fp32", _log(rng, 1, 32), _log(rng, 48, 1024), rng.choice((4, 8, 12)), rng.choice((32, 64)))
    if op == "train_bf16":
        return _case(None, "train", "bf16", _log(rng, 1, 64), _log(rng, 48, 8192), rng.choice((4, 8, 12, 16)), rng.choice((64, 128)))
    if op == "train_gqa":
        H = rng.choice((8, 16))
        return _case(None, "train_gqa", "bf16", _log(rng, 1, 8), _log(rng, 100, 2500), H, rng.choice((32, 64, 80, 96, 128)),
                     H // rng.choice((1, 2, 4)))
    H = rng.choice((8, 16))
    return _case(None, "train_layer", "bf16", _log(rng, 1, 8), _log(rng, 256, 4096), H, rng.choice((64, 128)), H // rng.choice((1, 2)))


# What a drawn case of an op may need at most (floating-point operations, bytes): the listed case of its kind or a few
# times that, and never more than the largest listed case.
_MOST = {("generate", "fp32"): (1e10, 1e8), ("decode", "fp32"): (1e10, 1e9), ("decode", "bf16"): (1e12, 1.08e9),
         ("decode_layer", "bf16"): (1e12, 1.08e9), ("prefill", "bf16"): (1e12, 1e9), ("train", "fp32"): (3e10, 1e9),
         ("train", "bf16"): (3.6e12, 1.6e9), ("train_gqa", "bf16"): (1e11, 1e9), ("train_layer", "bf16"): (2e12, 1e9)}


def draw(rng):
    while True:
        c = _draw_one(rng)
        w, (flops, nbytes) = work(c), _MOST[(c["op"], c["dtype"])]
        if w["flops"] <= flops and w["bytes"] <= nbytes:
            return c


def _normal(gen, shape, dtype, scale=1.0):
    """A Tensor of N(0, scale^2) values: what projections of normalised activations, and their gradients, look like."""
    t = torch.randn(shape, generator=gen, device="cuda")
    if scale != 1.0:
        t *= scale
    p = Precision.FP32 if dtype == "fp32" else Precision.BF16
    return Tensor((t if p is Precision.FP32 else t.to(torch.bfloat16)).reshape(-1), list(shape), p)


def prepare(case, seed):
    B, S, H, Hkv, D, dt = (case[k] for k in ("B", "S", "H", "Hkv", "D", "dtype"))
    op, hidden = case["op"], case["H"] * case["D"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = dict(case)
    qk = 1.0 if S < 4096 else 0.5    # long sequences: scores of a spread that attention keeps at that length
    if op in ("generate", "train"):
        for name, scale in (("q", qk), ("k", qk), ("v", 1.0)):
            st[name] = _normal(gen, [B, H, S, D], dt, scale)
        if op == "train":
            st["d_o"] = _normal(gen, [B, H, S, D], dt)
    elif op == "train_gqa":
        st["q"], st["d_o"] = _normal(gen, [B, S, H, D], dt), _normal(gen, [B, S, H, D], dt)
        st["k"], st["v"] = _normal(gen, [B, S, Hkv, D], dt), _normal(gen, [B, S, Hkv, D], dt)
    if op in ("decode", "decode_layer"):
        max_len = (S + 255) // 256 * 256    # a cache grows in blocks; S of its positions are valid
        st["k_cache"] = _normal(gen, [B, max_len, Hkv, D], dt, qk)
        st["v_cache"] = _normal(gen, [B, max_len, Hkv, D], dt)
    if op == "decode":
        st["q"] = _normal(gen, [B, H, D], dt, qk)
    if op in ("decode_layer", "prefill", "train_layer"):
        tokens = 1 if op == "decode_layer" else S
        st["x"] = _normal(gen, [B, tokens, hidden], dt)
        st["w_qkv"] = _normal(gen, [(H + 2 * Hkv) * D, hidden], dt, hidden ** -0.5)
        st["w_o"] = _normal(gen, [hidden, hidden], dt, hidden ** -0.5)
        if op == "train_layer":
            st["d_out"] = _normal(gen, [B * S, hidden], dt)
    return st


def run(st):
    B, S, H, Hkv, D, op = (st[k] for k in ("B", "S", "H", "Hkv", "D", "op"))
    if op == "generate":
        o = flash_attention(st["q"], st["k"], st["v"], True)
        return o.torch()
    if op == "decode":
        return attention_decode(st["q"], st["k_cache"], st["v_cache"], S).torch()
    if op == "decode_layer":
        # The new token's key and value go back to the caller, who appends them; the cache in hand holds S positions.
        q, k, v = qkv_rope_forward(st["x"], st["w_qkv"], H, Hkv, D, ROPE_BASE, S - 1)
        o = attention_decode(q.view([B, H, D]), st["k_cache"], st["v_cache"], S)
        return linear_forward(o.view([B, H * D]), st["w_o"]).torch(), k.torch(), v.torch()
    if op == "prefill":
        q, k, v = qkv_rope_forward(st["x"], st["w_qkv"], H, Hkv, D, ROPE_BASE)
        o = attention_gqa(q, k, v, True)
        return linear_forward(o.view([B * S, H * D]), st["w_o"]).torch(), k.torch(), v.torch()
    if op == "train":
        o = flash_attention(st["q"], st["k"], st["v"], True)
        grads = attention_backward_recompute(st["d_o"], st["q"], st["k"], st["v"], o, o.lse)
        return (o.torch(), o.lse.torch()) + tuple(g.torch() for g in grads)
    if op == "train_gqa":
        q, k = rope_qk(st["q"], st["k"], ROPE_BASE)
        o = attention_gqa(q, k, st["v"], True)
        grads = attention_gqa_backward(st["d_o"], q, k, st["v"], o, True, rope_base=ROPE_BASE)
        return (o.torch(), o.lse.torch()) + tuple(g.torch() for g in grads)
    n, hidden, width = B * S, H * D, (H + 2 * Hkv) * D
    qkv = qkv_rope_forward(st["x"], st["w_qkv"], H, Hkv, D, ROPE_BASE, packed=True)
    attn = attention_packed(qkv, H, Hkv, D, True)
    out = linear_forward(attn.view([n, hidden]), st["w_o"])
    d_attn, d_wo = linear_backward(st["d_out"], attn.view([n, hidden]), st["w_o"])
    d_qkv = attention_packed_backward(d_attn.view([B, S, H, D]), qkv, attn, H, Hkv, D, True, rope_base=ROPE_BASE)
    d_x, d_wqkv = linear_backward(d_qkv.view([n, width]), st["x"].view([n, hidden]), st["w_qkv"])
    return out.torch(), d_x.torch(), d_wo.torch(), d_wqkv.torch()


def work(case):
    """Operations: causal attention 2 B H S^2 D forward and 5 B H S^2 D backward, a projection 2 n in out (three of those with
    its backward).  Bytes: inputs once, outputs once."""
    B, S, H, Hkv, D, op = (case[k] for k in ("B", "S", "H", "Hkv", "D", "op"))
    e = 4 if case["dtype"] == "fp32" else 2
    hidden, width, square = H * D, (H + 2 * Hkv) * D, B * H * S * S * D
    qo, kv, lse = B * H * S * D * e, B * Hkv * S * D * e, 4 * B * H * S
    if op == "generate":
        return {"bytes": 2 * qo + 2 * kv + lse, "flops": 2 * square}
    if op == "decode":
        return {"bytes": 2 * kv + 2 * B * H * D * e + 4 * B * H, "flops": 4 * B * H * S * D}
    if op == "decode_layer":
        return {"bytes": 2 * kv + (width + hidden) * hidden * e + 2 * B * (hidden + Hkv * D) * e,
                "flops": 4 * B * H * S * D + 2 * B * hidden * (width + hidden)}
    if op == "prefill":
        n = B * S
        return {"bytes": (width + hidden) * hidden * e + 2 * n * (hidden + Hkv * D) * e,
                "flops": 2 * square + 2 * n * hidden * (width + hidden)}
    if op in ("train", "train_gqa"):
        return {"bytes": 4 * qo + 4 * kv + lse, "flops": 7 * square}
    n, weights = B * S, (width + hidden) * hidden
    return {"bytes": weights * (e + 4) + 4 * n * hidden * e, "flops": 7 * square + 6 * n * hidden * (width + hidden)}


def tolerance(case):
    """bf16 results carry 8 bits, and bf16 probabilities and score gradients inside; fp32 results are sums of fp32 products."""
    return {"rel": 1e-5, "max": 4e-4} if case["dtype"] == "fp32" else {"rel": 1e-2, "max": 0.25}
