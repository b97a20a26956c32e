"""Performance cases: the work that programs built on this package have it do, through its public entry points.

Five kinds of work ("op" of a case):
  prefill   function.sdpAttention without gradients: whole prompts, chunks of new queries against a cache, encoders
  train     function.sdpAttention and its gradients
  decode    op.sdpAttentionDecode / op.sdpAttentionDecodeAppend: one new token per sequence against a KV cache
  linear    fused.linear, alone or with its gradients
  layer     one decoder layer: the operators above plus fused.fusedAddRmsNorm and fused.siluMul, in a program's order
"""
import math

import torch

from tinytorch_b200 import function, fused, op

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # the package's headline: a batch of long prompts of a model without grouped heads
        dict(name="prefill_long_bf16", op="prefill", dtype="bf16", B=4, Hq=32, Hkv=32, L=4096, S=4096, D=128,
             causal="top-left", lens=False, std=1.0),
        # a batch of medium prompts of a grouped-query model
        dict(name="prefill_gqa_f16", op="prefill", dtype="f16", B=8, Hq=32, Hkv=8, L=2048, S=2048, D=128,
             causal="top-left", lens=False, std=0.5),
        # one user's prompt, of no particular length: what sets the time to the first token of a chat
        dict(name="prefill_prompt_bf16", op="prefill", dtype="bf16", B=1, Hq=32, Hkv=8, L=777, S=777, D=128,
             causal="top-left", lens=False, std=1.0),
        # chunked prefill: the next 256 tokens of two long requests against their caches, at their own lengths
        dict(name="prefill_chunk_bf16", op="prefill", dtype="bf16", B=2, Hq=32, Hkv=8, L=256, S=8192, D=128,
             causal="bottom-right", lens=True, std=1.0),
        # attention of a training step, head dimension 64
        dict(name="train_f16_d64", op="train", dtype="f16", B=8, Hq=16, Hkv=16, L=2048, D=64, causal=True, mask="none"),
        # ... of a grouped-query model with head dimension 128, one packed sequence per step
        dict(name="train_gqa_bf16_d128", op="train", dtype="bf16", B=1, Hq=32, Hkv=8, L=3000, D=128, causal=True,
             mask="none"),
        # the smallest training step (the size of the known-answer tests): a call's fixed cost
        dict(name="train_tiny_f32", op="train", dtype="f32", B=2, Hq=4, Hkv=4, L=128, D=64, causal=True, mask="none"),
        # single-precision training with an additive position bias
        dict(name="train_bias_f32", op="train", dtype="f32", B=4, Hq=8, Hkv=8, L=500, D=64, causal=False, mask="bias"),
        # decoding a large batch without grouped heads: the whole cache is read for every token
        dict(name="decode_large_bf16", op="decode", dtype="bf16", B=64, Hq=32, Hkv=32, cap=8192, D=128, append=False),
        # one layer of a token step for a few users: rotary embedding, cache append, projections, norms, gated MLP
        dict(name="layer_decode_bf16", op="layer", dtype="bf16", B=8, L=1, hidden=4096, Hq=32, Hkv=8, D=128, ffn=14336,
             cap=4096),
        # the same layer over two prompts
        dict(name="layer_prefill_bf16", op="layer", dtype="bf16", B=2, L=1000, hidden=4096, Hq=32, Hkv=8, D=128,
             ffn=14336, cap=0),
        # a projection of a training step, forward and gradients
        dict(name="linear_train_bf16", op="linear", dtype="bf16", M=4096, K=4096, N=12288, bias=True, grad=True),
    ]


# ------------------------------------------------------------------------------------------------ drawn cases --
def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _heads(rng):
    group = rng.choice([1, 1, 2, 4, 8])
    return rng.choice([2, 3, 4, 8, 16]) * group if group < 4 else rng.choice([1, 2, 4, 8]) * group, group


def _draw_prefill(rng):
    hq, group = _heads(rng)
    c = dict(op="prefill", dtype=rng.choice(["bf16", "bf16", "f16", "f32"]), B=_log(rng, 1, 16), Hq=hq, Hkv=hq // group,
             D=rng.choice([64, 128]), causal=rng.choice(["top-left", "top-left", "bottom-right", "none"]),
             std=rng.choice([0.5, 1.0]))
    if c["causal"] == "bottom-right":  # a chunk of new queries behind a cache
        c["L"] = _log(rng, 16, 1024)
        c["S"] = c["L"] + _log(rng, 128, 15000)
        c["lens"] = True
    else:
        c["L"] = c["S"] = _log(rng, 16, 8192)
        c["lens"] = c["causal"] == "none" and rng.random() < 0.5  # padded batches of an encoder
    return c


def _draw_train(rng):
    hq, group = _heads(rng)
    mask = rng.choice(["none", "none", "none", "padding", "bias"])
    return dict(op="train", dtype=rng.choice(["bf16", "f16", "f32"]), B=_log(rng, 1, 16), Hq=hq, Hkv=hq // group,
                L=_log(rng, 32, 8192), D=rng.choice([64, 128]), causal=mask == "none" and rng.random() < 0.75, mask=mask)


def _draw_decode(rng):
    hq, group = _heads(rng)
    return dict(op="decode", dtype=rng.choice(["bf16", "bf16", "f16", "f32"]), B=_log(rng, 1, 128), Hq=hq, Hkv=hq // group,
                cap=_log(rng, 128, 16384), D=rng.choice([64, 128]), append=rng.random() < 0.5)


def _draw_linear(rng):
    grad = rng.random() < 0.5
    return dict(op="linear", dtype=rng.choice(["bf16", "f16"]), M=_log(rng, 32 if grad else 1, 16384),
                K=8 * _log(rng, 32, 1792), N=8 * _log(rng, 32, 3584), bias=rng.random() < 0.5, grad=grad)


def _draw_layer(rng):
    D, group, hkv = rng.choice([64, 128]), rng.choice([1, 2, 4, 8]), rng.choice([2, 4, 8])
    hq = min(32, hkv * group)
    decode = rng.random() < 0.5
    hidden = hq * D
    return dict(op="layer", dtype=rng.choice(["bf16", "f16"]), B=_log(rng, 1, 128) if decode else _log(rng, 1, 4),
                L=1 if decode else _log(rng, 16, 2048), hidden=hidden, Hq=hq, Hkv=hkv, D=D,
                ffn=8 * int(hidden * rng.uniform(2.5, 4.0) / 8), cap=_log(rng, 128, 8192) if decode else 0)


def draw(rng):
    kind = rng.choice([_draw_prefill, _draw_train, _draw_decode, _draw_linear, _draw_layer])
    while True:
        c = kind(rng)
        w = work(c)
        # no more than the largest listed case; single precision within what CUDA cores do in about the same time
        if w["flops"] > (2e10 if c["dtype"] == "f32" else 8e11) or w["bytes"] > 4.5e9:
            continue
        if c.get("append") and 2 * c["B"] * c["Hkv"] * c["cap"] * c["D"] > 6e8:  # (the caches come back as results)
            continue
        if c["op"] == "layer" and 2 * c["B"] * c["Hkv"] * c["cap"] * c["D"] > 6e8:
            continue
        return c


# -------------------------------------------------------------------------------------------- inputs and plan --
def prepare(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]

    def normal(*shape, std=1.0, dtype=dt):
        t = torch.randn(shape, dtype=dtype, device="cuda", generator=g)
        return t if std == 1.0 else t.mul_(std)

    def lengths(lo, hi, n):  # valid rows per sequence, lo..hi
        return torch.randint(lo, hi + 1, (n,), dtype=torch.int32, device="cuda", generator=g)

    s = dict(case)
    kind = case["op"]
    if kind == "prefill":
        B, Hq, Hkv, L, S, D, std = (case[k] for k in ("B", "Hq", "Hkv", "L", "S", "D", "std"))
        s["q"], s["k"], s["v"] = normal(B, Hq, L, D, std=std), normal(B, Hkv, S, D, std=std), normal(B, Hkv, S, D, std=std)
        s["kv_lens"] = lengths(max(L if case["causal"] == "bottom-right" else 1, S // 2), S, B) if case["lens"] else None
        s["mode"] = False if case["causal"] == "none" else (True if case["causal"] == "top-left" else "bottom-right")
    elif kind == "train":
        B, Hq, Hkv, L, D = (case[k] for k in ("B", "Hq", "Hkv", "L", "D"))
        s["q"], s["k"], s["v"], s["grad"] = normal(B, Hq, L, D), normal(B, Hkv, L, D), normal(B, Hkv, L, D), normal(B, Hq, L, D)
        for n in "qkv":
            s[n].requires_grad_()
        s["attn_mask"] = None
        if case["mask"] == "padding":  # Bool [B,1,1,S]: true = the key takes part
            s["attn_mask"] = torch.arange(L, device="cuda")[None, None, None, :] < lengths(max(1, L // 2), L, B)[:, None, None, None]
        elif case["mask"] == "bias":  # additive, one per head
            s["attn_mask"] = normal(1, Hq, L, L)
    elif kind == "decode":
        B, Hq, Hkv, cap, D = (case[k] for k in ("B", "Hq", "Hkv", "cap", "D"))
        s["q"], s["k_cache"], s["v_cache"] = normal(B, Hq, 1, D), normal(B, Hkv, cap, D), normal(B, Hkv, cap, D)
        s["kv_lens"] = lengths(max(1, cap // 8), cap - 1, B)
        if case["append"]:
            s["k_new"], s["v_new"] = normal(B, Hkv, 1, D), normal(B, Hkv, 1, D)
            s["cos"], s["sin"] = op.ropeTables(cap, D)
    elif kind == "linear":
        M, K, N = case["M"], case["K"], case["N"]
        s["x"], s["w"] = normal(M, K), normal(N, K, std=K ** -0.5)
        s["b"] = normal(N) if case["bias"] else None
        if case["grad"]:
            s["grad_y"] = normal(M, N)
            s["leaves"] = [t for t in (s["x"], s["w"], s["b"]) if t is not None]
            for t in s["leaves"]:
                t.requires_grad_()
    else:
        B, L, hidden, Hq, Hkv, D, ffn, cap = (case[k] for k in ("B", "L", "hidden", "Hq", "Hkv", "D", "ffn", "cap"))
        s["x"], s["residual"] = normal(B, L, hidden), normal(B, L, hidden)
        s["norm1"], s["norm2"] = normal(hidden, std=0.1).add_(1), normal(hidden, std=0.1).add_(1)
        s["w_qkv"] = normal((Hq + 2 * Hkv) * D, hidden, std=hidden ** -0.5)
        s["w_o"] = normal(hidden, Hq * D, std=(Hq * D) ** -0.5)
        s["w_gate_up"], s["w_down"] = normal(2 * ffn, hidden, std=hidden ** -0.5), normal(hidden, ffn, std=ffn ** -0.5)
        if cap:
            s["k_cache"], s["v_cache"] = normal(B, Hkv, cap, D), normal(B, Hkv, cap, D)
            s["kv_lens"] = lengths(max(1, cap // 4), cap - cap // 4, B)
            s["cos"], s["sin"] = op.ropeTables(cap, D)
    return s


# ------------------------------------------------------------------------------------------------------ a pass --
def _run_layer(s):
    """The residual stream and the previous layer's output are updated in place, as in a stack of layers."""
    B, L, Hq, Hkv, D = s["B"], s["L"], s["Hq"], s["Hkv"], s["D"]
    x, r = s["x"], s["residual"]
    fused.fusedAddRmsNorm(x, r, s["norm1"], 1e-5)
    qkv = fused.linear(x, s["w_qkv"])
    # [B, L, heads, D] -> [B, heads, L, D], as views
    q, k, v = (t.view(B, L, -1, D).transpose(1, 2) for t in qkv.split([Hq * D, Hkv * D, Hkv * D], dim=2))
    new_lens = None
    if s["cap"]:
        o, _, new_lens = op.sdpAttentionDecodeAppend(q, k, v, s["k_cache"], s["v_cache"], s["kv_lens"], s["cos"], s["sin"])
    else:
        o = function.sdpAttention(q, k, v, isCausal=True)
    y = fused.linear(o.transpose(1, 2).reshape(B, L, Hq * D), s["w_o"])
    fused.fusedAddRmsNorm(y, r, s["norm2"], 1e-5)
    out = fused.linear(fused.siluMul(fused.linear(y, s["w_gate_up"])), s["w_down"])
    if s["cap"]:
        return out, r, new_lens, s["k_cache"], s["v_cache"]
    return out, r


def run(state):
    s = state
    kind = s["op"]
    if kind == "prefill":
        return function.sdpAttention(s["q"], s["k"], s["v"], isCausal=s["mode"], kvLens=s["kv_lens"])
    if kind == "train":
        o = function.sdpAttention(s["q"], s["k"], s["v"], isCausal=s["causal"], attnMask=s["attn_mask"])
        return (o,) + torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["grad"])
    if kind == "decode":
        if not s["append"]:
            return op.sdpAttentionDecode(s["q"], s["k_cache"], s["v_cache"], s["kv_lens"])[0]
        o, _, new_lens = op.sdpAttentionDecodeAppend(s["q"], s["k_new"], s["v_new"], s["k_cache"], s["v_cache"], s["kv_lens"],
                                                     s["cos"], s["sin"])
        return o, new_lens, s["k_cache"], s["v_cache"]
    if kind == "linear":
        y = fused.linear(s["x"], s["w"], s["b"])
        return (y,) + torch.autograd.grad(y, s["leaves"], s["grad_y"]) if s["grad"] else y
    return _run_layer(s)


# ------------------------------------------------------------------------------ work and tolerance of one pass --
def _mean_len(lo, hi):
    return 0.5 * (lo + hi)


def work(case):
    es = SIZE[case["dtype"]]
    kind = case["op"]
    if kind == "linear":
        M, K, N = case["M"], case["K"], case["N"]
        vec = N if case["bias"] else 0
        if case["grad"]:  # x, w, b, dy in; y, dx, dw, db out
            return {"bytes": es * 2.0 * (M * K + N * K + M * N + vec), "flops": 6.0 * M * N * K}
        return {"bytes": es * float(M * K + N * K + M * N + vec), "flops": 2.0 * M * N * K}
    B, Hq, Hkv, D = (case[k] for k in ("B", "Hq", "Hkv", "D"))
    if kind == "prefill":
        L, S = case["L"], case["S"]
        keys = _mean_len(max(L if case["causal"] == "bottom-right" else 1, S // 2), S) if case["lens"] else S
        pairs = {"none": L * keys, "top-left": L * (L + 1) / 2.0, "bottom-right": L * keys - L * (L - 1) / 2.0}[case["causal"]]
        return {"bytes": es * B * D * (2.0 * Hq * L + 2.0 * Hkv * keys), "flops": 4.0 * B * Hq * D * pairs}
    if kind == "train":
        L = case["L"]
        keys = _mean_len(max(1, L // 2), L) if case["mask"] == "padding" else L
        pairs = L * (L + 1) / 2.0 if case["causal"] else L * keys
        mask = {"none": 0, "padding": B * L, "bias": es * Hq * L * L}[case["mask"]]
        # q, k, v, dO in; o, dq, dk, dv out; two products forward, five backward
        return {"bytes": es * B * L * D * (4.0 * Hq + 4.0 * Hkv) + mask, "flops": 14.0 * B * Hq * D * pairs}
    if kind == "decode":
        cap = case["cap"]
        keys = _mean_len(max(1, cap // 8), cap - 1)
        new = 4.0 * Hkv if case["append"] else 0.0
        return {"bytes": es * B * D * (2.0 * Hkv * keys + 2.0 * Hq + new), "flops": 4.0 * B * Hq * D * keys}
    L, hidden, ffn, cap = case["L"], case["hidden"], case["ffn"], case["cap"]
    weights = hidden * ((Hq + 2 * Hkv) * D + Hq * D + 3 * ffn)
    M = B * L
    keys = _mean_len(max(1, cap // 4), cap - cap // 4) if cap else 0.0
    pairs = keys if cap else L * (L + 1) / 2.0
    # weights, valid cache rows, the layer's input and residual in; its output and residual out
    return {"bytes": es * (weights + 2.0 * B * Hkv * keys * D + 4.0 * M * hidden),
            "flops": 2.0 * M * weights + 4.0 * B * Hq * D * pairs}


def tolerance(case):
    # single precision: sums of products in another order; 16-bit types: one rounding of the results and of the
    # intermediate values that the tensor cores take in 16 bits
    return {"rel": {"f32": 1e-5, "f16": 3e-3, "bf16": 1e-2}[case["dtype"]]}
