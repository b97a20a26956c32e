"""Operator layer: the three attention ops a TinyTorch build registers in its
dispatch tables (reference mechanism: DEFINE_OP / REGISTER_OP_IMPL,
src/Tensor/Dispatch.h:21-142), here bound to torch tensors used purely as
device-memory handles.  Every op goes through the C ABI of libtt_attn.so and
launches on the current CUDA stream of the tensors' device, as reference ops do
(src/Utils/CUDAUtils.cpp:123-135).  No op has a CPU implementation.

Argument checks, output and scratch allocation and the calls themselves are in
the extension module (csrc/binding.cpp); this layer holds the signatures.
"""
import math

import torch

from . import _capi

_DTYPES = {torch.float32: _capi.F32, torch.float16: _capi.F16, torch.bfloat16: _capi.BF16}


def _causal_mode(isCausal):
    """False/True as in the reference (top-left aligned triangle), or the string
    "bottom-right" for a chunk of new queries at the end of the key sequence."""
    if isCausal == "bottom-right":
        return _capi.CAUSAL_BOTTOM_RIGHT
    if isCausal in ("top-left", True, 1):
        return _capi.CAUSAL_TOP_LEFT
    if isCausal in (False, None, 0):
        return _capi.CAUSAL_NONE
    raise ValueError("isCausal must be a bool or 'top-left' / 'bottom-right'")


def default_scale(D):
    """1/sqrt(D) in fp32, the reference default (src/Function/FuncNNLayer.h:235)."""
    return 1.0 / math.sqrt(float(D))


def sdpAttentionFwd(q, k, v, isCausal=False, scale=None, kvLens=None, needLse=True, status=None, attnMask=None):
    """softmax(scale * Q K^T + bias) V  ->  (O [B,Hq,L,D], LSE [B,Hq,L] fp32 or None).

    attnMask of the reference (src/Function/FuncNNLayer.h:249-256): Bool -> keys that participate, otherwise added
    to the scaled scores; any shape that broadcasts against [B, Hq, L, S] by trailing-dimension alignment."""
    return _capi.native().attn_fwd(q, k, v, _causal_mode(isCausal), scale, kvLens, needLse, status, attnMask)


def sdpAttentionBwd(dO, q, k, v, o, lse, isCausal=False, scale=None, kvLens=None, needs=(True, True, True),
                    attnMask=None):
    """Gradients (dQ, dK, dV); entries of `needs` that are False come back as None."""
    return _capi.native().attn_bwd(dO, q, k, v, o, lse, _causal_mode(isCausal), scale, kvLens, needs[0], needs[1],
                                   needs[2], attnMask)


def sdpAttentionDecode(q, kCache, vCache, kvLens=None, scale=None, needLse=False, workspace=None):
    """One query per sequence against a KV cache [B,Hkv,capacity,D] -> (O [B,Hq,1,D], LSE [B,Hq] or None)."""
    return _capi.native().decode(q, kCache, vCache, kvLens, scale, needLse, workspace)


def ropeTables(positions, D, theta=10000.0, device="cuda"):
    """cos / sin tables [positions, D/2] fp32 of the usual rotary embedding: pair i at
    position p turns by p * theta^(-2i/D)."""
    inv = theta ** (-torch.arange(0, D, 2, dtype=torch.float64) / D)
    ang = torch.arange(positions, dtype=torch.float64)[:, None] * inv[None, :]
    return ang.cos().float().to(device).contiguous(), ang.sin().float().to(device).contiguous()


def sdpAttentionDecodeAppend(q, kNew, vNew, kCache, vCache, kvLens, ropeCos=None, ropeSin=None, interleaved=False,
                             scale=None, needLse=False, status=None):
    """One step of a token loop: rotate q and kNew to position kvLens[b], write kNew / vNew
    into row kvLens[b] of the caches (in place), attend over rows [0, kvLens[b]].
    Returns (O [B,Hq,1,D], LSE or None, newLens = kvLens + 1)."""
    return _capi.native().decode_append(q, kNew, vNew, kCache, vCache, kvLens, ropeCos, ropeSin, interleaved, scale,
                                        needLse, status)


def workspaceBytes(kind, dtype, B, Hq, Hkv, Lq, Skv, D):
    return int(_capi.lib().tt_attn_workspace_bytes(kind, _DTYPES[dtype], B, Hq, Hkv, Lq, Skv, D))
