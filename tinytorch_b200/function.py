"""Function layer: ``sdpAttention`` with the reference's signature and a working
backward.

Mirrors function::sdpAttention / FuncSDPAttention
(src/Function/FuncNNLayer.h:229-268, 298-302): same argument order and meaning
(query, key, value, isCausal, attnMask, dropoutP, scale), same default scale
1/sqrt(D), same top-left causal alignment, same assertion that isCausal and a
mask are mutually exclusive, same mask semantics (Bool: true = the key takes
part; otherwise added to the scaled scores; broadcast against [B, H, L, S],
src/Function/FuncNNLayer.h:249-256).  Differences, all forced by the fused path:
  * forward saves (O, LSE) for backward, as the reference's implemented
    backwards save what they need (AutogradContext::pushData,
    src/Tensor/Function.h:24-31);
  * backward exists (the reference traps, FuncNNLayer.h:267) and hands dQ, dK, dV
    to autograd, which accumulates them like AutogradMeta::addGrad
    (src/Tensor/AutogradMeta.cpp:29-43);
  * ``kvLens`` (int32 [B]) is the cheap form of the reference's per-batch length
    mask and may be combined with isCausal; isCausal may also be the string
    "bottom-right" (a chunk of new queries at the end of the keys);
  * a query row with no participating key gives O = 0 (the reference gives NaN);
  * the mask receives no gradient; dropoutP must be 0 (dropout stays on the
    reference's generic-op composition, which this package does not contain).
"""
from . import _capi
from .op import _causal_mode


class FuncSDPAttention:
    """The differentiable operator; its node (forward saves q, k, v, O and LSE, backward computes dQ, dK, dV) is
    AttentionBackward in csrc/binding.cpp."""

    @staticmethod
    def apply(query, key, value, isCausal, kvLens, scale, attnMask=None):
        return _capi.native().sdp_attention(query, key, value, _causal_mode(isCausal), kvLens, scale, attnMask)


def sdpAttention(query, key, value, isCausal=False, attnMask=None, dropoutP=0.0, scale=None, kvLens=None):
    """Drop-in for function::sdpAttention (src/Function/FuncNNLayer.h:298-302)."""
    if isCausal and attnMask is not None:
        raise AssertionError("isCausal and attnMask are mutually exclusive (FuncNNLayer.h:242)")
    if dropoutP > 0.0:
        raise NotImplementedError("dropoutP > 0 is not on the fused path")
    if not isinstance(isCausal, str):
        isCausal = bool(isCausal)
    return _capi.native().sdp_attention(query, key, value, _causal_mode(isCausal), kvLens, scale, attnMask)
