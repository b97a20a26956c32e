"""GPU: gradients of fp32 attention where an additive mask has one large finite value for all keys of a row, as padded queries have.  The scores
are rounded at the mask's size, so probabilities are those of the rounded sums: equal ones from some 1e9 on.

Reference: the composition in fp64 with the scores alone.  Bound: a sum's exponent is off by half the spacing of floats of the mask's size (in units of log2), and so
is that of the row's sum; a probability by the factor 2^spacing, from 1e9 on (where scores are below half the spacing) by none.  That factor, taken through the
formulas of the gradients, and 1e-5 of the largest element, the bound of the fp32 tests."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from gpu_util import TOL_REL_FP32

pytestmark = pytest.mark.gpu


def _case(B, H, L, S, D, value, zero):
    gen = torch.Generator("cuda").manual_seed(11)
    q, k, v, g = (torch.randn((B, H, n, D), device="cuda", generator=gen) for n in (L, S, S, L))
    mask = torch.randn((1, 1, L, S), device="cuda", generator=gen)
    large = torch.arange(L, device="cuda") % 5 == 2
    mask[:, :, large] = value
    if zero:  # what padded queries' gradients usually are
        g[:, :, large] = 0.0
    return q, k, v, g, mask, large


def _check(grads, q, k, v, g, mask, large, value, n=None):
    scale = q.shape[3] ** -0.5
    spacing = float(np.spacing(np.float32(abs(value) * math.log2(math.e))))
    rel = 2.0 ** spacing - 1 if abs(value) < 1e9 else 0.0
    q, k, v, g = (t.double() for t in (q, k, v, g))
    s = q @ k.transpose(2, 3) * scale
    s = torch.where(large[:, None], s if abs(value) < 1e9 else torch.zeros_like(s), s + mask.double())
    if n is not None:
        s = s.masked_fill(torch.arange(s.shape[3], device="cuda") >= n.long().view(-1, 1, 1, 1), -math.inf)
    p = s.softmax(-1)
    o = p @ v
    ds = p * (g @ v.transpose(2, 3) - (g * o).sum(-1, keepdim=True))
    off = rel * large[:, None] * p
    off_s = off * ((g @ v.transpose(2, 3) - (g * o).sum(-1, keepdim=True)).abs() + (g.abs() * (p @ v.abs())).sum(-1, keepdim=True))
    want = (ds @ k * scale, ds.transpose(2, 3) @ q * scale, p.transpose(2, 3) @ g)
    slack = (off_s @ k.abs() * scale, off_s.transpose(2, 3) @ q.abs() * scale, off.transpose(2, 3) @ g.abs())
    for t, w, e in zip(grads, want, slack):
        assert bool(((t.double() - w).abs() <= e + TOL_REL_FP32 * max(1.0, float(w.abs().max()))).all()), float((t.double() - w).abs().max())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("zero", [False, True])
@pytest.mark.parametrize("value", [-1.0e4, -1.0e6, -1.0e9, -1.0e38, 1.0e9])
@pytest.mark.parametrize("B,H,L,S", [(1, 2, 70, 90), (4, 8, 300, 310)])  # dQ by the query CTAs; of stored dS
def test_gradients_of_rows_with_one_large_mask(B, H, L, S, value, zero, D):
    from tinytorch_b200 import op
    q, k, v, g, mask, large = _case(B, H, L, S, D, value, zero)
    o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask)
    _check(op.sdpAttentionBwd(g, q, k, v, o, lse, attnMask=mask), q, k, v, g, mask, large, value)


@pytest.mark.parametrize("D", [64, 128])
def test_lengths_and_one_large_mask(D):
    from tinytorch_b200 import op
    q, k, v, g, mask, large = _case(3, 2, 70, 90, D, -1.0e9, False)
    n = torch.tensor([90, 1, 65], dtype=torch.int32, device="cuda")
    o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask, kvLens=n)
    _check(op.sdpAttentionBwd(g, q, k, v, o, lse, attnMask=mask, kvLens=n), q, k, v, g, mask, large, -1.0e9, n)


@pytest.mark.parametrize("D", [64, 128])
def test_a_workspace_without_room_for_the_rows(D):
    """The rows count for nothing then: gradients that are finite, and right where the rows' own are zero."""
    from tinytorch_b200 import _capi, op
    B, H, L, S = 1, 2, 70, 90
    for zero in (True, False):
        q, k, v, g, mask, large = _case(B, H, L, S, D, -1.0e9, zero)
        o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask)
        grads = [torch.full_like(t, math.nan) for t in (q, k, v)]
        ws = torch.empty((B * H * L * 4 + 255) // 256 * 256, dtype=torch.uint8, device="cuda")
        p = _capi.BwdParams()
        p.struct_size, p.dtype, p.B, p.Hq, p.Hkv, p.Lq, p.Skv, p.D = C.sizeof(p), _capi.F32, B, H, H, L, S, D
        for name, t in (("q", q), ("k", k), ("v", v), ("o", o), ("d_o", g), ("lse", lse), ("dq", grads[0]), ("dk", grads[1]), ("dv", grads[2])):
            setattr(p, name, t.data_ptr())
        p.mask, p.mask_kind, p.mask_strides[2] = mask.data_ptr(), _capi.MASK_ADD_F32, S
        p.scale, p.device, p.stream = D ** -0.5, torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
        p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
        _capi.check(_capi.lib().tt_attn_bwd(C.byref(p)))
        assert all(bool(torch.isfinite(t).all()) for t in grads)
        if zero:
            _check(grads, q, k, v, g, mask, large, -1.0e9)


@pytest.mark.parametrize("D", [64, 128])
def test_grouped_heads_and_one_large_mask(D):
    """Query heads that share a kv head, each with a mask of its own."""
    from tinytorch_b200 import op
    B, H, group, L, S, value = 2, 2, 3, 70, 90, -1.0e9
    q, _, _, g, _, large = _case(B, H * group, L, S, D, value, False)
    _, k, v, _, _, _ = _case(B, H, L, S, D, value, False)
    mask = torch.randn((1, H * group, L, S), device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    mask[:, :, large] = value
    o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask)
    dq, dk, dv = op.sdpAttentionBwd(g, q, k, v, o, lse, attnMask=mask)
    _check((dq,), q, *(t.repeat_interleave(group, 1) for t in (k, v)), g, mask, large, value)
    # the kv heads' gradients: the sums of what each query head gives with a copy of its own
    kk, vv = (t.repeat_interleave(group, 1).contiguous() for t in (k, v))
    each = op.sdpAttentionBwd(g, q, kk, vv, o, lse, attnMask=mask)
    for t, w in zip((dk, dv), each[1:]):
        w = w.double().unflatten(1, (H, group)).sum(2)
        assert float((t.double() - w).abs().max()) <= TOL_REL_FP32 * max(1.0, float(w.abs().max()))
