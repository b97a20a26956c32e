"""GPU: the fp32 backward with values that are not finite: its CTAs walk their tiles a second time then.  Infinities and NaN in q, k, v and dO, dQ by CTAs of its
own and of stored dS, odd and even numbers of tiles, walks undivided and divided over clusters, both head dimensions.

Reference: the formulas in fp64, with the probabilities that belong to the forward's log-sum-exp (which is -inf for rows whose scores are not numbers).  Which elements are
infinite or NaN has to agree, the rest is as close as ever, and no wait runs out.  The plan of ordinary calls is asked for as well, so that
both paths are known to be taken by some."""
import ctypes as C
import math

import pytest
import torch

from gpu_util import TOL_REL_FP32

pytestmark = pytest.mark.gpu


def _params(q, k, v, o, lse, g, grads, status):
    from tinytorch_b200 import _capi
    p = _capi.BwdParams()
    (B, Hq, L, D), (Hkv, S) = q.shape, k.shape[1:3]
    p.struct_size, p.dtype, p.B, p.Hq, p.Hkv, p.Lq, p.Skv, p.D = C.sizeof(p), _capi.F32, B, Hq, Hkv, L, S, D
    for name, t in (("q", q), ("k", k), ("v", v), ("o", o), ("d_o", g), ("lse", lse), ("dq", grads[0]), ("dk", grads[1]), ("dv", grads[2])):
        setattr(p, name, t.data_ptr())
    p.scale, p.status = D ** -0.5, status.data_ptr()
    p.device, p.stream = torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
    return p


def run(q, k, v, o, lse, g, path, causal=0, lens=None, mask=None):
    """The gradients by path 0 or 1."""
    from tinytorch_b200 import _capi
    B, Hq, L, S = q.shape[0], q.shape[1], q.shape[2], k.shape[2]
    grads = [torch.full_like(t, 7.0) for t in (q, k, v)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.full((B * Hq * (L * 4 + (L + 63) // 64 * ((S + 63) // 64) * 64 * 64 * 4) + 512,), 171, dtype=torch.uint8, device="cuda")
    p = _params(q, k, v, o, lse, g, grads, status)
    p.workspace, p.workspace_bytes, p.is_causal = ws.data_ptr(), ws.numel(), causal
    if lens is not None:
        p.kv_lens = lens.data_ptr()
    if mask is not None:
        p.mask, p.mask_kind = mask.data_ptr(), _capi.MASK_BOOL if mask.dtype == torch.bool else _capi.MASK_ADD_F32
        p.mask_strides[1], p.mask_strides[2] = mask.stride(1), mask.stride(2)
    _capi.check(_capi.lib().tt_attn_bwd_selftest(C.byref(p), path, None))
    assert int(status) == 0
    return grads


def formula(q, k, v, o, lse, g):
    group = q.shape[1] // k.shape[1]
    q, k, v, o, g = (t.double() for t in (q, k, v, o, g))
    kk, vv, scale = k.repeat_interleave(group, 1), v.repeat_interleave(group, 1), q.shape[3] ** -0.5
    s, none = q @ kk.transpose(2, 3) * scale, torch.isneginf(lse)[..., None]
    lost = torch.where(torch.isnan(s) | torch.isposinf(s), torch.full_like(s, math.nan), torch.zeros_like(s))
    p = torch.where(none, lost, torch.exp(s - lse.double()[..., None]))
    ds = p * (g @ vv.transpose(2, 3) - (g * o).sum(-1, keepdim=True))
    per_head = lambda t: t.unflatten(1, (k.shape[1], group)).sum(2)
    return ds @ kk * scale, per_head(ds.transpose(2, 3) @ q) * scale, per_head(p.transpose(2, 3) @ g)


WHERE = ["q", "k", "v", "dO", "q nan", "k nan", "v nan", "dO nan", "k hidden"]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("path", [0, 1])
@pytest.mark.parametrize("where", WHERE)
@pytest.mark.parametrize("B,Hq,Hkv,L,S", [
    (1, 2, 2, 140, 150),   # three tiles either way, divided
    (2, 4, 2, 128, 250),   # four tiles
    (1, 4, 1, 30, 500),    # a group's queries share tiles
    (12, 8, 8, 60, 120),   # more CTAs than can share a walk; walks of one and two tiles
])
def test_places_of_infinities(B, Hq, Hkv, L, S, where, path, D):
    from tinytorch_b200 import op
    gen = torch.Generator("cuda").manual_seed(D + L)
    q, k, v, g = (torch.randn(s, device="cuda", generator=gen) for s in ((B, Hq, L, D), (B, Hkv, S, D), (B, Hkv, S, D), (B, Hq, L, D)))
    t = {"q": q, "k": k, "v": v, "dO": g}[where.split()[0]]
    if where == "k hidden":  # -inf for every query: no part in anything but dQ's column (0 times an infinity)
        q[..., 3] = q[..., 3].abs() + 0.5
        k[0, 0, S - 2, 3] = -math.inf
    else:
        t[0, 0, -1, 3] = math.nan if "nan" in where else math.inf
        t[-1, -1, 0, D - 1] = math.nan if "nan" in where else -math.inf
    o, lse = op.sdpAttentionFwd(q, k, v)
    for name, x, w in zip(("dq", "dk", "dv"), run(q, k, v, o, lse, g, path), formula(q, k, v, o, lse, g)):
        assert torch.equal(torch.isnan(x), torch.isnan(w)), name
        assert torch.equal(torch.isinf(x), torch.isinf(w)), name
        assert torch.equal(torch.sign(x[torch.isinf(x)]).double(), torch.sign(w[torch.isinf(w)])), name
        ok = torch.isfinite(w)
        if bool(ok.any()):
            assert float((x.double() - w)[ok].abs().max()) <= TOL_REL_FP32 * max(1.0, float(w[ok].abs().max())), name


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S", [(1, 1, 1, 1, 1), (1, 2, 2, 64, 64), (2, 4, 2, 65, 63), (1, 2, 1, 300, 1000), (1, 1, 1, 2000, 40), (40, 4, 4, 129, 130)])
def test_both_paths_at_any_size(B, Hq, Hkv, L, S, D):
    from tinytorch_b200 import op
    gen = torch.Generator("cuda").manual_seed(S)
    q, k, v, g = (torch.randn(s, device="cuda", generator=gen) for s in ((B, Hq, L, D), (B, Hkv, S, D), (B, Hkv, S, D), (B, Hq, L, D)))
    o, lse = op.sdpAttentionFwd(q, k, v)
    want = formula(q, k, v, o, lse, g)
    for path in (0, 1):
        for x, w in zip(run(q, k, v, o, lse, g, path), want):
            assert float((x.double() - w).abs().max()) <= TOL_REL_FP32 * max(1.0, float(w.abs().max()))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,causal,lens,kind", [
    (3, 4, 2, 129, 400, "bottom-right", (400, 129, 3), None),
    (4, 8, 8, 300, 300, True, None, None),
    (2, 6, 3, 321, 640, False, (640, 17), None),
    (1, 2, 1, 500, 700, True, None, None),
    (3, 6, 2, 130, 190, False, None, "add"),
    (1, 6, 2, 330, 451, False, None, "bool"),
])
def test_both_paths_with_lengths_and_masks(B, Hq, Hkv, L, S, causal, lens, kind, D):
    """Against the formulas, with what does not take part left out."""
    from tinytorch_b200 import op
    gen = torch.Generator("cuda").manual_seed(S)
    q, k, v, g = (torch.randn(s, device="cuda", generator=gen) for s in ((B, Hq, L, D), (B, Hkv, S, D), (B, Hkv, S, D), (B, Hq, L, D)))
    n = None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda")
    mask = None if kind is None else torch.randn((1, Hq, L, S), device="cuda", generator=gen)
    mask = mask < 0.3 if kind == "bool" else mask
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=n, attnMask=mask)
    j, i = torch.arange(S, device="cuda"), torch.arange(L, device="cuda")[:, None]
    end = torch.full((B, 1, 1, 1), S, device="cuda") if n is None else n.long().view(-1, 1, 1, 1)
    seen = (j < end) & ((j <= i + (end - L if causal == "bottom-right" else 0)) if causal else True)
    seen = seen & mask if kind == "bool" else seen
    group, scale = Hq // Hkv, D ** -0.5
    Q, K, V, G = q.double(), k.double().repeat_interleave(group, 1), v.double().repeat_interleave(group, 1), g.double()
    p = torch.exp(Q @ K.transpose(2, 3) * scale + (mask.double() if kind == "add" else 0.0) - lse.double().nan_to_num(neginf=0.0)[..., None])
    p = torch.where(seen, p, torch.zeros_like(p))
    ds = p * (G @ V.transpose(2, 3) - (G * o.double()).sum(-1, keepdim=True))
    per_head = lambda t: t.unflatten(1, (Hkv, group)).sum(2)
    want = ds @ K * scale, per_head(ds.transpose(2, 3) @ Q) * scale, per_head(p.transpose(2, 3) @ G)
    for path in (0, 1):
        for x, w in zip(run(q, k, v, o, lse, g, path, op._causal_mode(causal), n, mask), want):
            assert float((x.double() - w).abs().max()) <= TOL_REL_FP32 * max(1.0, float(w.abs().max()))


def test_ordinary_calls_take_both():
    from tinytorch_b200 import _capi
    taken = {}
    for D in (64, 128):
        for B, H, L in ((1, 2, 140), (4, 8, 500)):
            q = torch.randn((B, H, L, D), device="cuda")
            p = _params(q, q, q, q, q, q, [q, q, q], torch.zeros(1, dtype=torch.int32, device="cuda"))
            planned = C.c_int32(-1)
            _capi.check(_capi.lib().tt_attn_bwd_selftest(C.byref(p), -1, C.byref(planned)))
            taken[D, L] = planned.value
    assert taken == {(64, 140): 0, (64, 500): 1, (128, 140): 0, (128, 500): 1}


def test_selftest_refuses():
    from tinytorch_b200 import _capi
    q = torch.randn((1, 2, 64, 64), device="cuda")
    p = _params(q, q, q, q, q, q, [q, q, q], torch.zeros(1, dtype=torch.int32, device="cuda"))
    f = _capi.lib().tt_attn_bwd_selftest
    assert f(C.byref(p), -1, None) == -1 and f(C.byref(p), 2, None) == -3
    p.workspace, p.workspace_bytes = q.data_ptr(), 512
    assert f(C.byref(p), 1, None) == -6  # (dS does not fit)
    p.dk = p.dv = None
    assert f(C.byref(p), 1, None) == -3
    p.dtype = _capi.F16
    assert f(C.byref(p), 0, None) == -2
