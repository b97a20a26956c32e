"""GPU: the fp32 backward whose dQ pass reads the dS tiles that the dK / dV pass leaves: ragged tiles, several query heads per kv head,
both causal alignments, sequences of no or few keys, masks, undivided and divided walks; and the same call without room for dS, in a
caller's buffer or from an allocator.

Reference: the composition in fp64.  Bound: that of the fp32 tests, 1e-5 of the largest element, and of 1.  For dK the roundings of dP = dO V
and delta = dO O come on top.  Where all rows see one and the same key the two are equal, dS is what their roundings leave, and dK, which
is 0, the sum of that over all rows; with n keys every term carries a probability of about 1 / n.  A sum of D products rounds to within
2^-24 times its partial sums, which for terms of mixed signs grow like sqrt(k) |dO o V| / sqrt(D): the error has a standard deviation below
2^-24 sqrt(D) |dO o V| (Euclidean norm of the products), so that of dP - delta is below sqrt(2) of it, and dK's, rows independent of one another,
2^-24 sqrt(2 D sum over the rows of (P scale Q |dO o V|)^2).  Eight of them are allowed; the formula itself, in fp32, leaves up to 0.083 of that (one key, 642 rows)."""
import ctypes as C

import pytest
import torch

from gpu_util import TOL_REL_FP32

pytestmark = pytest.mark.gpu


def _scores(q, k, seen, bias):
    group = q.shape[1] // k.shape[1]
    s = q @ k.repeat_interleave(group, 1).transpose(2, 3) * q.shape[3] ** -0.5
    if bias is not None:
        s = s + bias.double()
    return torch.nan_to_num(s.masked_fill(~seen, float("-inf")).softmax(-1))


def _reference(q, k, v, g, seen, bias):
    q, k, v = (t.double().requires_grad_() for t in (q, k, v))
    o = _scores(q, k, seen, bias) @ v.repeat_interleave(q.shape[1] // k.shape[1], 1)
    return torch.autograd.grad(o, (q, k, v), g.double())


def _noise(q, k, v, g, seen, bias):  # of dK, see above
    q, k, v, g = (t.double() for t in (q, k, v, g))
    B, H, L, D = q.shape
    products = (g * g) @ (v * v).repeat_interleave(H // k.shape[1], 1).transpose(2, 3)  # |dO o V|^2
    per_head = (_scores(q, k, seen, bias) ** 2 * products).transpose(2, 3) @ (q * q) / D  # (scale^2 = 1 / D)
    return 8 * 2.0 ** -24 * (2 * D * per_head.view(B, k.shape[1], -1, *k.shape[2:]).sum(2)).sqrt()


def _seen(B, L, S, causal, lens):
    j, i = torch.arange(S, device="cuda"), torch.arange(L, device="cuda")[:, None]
    n = torch.full((B, 1, 1), S, device="cuda") if lens is None else lens.long()[:, None, None]
    seen = (j < n).expand(B, L, S)
    if causal:
        seen = seen & (j <= i + (n - L if causal == "bottom-right" else 0))
    return seen[:, None]


def _params(q, k, v, o, lse, g, grads, causal, n):
    from tinytorch_b200 import _capi, op
    p = _capi.BwdParams()
    (B, Hq, L, D), (Hkv, S) = q.shape, k.shape[1:3]
    p.struct_size, p.dtype, p.B, p.Hq, p.Hkv, p.Lq, p.Skv, p.D = C.sizeof(p), _capi.F32, B, Hq, Hkv, L, S, D
    for name, t in (("q", q), ("k", k), ("v", v), ("o", o), ("d_o", g), ("lse", lse), ("dq", grads[0]), ("dk", grads[1]), ("dv", grads[2])):
        setattr(p, name, t.data_ptr())
    if n is not None:
        p.kv_lens = n.data_ptr()
    p.is_causal, p.scale = op._causal_mode(causal), D ** -0.5
    p.device, p.stream = torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
    return p


def _make(D, B, Hq, Hkv, L, S):
    gen = torch.Generator("cuda").manual_seed(D + L)
    return (gen,) + tuple(torch.randn(s, device="cuda", generator=gen) for s in ((B, Hq, L, D), (B, Hkv, S, D), (B, Hkv, S, D), (B, Hq, L, D)))


def _stored(D, B, Hq, Hkv, L, S):  # whether dS is stored at this size
    from tinytorch_b200 import _capi, op
    rows = B * Hq * L * 4
    return op.workspaceBytes(_capi.KIND_BWD, torch.float32, B, Hq, Hkv, L, S, D) > (rows + 255) // 256 * 256


def _bounds(want, q, k, v, g, seen, bias=None):
    bounds = [TOL_REL_FP32 * max(1.0, float(w.abs().max())) for w in want]
    return [bounds[0], bounds[1] + _noise(q, k, v, g, seen, bias), bounds[2]]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,causal,lens", [
    (3, 6, 2, 330, 450, False, None),
    (4, 8, 8, 300, 300, True, None),
    (5, 4, 2, 129, 1000, "bottom-right", (1000, 129, 0, 64, 577)),
    (1, 2, 1, 1601, 1601, True, None),          # few query tiles: their walks are divided
    (2, 6, 3, 321, 640, False, (640, 65)),
    (2, 6, 3, 321, 640, False, (1, 17)),        # less than a key tile
])
def test_dq_from_stored_tiles(D, B, Hq, Hkv, L, S, causal, lens):
    from tinytorch_b200 import _capi, op
    _, q, k, v, g = _make(D, B, Hq, Hkv, L, S)
    assert _stored(D, B, Hq, Hkv, L, S)
    n = None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda")
    seen = _seen(B, L, S, causal, n)
    want = _reference(q, k, v, g, seen, None)
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=n)
    got = op.sdpAttentionBwd(g, q, k, v, o, lse, isCausal=causal, kvLens=n)
    again = op.sdpAttentionBwd(g, q, k, v, o, lse, isCausal=causal, kvLens=n)
    dq, = (t for t in op.sdpAttentionBwd(g, q, k, v, o, lse, isCausal=causal, kvLens=n, needs=(True, False, False)) if t is not None)
    # the same call with the scratch memory of the other path
    ws = torch.empty((B * Hq * L * 4 + 255) // 256 * 256, dtype=torch.uint8, device="cuda")
    grads = [torch.empty_like(t) for t in (q, k, v)]
    p = _params(q, k, v, o, lse, g, grads, causal, n)
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    _capi.check(_capi.lib().tt_attn_bwd(C.byref(p)))
    for i, (w, bound) in enumerate(zip(want, _bounds(want, q, k, v, g, seen))):
        assert torch.equal(got[i], again[i])
        for t in (got[i], grads[i]) + ((dq,) if i == 0 else ()):
            assert bool(((t.double() - w).abs() <= bound).all()), (i, float((t.double() - w).abs().max()))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["bool", "row", "add"])
@pytest.mark.parametrize("B,Hq,Hkv,L,S", [(16, 8, 8, 130, 190), (3, 6, 2, 330, 450)])  # undivided; divided
def test_dq_from_stored_tiles_masked(D, kind, B, Hq, Hkv, L, S):
    from tinytorch_b200 import op
    gen, q, k, v, g = _make(D, B, Hq, Hkv, L, S)
    assert _stored(D, B, Hq, Hkv, L, S)
    bias, seen = None, torch.ones(1, 1, 1, 1, dtype=torch.bool, device="cuda")
    if kind == "add":
        mask = bias = torch.randn(1, Hq, L, S, device="cuda", generator=gen)
    else:
        mask = seen = torch.rand((B, 1, 1, S) if kind == "row" else (B, Hq, L, S), device="cuda", generator=gen) < 0.7
        if kind == "bool":
            mask[0, :, 3] = False  # a row without any key
    want = _reference(q, k, v, g, seen, bias)
    o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask)
    for t, w, bound in zip(op.sdpAttentionBwd(g, q, k, v, o, lse, attnMask=mask), want, _bounds(want, q, k, v, g, seen, bias)):
        assert bool(((t.double() - w).abs() <= bound).all()), float((t.double() - w).abs().max())


def test_an_allocator_without_room_for_the_tiles():
    """It is asked once more, for what the other path needs, and gets back what it gave."""
    from tinytorch_b200 import _capi, op
    D, B, Hq, Hkv, L, S = 64, 4, 8, 8, 300, 300
    _, q, k, v, g = _make(D, B, Hq, Hkv, L, S)
    assert _stored(D, B, Hq, Hkv, L, S)
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=True)
    least = (B * Hq * L * 4 + 255) // 256 * 256
    asked, freed, ws = [], [], torch.empty(least, dtype=torch.uint8, device="cuda")

    def alloc(ctx, size, device):
        asked.append(size)
        return ws.data_ptr() if size <= least else None

    hook = _capi.AllocHook(_capi.ALLOC_FN(alloc), _capi.FREE_FN(lambda ctx, ptr, device: freed.append(ptr)), None)
    grads = [torch.empty_like(t) for t in (q, k, v)]
    p = _params(q, k, v, o, lse, g, grads, True, None)
    p.alloc = C.pointer(hook)
    _capi.check(_capi.lib().tt_attn_bwd(C.byref(p)))
    assert len(asked) == 2 and asked[0] > least and asked[1] == least and freed == [ws.data_ptr()]
    # the bits of the same path in a caller's buffer
    want = [torch.empty_like(t) for t in (q, k, v)]
    p = _params(q, k, v, o, lse, g, want, True, None)
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    _capi.check(_capi.lib().tt_attn_bwd(C.byref(p)))
    assert all(torch.equal(a, b) for a, b in zip(grads, want))
