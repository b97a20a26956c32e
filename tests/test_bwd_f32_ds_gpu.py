"""GPU: the fp32 backward whose dQ pass reads the dS tiles that the dK / dV pass leaves: ragged tiles, several query heads per kv head,
both causal alignments, sequences without keys, masks, undivided and divided walks; and the same call without room for dS.

Reference: the composition in fp64.  Bound: that of the fp32 tests (1e-5 of the largest element, and of 1).  It does not hold for a
sequence of which all rows see one and the same key: dS is then the difference of two equal sums of D products, dO V and dO O, and dK,
which is 0, the sum of their roundings over all rows; 642 rows leave up to 1.2e-5 (D = 64) or 1.6e-5 (D = 128) of the formula itself,
evaluated in fp32 on the CPU.  With n keys every term carries a probability of about 1 / n; the shortest such sequence here has 65."""
import ctypes as C

import pytest
import torch

from gpu_util import TOL_REL_FP32

pytestmark = pytest.mark.gpu


def _reference(q, k, v, g, seen):
    q, k, v = (t.double().requires_grad_() for t in (q, k, v))
    group = q.shape[1] // k.shape[1]
    s = (q @ k.repeat_interleave(group, 1).transpose(2, 3) * q.shape[3] ** -0.5).masked_fill(~seen, float("-inf"))
    o = torch.nan_to_num(s.softmax(-1)) @ v.repeat_interleave(group, 1)
    return torch.autograd.grad(o, (q, k, v), g.double())


def _seen(B, L, S, causal, lens):
    j, i = torch.arange(S, device="cuda"), torch.arange(L, device="cuda")[:, None]
    n = torch.full((B, 1, 1), S, device="cuda") if lens is None else lens.long()[:, None, None]
    seen = (j < n).expand(B, L, S)
    if causal:
        seen = seen & (j <= i + (n - L if causal == "bottom-right" else 0))
    return seen[:, None]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,causal,lens", [
    (3, 6, 2, 330, 450, False, None),
    (4, 8, 8, 300, 300, True, None),
    (5, 4, 2, 129, 1000, "bottom-right", (1000, 129, 0, 64, 577)),
    (1, 2, 1, 1601, 1601, True, None),          # few query tiles: their walks are divided
    (2, 6, 3, 321, 640, False, (640, 65)),
])
def test_dq_from_stored_tiles(D, B, Hq, Hkv, L, S, causal, lens):
    from tinytorch_b200 import _capi, op
    gen = torch.Generator("cuda").manual_seed(D + L)
    q, k, v, g = (torch.randn(s, device="cuda", generator=gen) for s in ((B, Hq, L, D), (B, Hkv, S, D), (B, Hkv, S, D), (B, Hq, L, D)))
    rows = B * Hq * L * 4
    assert op.workspaceBytes(_capi.KIND_BWD, torch.float32, B, Hq, Hkv, L, S, D) > (rows + 255) // 256 * 256
    n = None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda")
    want = _reference(q, k, v, g, _seen(B, L, S, causal, n))
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=n)
    got = op.sdpAttentionBwd(g, q, k, v, o, lse, isCausal=causal, kvLens=n)
    again = op.sdpAttentionBwd(g, q, k, v, o, lse, isCausal=causal, kvLens=n)
    dq, = (t for t in op.sdpAttentionBwd(g, q, k, v, o, lse, isCausal=causal, kvLens=n, needs=(True, False, False)) if t is not None)
    # the same call with the scratch memory of the other path
    p, ws = _capi.BwdParams(), torch.empty((rows + 255) // 256 * 256, dtype=torch.uint8, device="cuda")
    grads = [torch.empty_like(t) for t in (q, k, v)]
    p.struct_size, p.dtype, p.B, p.Hq, p.Hkv, p.Lq, p.Skv, p.D = C.sizeof(p), _capi.F32, B, Hq, Hkv, L, S, D
    for name, t in (("q", q), ("k", k), ("v", v), ("o", o), ("d_o", g), ("lse", lse), ("dq", grads[0]), ("dk", grads[1]), ("dv", grads[2])):
        setattr(p, name, t.data_ptr())
    if n is not None:
        p.kv_lens = n.data_ptr()
    p.is_causal, p.scale = op._causal_mode(causal), D ** -0.5
    p.device, p.stream = torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    _capi.check(_capi.lib().tt_attn_bwd(C.byref(p)))
    for i, w in enumerate(want):
        bound = TOL_REL_FP32 * max(1.0, float(w.abs().max()))
        assert torch.equal(got[i], again[i])
        for t in (got[i], grads[i]) + ((dq,) if i == 0 else ()):
            assert float((t.double() - w).abs().max()) <= bound
