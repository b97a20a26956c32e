"""GPU: masks of the fp32 kernels where their tiles are staged through shared memory: boolean rows at every byte offset,
masks that are the same for all rows (of a sequence, or of a head), additive ones; tiles ragged in both directions; rows without any key; with
and without a divided walk, over enough key tiles that each of two places is used again.

Reference: the composition in fp64.  Bound: that of the fp32 tests (1e-5 of the largest element)."""
import pytest
import torch

from gpu_util import TOL_REL_FP32

pytestmark = pytest.mark.gpu


def _reference(q, k, v, g, mask):
    q, k, v = (t.double().requires_grad_() for t in (q, k, v))
    group = q.shape[1] // k.shape[1]
    s = q @ k.repeat_interleave(group, 1).transpose(2, 3) * q.shape[3] ** -0.5
    s = s.masked_fill(~mask, float("-inf")) if mask.dtype == torch.bool else s + mask.double()
    p = torch.nan_to_num(s.softmax(-1))  # a row without any key: zeros
    o = p @ v.repeat_interleave(group, 1)
    return (o.detach(),) + torch.autograd.grad(o, (q, k, v), g.double())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["bool", "row", "headrow", "add", "addrow", "lowest"])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,offset", [
    (1, 2, 1, 65, 131, 0),      # rows of an odd length: every alignment in turn; a divided walk
    (2, 2, 2, 64, 64, 3),       # ... and a mask that starts in the middle of a word
    (1, 1, 1, 1, 5, 1),
    (9, 8, 4, 130, 193, 2),     # more CTAs than SMs
    (3, 32, 32, 300, 333, 1),   # ... than two to an SM
])
def test_staged_masks(D, kind, B, Hq, Hkv, L, S, offset):
    from tinytorch_b200 import op
    gen = torch.Generator("cuda").manual_seed(D + L + S + offset)
    q, k, v, g = (torch.randn(s, device="cuda", generator=gen) for s in ((B, Hq, L, D), (B, Hkv, S, D), (B, Hkv, S, D), (B, Hq, L, D)))
    shape = {"row": (B, 1, 1, S), "addrow": (B, 1, 1, S), "headrow": (1, Hq, 1, S)}.get(kind, (1, Hq, L, S))
    n = torch.Size(shape).numel()
    if kind in ("bool", "row", "headrow"):
        mask = (torch.rand(n + offset, device="cuda", generator=gen) < 0.6)[offset:].view(shape)
        if kind == "bool" and L > 2:
            mask[0, :, 2] = False  # a row without any key
    else:
        mask = torch.randn(n + offset, device="cuda", generator=gen)[offset:].view(shape)
        if kind == "lowest":
            mask = torch.where(mask > 0.5, torch.finfo(torch.float32).min, 0.0)
            mask[..., 0] = 0.0
    o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask)
    got = (o,) + tuple(op.sdpAttentionBwd(g, q, k, v, o, lse, attnMask=mask))
    for a, b in zip(got, _reference(q, k, v, g, mask)):
        assert float((a.double() - b).abs().max()) <= TOL_REL_FP32 * max(1.0, float(b.abs().max()))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,L,S", [(1, 2, 70, 300), (5, 16, 150, 200)])  # divided and undivided
@pytest.mark.parametrize("rows", [False, True])
def test_hidden_keys_may_hold_anything(D, B, H, L, S, rows):
    """A key that a boolean mask hides takes no part whatever its score comes to."""
    from tinytorch_b200 import op
    gen = torch.Generator("cuda").manual_seed(D + L)
    q, k, v = (torch.randn(s, device="cuda", generator=gen) for s in ((B, H, L, D), (B, H, S, D), (B, H, S, D)))
    hidden = torch.rand(S, device="cuda", generator=gen) < 0.4
    mask = (~hidden).expand(1, 1, L, S).contiguous() if rows else (~hidden).view(1, 1, 1, S)
    want, _ = op.sdpAttentionFwd(q, k, v, attnMask=mask)
    for bad in (float("nan"), float("inf"), 3e38):
        got, _ = op.sdpAttentionFwd(q, torch.where(hidden[:, None], bad, k), v, attnMask=mask)
        assert torch.equal(got, want)
