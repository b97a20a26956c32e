"""GPU: fp32 attention, forward and backward, whose products are sums of bf16 ones on the tensor cores (csrc/f32_pieces.cuh): the edges of
its tiles (128 rows of a group's queries, 64 keys), strided operands, scales of both signs and zero, masks at any offset, walks divided
over clusters, and values that are not finite.

Reference: the composition in fp64, formula by formula (a probability that is 0 takes part in products, as in the reference's).  Bound:
that of the fp32 tests, 1e-5 of the largest element, and of 1.  The error of a whole result (2-norm): a probability's relative error is the
absolute one of its exponent, score - lse, whose roundings grow with it; for inputs from N(0, 1) scores have the standard deviation
scale sqrt(D), and with 1 of it 8 * 2^-23 is twice the largest error measured (3.9e-7) and a tenth of the other bound."""
import math

import pytest
import torch

from gpu_util import TOL_REL_FP32

pytestmark = pytest.mark.gpu


def _reference(q, k, v, g=None, causal=False, lens=None, mask=None, scale=None):
    q, k, v = (t.detach().double().requires_grad_(g is not None) for t in (q, k, v))
    group, L, S = q.shape[1] // k.shape[1], q.shape[2], k.shape[2]
    kk, vv = k.repeat_interleave(group, 1), v.repeat_interleave(group, 1)
    s = q @ kk.transpose(2, 3) * (q.shape[3] ** -0.5 if scale is None else scale)
    if mask is not None:
        s = s.masked_fill(~mask, -math.inf) if mask.dtype == torch.bool else s + mask.double()
    j, i = torch.arange(S, device="cuda"), torch.arange(L, device="cuda")[:, None]
    n = torch.full((q.shape[0], 1, 1, 1), S, device="cuda") if lens is None else lens.long().view(-1, 1, 1, 1)
    seen = j < n
    if causal:
        seen = seen & (j <= i + (n - L if causal == "bottom-right" else 0))
    s = s.masked_fill(~seen, -math.inf)
    top = s.max(-1, keepdim=True).values
    p = torch.exp(s - torch.where(top == -math.inf, torch.zeros_like(top), top))
    total = p.sum(-1, keepdim=True)
    o = p @ vv / torch.where(total == 0, torch.ones_like(total), total)  # (0 where no key takes part)
    return (o.detach(),) + (torch.autograd.grad(o, (q, k, v), g.double()) if g is not None else ())


def _check(got, want, spread=1.0):  # of the scores
    for t, w in zip(got, want):
        err = (t.double() - w).abs()
        assert float(err.max()) <= TOL_REL_FP32 * max(1.0, float(w.abs().max()))
        if w.numel() >= 4096 and float(w.norm()) > 1e-3 * w.numel() ** 0.5:
            assert float(err.norm()) <= 8 * 2.0 ** -23 * max(1.0, spread) * float(w.norm())


def _run(q, k, v, g, **kw):
    from tinytorch_b200 import op
    names = dict(causal="isCausal", lens="kvLens", mask="attnMask", scale="scale")
    kw = {names[n]: x for n, x in kw.items() if x is not None}
    o, lse = op.sdpAttentionFwd(q, k, v, **kw)
    grads = op.sdpAttentionBwd(g, q, k, v, o, lse, **kw)
    torch.cuda.synchronize()
    return (o,) + tuple(grads)


def _tensors(B, Hq, Hkv, L, S, D, seed=7):
    gen = torch.Generator("cuda").manual_seed(seed)
    return [torch.randn(s, device="cuda", generator=gen) for s in ((B, Hq, L, D), (B, Hkv, S, D), (B, Hkv, S, D), (B, Hq, L, D))]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,causal,lens", [
    (1, 2, 2, 128, 64, False, None),            # one full tile
    (2, 6, 2, 43, 65, False, None),             # 129 rows of a group; one key more than a tile
    (1, 8, 2, 32, 63, True, None),              # a full tile of a group's rows
    (2, 4, 4, 127, 129, True, (129, 66)),
    (3, 4, 1, 70, 200, "bottom-right", (200, 70, 3)),   # queries that see no key
    (2, 2, 2, 5, 7, False, (0, 1)),             # a sequence without keys
    (64, 4, 4, 129, 130, False, None),          # more CTAs than SMs: nothing divided
    (1, 3, 1, 300, 1000, True, None),           # divided
])
def test_edges(D, B, Hq, Hkv, L, S, causal, lens):
    q, k, v, g = _tensors(B, Hq, Hkv, L, S, D)
    n = None if lens is None else torch.tensor(lens, dtype=torch.int32, device="cuda")
    if n is not None:  # rows behind the lengths are not looked at
        for b, m in enumerate(lens):
            k[b, :, m:], v[b, :, m:] = math.nan, math.inf
    got = _run(q, k, v, g, causal=causal, lens=n)
    for t in (k, v):
        t.nan_to_num_(0.0, 0.0)
    _check(got, _reference(q, k, v, g, causal=causal, lens=n))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("scale", [-0.2, 0.0, 1.5])
def test_strides_and_scales(D, scale):
    q, k, v, g = (torch.randn(s, device="cuda") for s in ((2, 70, 6, D), (2, 90, 2, D), (2, 90, 2, D), (2, 70, 6, D)))
    q, k, v, g = (t.transpose(1, 2) for t in (q, k, v, g))  # [B, S, heads, D] in memory
    _check(_run(q, k, v, g, scale=scale), _reference(q, k, v, g, scale=scale), abs(scale) * D ** 0.5)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["bool", "add", "row", "head row", "odd bool", "odd add"])
@pytest.mark.parametrize("B,Hq,Hkv,L,S", [(2, 6, 3, 75, 133), (40, 8, 8, 131, 132)])
def test_masks(D, kind, B, Hq, Hkv, L, S):
    q, k, v, g = _tensors(B, Hq, Hkv, L, S, D)
    shape = {"row": (B, 1, 1, S), "head row": (1, Hq, 1, S)}.get(kind.replace("odd ", ""), (1, Hq, L, S))
    if kind.startswith("odd"):  # a view that starts anywhere, with rows that lie anywhere
        mask = torch.randn(shape[:3] + (S + 3,), device="cuda")[..., 1:S + 1]
    else:
        mask = torch.randn(shape, device="cuda")
    if "bool" in kind:
        mask = (torch.randn(mask.shape[:3] + (S + 3,), device="cuda") < 0.5)[..., 3:] if "odd" in kind else mask < 0.5
        mask[:, :, L // 2:, 0] = True  # (rows before may see no key)
    _check(_run(q, k, v, g, mask=mask), _reference(q, k, v, g, mask=mask))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("where", ["q", "k", "v", "k nan", "v nan", "hidden k", "largest"])
def test_values_that_are_not_finite(D, where):
    """Infinities stay what they are: x * inf is an infinity, whatever pieces x consists of; what they do not reach is as accurate as ever."""
    from tinytorch_b200 import op
    q, k, v, _ = _tensors(1, 2, 2, 140, 150, D)
    q[:, :, :, 3] = torch.where(q[:, :, :, 3] > 0, 0.5, -2.0)  # (one piece: the others are zero)
    mask = None
    if where == "q":
        q[0, 0, 130, 3] = -math.inf
    elif where == "k":
        k[0, 0, 70, 3] = math.inf
    elif where == "v":
        v[0, 0, 140, 5], v[0, 1, 2, 6] = -math.inf, math.inf
    elif where == "k nan":
        k[0, 1, 9, 0] = math.nan
    elif where == "v nan":
        v[0, 1, 9, 0] = math.nan
    elif where == "hidden k":  # hidden, whatever the score
        mask = torch.ones(1, 1, 140, 150, dtype=torch.bool, device="cuda")
        mask[..., 70] = False
        k[0, 0, 70], k[0, 1, 70] = math.nan, 3.0e38
    else:  # too large for a bf16, and the small beside it
        v[0, 0, 11, 1], v[0, 0, :, 2] = 3.4e38, 1e-30
    o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask)
    kk = k if mask is None else torch.where(torch.isfinite(k) & (k.abs() < 1e38), k, torch.zeros_like(k))
    want, = _reference(q, kk, v, mask=mask)
    want = want.where(want.abs() < 3.4028235e38, want * math.inf)
    assert torch.equal(torch.isnan(o), torch.isnan(want)) and torch.equal(torch.isinf(o), torch.isinf(want))
    assert torch.equal(torch.sign(o[torch.isinf(o)]).double(), torch.sign(want[torch.isinf(want)]))
    ok = torch.isfinite(want)
    assert bool(((o.double() - want)[ok].abs() <= TOL_REL_FP32 * torch.clamp(want[ok].abs(), min=1.0)).all())


def test_gradients_of_infinite_inputs_are_not_spread():
    """An infinite element of dO reaches its row of dQ and its column of dV, and the keys' gradients, and nothing else."""
    q, k, v, g = _tensors(2, 2, 2, 140, 150, 64)
    g[0, 0, 131, 5] = math.inf
    o, dq, dk, dv = _run(q, k, v, g)
    assert bool(torch.isposinf(dv[0, 0, :, 5]).all())
    bad = [~torch.isfinite(t) for t in (dq, dk, dv)]
    assert int(bad[0].sum()) == 64 and bool(bad[0][0, 0, 131].all()) and int(bad[1].sum()) == 150 * 64 and int(bad[2].sum()) == 150
    g[0, 0, 131, 5] = 0.0
    want = _reference(q, k, v, g)
    for t, w, b in zip((dq, dk, dv), want[1:], bad):
        assert float((t.double() - w)[~b].abs().max()) <= TOL_REL_FP32 * max(1.0, float(w.abs().max()))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("value", [-2.0e38, -1.0e38, 2.0e38, -math.inf, torch.finfo(torch.float32).min])
def test_masks_of_large_values(D, value):
    """A row whose mask is one large value for all keys: their mean (the scores are lost in it); nothing where the value times log2(e),
    the unit of the exponents, is -inf.  A row that has it for some keys: the others'."""
    from tinytorch_b200 import op
    q, k, v, _ = _tensors(1, 2, 2, 70, 90, D)
    mask = torch.zeros(1, 1, 70, 90, device="cuda")
    mask[:, :, 5] = value
    mask[:, :, 6, 40:] = value
    o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask)
    plain = abs(value) * 1.4426950408889634 < 3.4028235e38
    # rounded additions of up to 90 terms of size 1, equally weighted
    want = v.double().mean(2) if plain else torch.zeros(1, 2, D, device="cuda", dtype=torch.float64)
    assert (o[:, :, 5] - want).abs().max() < 90 * 2.0 ** -24
    if not plain:
        assert torch.isneginf(lse[:, :, 5]).all()
    part = slice(40, 90) if value > 0 else slice(0, 40)
    if value < 0:
        want, = _reference(q[:, :, 6:7], k[:, :, part], v[:, :, part])
        assert (o[:, :, 6:7] - want).norm() < 1e-6 * want.norm()
    else:
        assert (o[:, :, 6] - v[:, :, part].double().mean(2)).abs().max() < 90 * 2.0 ** -24
    assert torch.isfinite(o).all()
