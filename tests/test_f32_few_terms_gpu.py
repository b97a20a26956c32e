"""GPU: fp32 attention whose rows have few terms.  An infinity, or a sum that is too large for a float, stays an infinity whatever the number of
terms: with 1, 7, 32 and 33 keys (queries, for the keys' gradients), under a causal mask, where the first rows of every call have few, and
in both head dimensions; and so does one whose factor is so small that the lower pieces of it are below what a bf16 holds.

Reference: the composition in fp64, formula by formula; which elements are infinite or NaN has to agree."""
import math

import pytest
import torch

from gpu_util import TOL_REL_FP32

pytestmark = pytest.mark.gpu


def _tensors(L, S, D, seed=3):
    gen = torch.Generator("cuda").manual_seed(seed)
    return [torch.randn((2, 2, n, D), device="cuda", generator=gen) for n in (L, S, S, L)]


def _probabilities(q, k, causal):
    s = q.double() @ k.double().transpose(2, 3) * q.shape[3] ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(s.shape[2:], device="cuda").triu(1).bool(), -math.inf)
    return s.softmax(-1)


def _same(got, want):
    """Infinities and NaN in the same places, the rest close."""
    want = want.where(want.abs() < 3.4028235e38, want * math.inf)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(torch.sign(got[torch.isinf(got)]).double(), torch.sign(want[torch.isinf(want)]))
    ok = torch.isfinite(want)
    assert bool(((got.double() - want)[ok].abs() <= TOL_REL_FP32 * want[ok].abs().clamp_min(1.0)).all())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("S", [1, 7, 32, 33, 150])
def test_infinities_in_v(S, causal, D):
    from tinytorch_b200 import op
    q, k, v, _ = _tensors(S, S, D)
    v[0, 0, S // 2, 5], v[1, 1, 0, 0], v[1, 1, S - 1, D - 1] = math.inf, -math.inf, math.inf
    o, _ = op.sdpAttentionFwd(q, k, v, isCausal=causal)
    p = _probabilities(q, k, causal)
    seen = p > 0
    want = p @ v.double()
    if causal:  # what lies behind the diagonal reaches the rows that share a tile with it, or none: not compared
        spoilt = torch.isnan(want)
        assert bool((~torch.isnan(o) | spoilt).all())
        o, want = o.where(~spoilt, torch.zeros_like(o)), want.where(~spoilt, torch.zeros_like(want))
    assert bool(seen[..., 0].all())
    _same(o, want)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("S", [2, 7, 32, 33])
def test_sums_of_v_that_overflow(S, causal, D):
    """Equal scores: the sum over the keys, before it is divided by their number, is beyond a float's range from the second key on."""
    from tinytorch_b200 import op
    q, k, v, _ = _tensors(S, S, D)
    k.zero_()
    v[0, 1, :, 7], v[0, 1, :, 8] = 3.0e38, -3.0e38
    o, _ = op.sdpAttentionFwd(q, k, v, isCausal=causal)
    want = _probabilities(q, k, causal) @ v.double()
    first = 1 if causal else 0
    want[0, 1, first:, 7], want[0, 1, first:, 8] = math.inf, -math.inf
    _same(o, want)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("value", [math.inf, 3.0e38])
@pytest.mark.parametrize("L,S", [(1, 40), (7, 7), (32, 130), (33, 33), (40, 1), (130, 32)])
def test_dv_and_dq_of_large_gradients(L, S, value, D):
    """A column of dO that is infinite, or whose sums over the queries are; equal scores, so that nothing else is lost in them."""
    from tinytorch_b200 import op
    q, k, v, g = _tensors(L, S, D)
    k.zero_()
    g[0, 0, :, 5] = value
    o, lse = op.sdpAttentionFwd(q, k, v)
    dq, dk, dv = op.sdpAttentionBwd(g, q, k, v, o, lse)
    p = _probabilities(q, k, False)
    _same(dv, p.transpose(2, 3) @ g.double())  # (each term has a probability of 1 / S)
    if S == 1 and value == 3.0e38:  # dP and delta are one and the same infinity, or the same number
        return
    finite = torch.ones_like(dq, dtype=torch.bool)
    finite[0, 0] = False
    assert bool(torch.isfinite(dq[finite]).all()) and bool((dq[finite] == 0).all())  # (dQ = dS K, and K is 0)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S", [2, 31, 32, 33])
def test_dq_that_overflows(S, D):
    """dQ = dS K with finite dS and finite K whose products are too large together."""
    from tinytorch_b200 import op
    q, k, v, g = _tensors(40, S, D)
    sign = torch.where(torch.arange(S, device="cuda") % 2 == 0, 1.0, -1.0)
    q[0, 0, :, 3], k[0, 0] = 0.0, 0.0  # (scores of 0: probabilities of 1 / S)
    k[0, 0, :, 3] = 2.0e38 * sign
    v[0, 0], g[0, 0] = 0.0, 0.0
    v[0, 0, :, 0], g[0, 0, :, 0] = 40.0 * sign, 1.0  # dS of about +-40 / S
    o, lse = op.sdpAttentionFwd(q, k, v)
    dq = op.sdpAttentionBwd(g, q, k, v, o, lse)[0]
    assert bool(torch.isposinf(dq[0, 0, :, 3]).all())
    rest = torch.ones(D, dtype=torch.bool, device="cuda")
    rest[3] = False
    assert bool(torch.isfinite(dq[0, 0][:, rest]).all()) and bool(torch.isfinite(dq[0, 1]).all()) and bool(torch.isfinite(dq[1]).all())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S", [2, 90])
def test_infinities_with_small_probabilities(S, D):
    """Probabilities from 1 down to 2^-118 (and 1 / 89 of that), with an infinite V and with an infinite dO."""
    from tinytorch_b200 import op
    L = 252
    q, k, v, g = (torch.zeros((1, 1, n, D), device="cuda") for n in (L, S, S, L))
    v.normal_(), g.normal_()
    steps = torch.arange(L, device="cuda") * 0.47  # what the last key's exponents are below the others
    q[0, 0, :, 0], k[0, 0, S - 1, 0] = steps, -1.0
    v[0, 0, S - 1, 3], g[0, 0, :, 5] = math.inf, -math.inf
    o, lse = op.sdpAttentionFwd(q, k, v, scale=math.log(2.0))
    assert bool(torch.isposinf(o[..., 3]).all()) and int((~torch.isfinite(o)).sum()) == L
    v[0, 0, S - 1, 3] = 0.0
    o, lse = op.sdpAttentionFwd(q, k, v, scale=math.log(2.0))
    for row in (slice(0, L), slice(200, 201), slice(L - 1, L)):  # all rows; one whose probability of the last key is small
        dv = op.sdpAttentionBwd(g[:, :, row], q[:, :, row], k, v, o[:, :, row], lse[:, :, row].clone(), scale=math.log(2.0))[2]
        assert bool(torch.isneginf(dv[..., 5]).all()) and int((~torch.isfinite(dv)).sum()) == S


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("small", [0.5, 1e-30, 1e-34, 1e-37, 2.0 ** -126, 2.0 ** -133, 1e-42])
def test_keys_hidden_by_small_queries(small, D):
    """A small number times -inf is -inf: the key takes no part, and the others are what they would be without it."""
    from tinytorch_b200 import op
    q, k, v, _ = _tensors(40, 90, D)
    q[..., 3], k[..., 3] = small, 0.0
    k[:, :, 70, 3] = -math.inf
    o, lse = op.sdpAttentionFwd(q, k, v)
    others = torch.arange(90, device="cuda") != 70
    want = _probabilities(q, k[:, :, others], False) @ v[:, :, others].double()
    _same(o, want)
    assert bool(torch.isfinite(lse).all())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("small", [1e-20, 1e-30, 3e-33])
@pytest.mark.parametrize("large", [3.4e38, math.inf])
def test_small_values_beside_large_ones(large, small, D):
    """What has been split a second time, into truncated pieces, is as accurate relative to itself, however small.  (The products of pieces that are left out all
    have the sign of the whole then, and take up to 2^-20 of it; the third pieces of 3e-33 are the smallest numbers that a bf16 has.)"""
    from tinytorch_b200 import op
    q, k, v, g = _tensors(140, 150, D)
    v[0, 0, 11, 1] = large
    v[0, 0, :, 2] = small * (1 + torch.rand(150, device="cuda"))
    g[1, 1, 7, 3] = large
    g[1, 1, :, 4] = small * (1 + torch.rand(140, device="cuda"))
    o, lse = op.sdpAttentionFwd(q, k, v)
    p = _probabilities(q, k, False)
    want = (p @ v.double())[0, 0, :, 2]
    assert bool(((o[0, 0, :, 2].double() - want).abs() <= TOL_REL_FP32 * want).all())
    v[0, 0, 11, 1] = 0.0
    o, lse = op.sdpAttentionFwd(q, k, v)
    dv = op.sdpAttentionBwd(g, q, k, v, o, lse)[2]
    want = (p.transpose(2, 3) @ g.double())[1, 1, :, 4]
    assert bool(((dv[1, 1, :, 4].double() - want).abs() <= TOL_REL_FP32 * want).all())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("exponent,bits", [(-100, 23), (-108, 23), (-115, 18), (-120, 13), (-124, 9)])
def test_how_accurate_small_values_are(exponent, bits, D):
    """One key: O is V.  A float is the sum of its pieces, exactly, down to 2^-110; below, the last piece is a multiple of 2^-133 and the
    value is off by half of that at most, 2^(-134 - exponent) of itself."""
    from tinytorch_b200 import op
    q, k, v, g = _tensors(40, 1, D)
    v = (1 + torch.rand_like(v)) * 2.0 ** exponent
    o, lse = op.sdpAttentionFwd(q, k, v)
    assert bool(((o - v).abs().double() <= 2.0 ** -bits * v.double()).all())
    dv = op.sdpAttentionBwd(v.expand(2, 2, 40, D).contiguous(), q, k, v, o, lse)[2]
    want = 40 * v.double()
    assert bool(((dv - want).abs() <= (2.0 ** -bits + TOL_REL_FP32) * want).all())
