"""GPU: how far fp32 attention is from 64 bits, on operands of all kinds: mixed signs, one sign, a common offset, small integers, rows with a
single element, scores so far apart that one key takes nearly all.

Bound (2-norm of the whole result): the distance that the reference's own fp32 arithmetic has on the same operands (the oracle: sums of
products one after the other, every addition rounded), and 2^-24 of the result for its last rounding.  For the gradients the kernels' probabilities come
of the log-sum-exp that the forward leaves in fp32, which is rounded three times on its way (as a sum, and by the factors to natural units and
back), each time by at most 2^-24 of itself: with the roundings independent and evenly distributed, a relative error of 2^-24 |lse| (2-norm over the rows) of
every probability, and twice that is allowed."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def _operands(kind, L, S, D):
    gen = torch.Generator("cuda").manual_seed(L + D)
    q, k, v, g = (torch.randn((1, 2, n, D), device="cuda", generator=gen) for n in (L, S, S, L))
    scale = D ** -0.5
    if kind == "positive":
        q, k, v, g = (t.uniform_(0.5, 1.5, generator=gen) for t in (q, k, v, g))
    elif kind == "offset":
        k, v = k + 4, v + 4
    elif kind == "integer":
        q, k = (torch.randint(-2, 3, t.shape, device="cuda", generator=gen).float() for t in (q, k))
    elif kind == "one-hot keys":
        k = torch.zeros_like(k)
        k[..., torch.arange(S), torch.arange(S) % D] = 1.0
        scale = 1.0
    elif kind == "sharp":
        scale = 1.0
    return q, k, v, g, scale


def _exact(q, k, v, g, scale, causal):
    q, k, v = (t.double().requires_grad_() for t in (q, k, v))
    s = q @ k.transpose(2, 3) * scale
    if causal:
        s = s.masked_fill(torch.ones(s.shape[2:], device="cuda").triu(1).bool(), -math.inf)
    o = s.softmax(-1) @ v
    return (o.detach(),) + torch.autograd.grad(o, (q, k, v), g.double())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["normal", "positive", "offset", "integer", "one-hot keys", "sharp"])
@pytest.mark.parametrize("L,S,causal", [(500, 500, False), (200, 200, True), (40, 40, False)])
def test_no_further_than_the_reference(oracle, kind, L, S, causal, D):
    from tinytorch_b200 import op
    q, k, v, g, scale = _operands(kind, L, S, D)
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, scale=scale)
    got = (o,) + tuple(op.sdpAttentionBwd(g, q, k, v, o, lse, isCausal=causal, scale=scale))
    want = _exact(q, k, v, g, scale, causal)
    host = [t.cpu().numpy() for t in (q, k, v, g)]
    theirs = (oracle.fwd(*host[:3], causal=causal, scale=scale)[0],) + tuple(oracle.bwd(*host, causal=causal, scale=scale))
    lse_rms = float(lse.double().square().mean().sqrt())
    for name, t, w, x in zip(("o", "dq", "dk", "dv"), got, want, theirs):
        norm = float(w.norm())
        ours = float((t.double() - w).norm()) / norm
        ref = float((torch.from_numpy(np.asarray(x)).cuda().double() - w).norm()) / norm
        bound = ref + U * (1 + (0 if name == "o" else 2 * lse_rms))
        print("%s %s D%d %d: ours %.2e reference %.2e ratio to bound %.2f" % (kind, name, D, L, ours, ref, ours / bound))
        assert ours <= bound


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S", [7, 33, 64, 500])
def test_one_key_that_takes_all_is_returned_as_it_is(S, D):
    """Probabilities of 1 and 0 (to a float): the output is the key's row of V, bit for bit."""
    from tinytorch_b200 import op
    gen = torch.Generator("cuda").manual_seed(S)
    signs = torch.randint(0, 2, (1, 2, S, D), device="cuda", generator=gen) * 2.0 - 1
    which = torch.randint(0, S, (1, 2, 150), device="cuda", generator=gen)[..., None].expand(1, 2, 150, D)
    v = torch.randn((1, 2, S, D), device="cuda", generator=gen)
    o, _ = op.sdpAttentionFwd(torch.gather(signs, 2, which), signs, v, scale=16.0)  # (scores apart by 16 for each sign that differs)
    assert torch.equal(o, torch.gather(v, 2, which))
