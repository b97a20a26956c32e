"""GPU: the fp32 backward where the walk of a tile is divided among the CTAs of a cluster (few tiles, or several query heads per
kv head), against the CPU oracle: shares of unequal length, shares without steps, keys and rows that take no part, masks.
Tolerance: that of test_bwd_gpu.py for fp32."""
import numpy as np
import pytest
import torch

from conftest import rel_err
from gpu_util import TOL_REL_FP32, make, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,causal,lens,mask", [
    (1, 8, 1, 130, 130, True, None, None),         # walks of 8 .. 24 steps in 8 shares
    (1, 2, 2, 500, 500, True, None, None),         # late key tiles and early query tiles: fewer steps than shares (8; D = 128: 4)
    (2, 4, 2, 65, 300, False, (300, 70), None),    # key tiles without keys, 4 shares
    (1, 2, 2, 100, 65, False, None, None),         # 2 shares
    (8, 8, 8, 100, 100, True, None, None),         # not divided
    (1, 3, 1, 200, 129, False, None, "f32"),
    (2, 2, 1, 100, 190, False, None, "bool"),
])
def test_divided_walks_fp32(oracle, D, B, Hq, Hkv, L, S, causal, lens, mask):
    from tinytorch_b200 import op
    q, qn = make((B, Hq, L, D), torch.float32, 71)
    k, kn = make((B, Hkv, S, D), torch.float32, 72)
    v, vn = make((B, Hkv, S, D), torch.float32, 73)
    do, don = make((B, Hq, L, D), torch.float32, 74)
    rng = np.random.default_rng(75)
    kw, t = {}, None
    if mask == "f32":
        m = rng.standard_normal((1, Hq, L, S)).astype(np.float32)
        t, kw["bias"] = torch.from_numpy(m).cuda(), np.broadcast_to(m, (B, Hq, L, S))
    elif mask == "bool":
        m = rng.random((B, 1, L, S)) < 0.6
        m[..., 0] = True
        t, kw["bias"] = torch.from_numpy(m).cuda(), np.where(m, np.float32(0), np.float32(-np.inf))
    ln = None if lens is None else np.array(lens, dtype=np.int32)
    dl = None if ln is None else torch.from_numpy(ln).cuda()
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=dl, attnMask=t)
    got = op.sdpAttentionBwd(do, q, k, v, o, lse, isCausal=causal, kvLens=dl, attnMask=t)
    again = op.sdpAttentionBwd(do, q, k, v, o, lse, isCausal=causal, kvLens=dl, attnMask=t)
    if mask is None:
        kw = dict(causal=causal, kv_lens=ln)
    want = oracle.bwd(qn, kn, vn, don, **kw)
    for g, a, w in zip(got, again, want):
        assert torch.equal(g, a)  # (summed in order)
        assert rel_err(to_np(g), w) <= TOL_REL_FP32
