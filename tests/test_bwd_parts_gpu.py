"""GPU: the tensor-core backward where the walk of a key tile is divided among work items (few key tiles), against the CPU
oracle: shares of unequal length, shares without steps (late key tiles under a causal mask), key tiles that no query sees.
Tolerance: that of test_bwd_gpu.py."""
import numpy as np
import pytest
import torch

from gpu_util import assert_close_16bit, make, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,causal,lens", [
    (1, 4, 1, 640, 640, True, None),                   # 20 .. 4 steps per key tile in 7 shares
    (2, 3, 1, 300, 500, False, (500, 129)),            # 9 steps in 5 shares, key tiles without keys
    (1, 2, 2, 1100, 1100, True, None),
    (1, 4, 2, 260, 700, "bottom-right", None),
    (1, 2, 1, 200, 130, False, None),                  # a ragged second key tile (D = 64: not divided)
])
def test_divided_key_tiles(oracle, dt, D, B, Hq, Hkv, L, S, causal, lens):
    from tinytorch_b200 import op
    dtype = {"bf16": torch.bfloat16, "f16": torch.float16}[dt]
    q, qn = make((B, Hq, L, D), dtype, 31)
    k, kn = make((B, Hkv, S, D), dtype, 32)
    v, vn = make((B, Hkv, S, D), dtype, 33)
    do, don = make((B, Hq, L, D), dtype, 34)
    ln = None if lens is None else np.array(lens, dtype=np.int32)
    dl = None if ln is None else torch.from_numpy(ln).cuda()
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=dl)
    got = op.sdpAttentionBwd(do, q, k, v, o, lse, isCausal=causal, kvLens=dl)
    again = op.sdpAttentionBwd(do, q, k, v, o, lse, isCausal=causal, kvLens=dl)
    assert torch.equal(got[1], again[1]) and torch.equal(got[2], again[2])  # (the shares are added in order)
    kw = dict(causal=causal, kv_lens=ln)
    if causal == "bottom-right":  # as an additive mask
        lim = np.arange(L)[:, None] + (S - L)
        bias = np.where(np.arange(S)[None, :] <= lim, 0.0, -1e30).astype(np.float32)[None, None]
        kw = dict(bias=np.broadcast_to(bias, (B, 1, L, S)))
    want = oracle.bwd(qn, kn, vn, don, **kw)
    for name, g, w in zip(("dq", "dk", "dv"), got, want):
        assert_close_16bit(to_np(g), w, dtype, name)


def test_only_some_gradients_wanted():
    from tinytorch_b200 import op
    q, _ = make((1, 4, 640, 64), torch.bfloat16, 41)
    k, _ = make((1, 1, 640, 64), torch.bfloat16, 42)
    v, _ = make((1, 1, 640, 64), torch.bfloat16, 43)
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=True)
    dq, dk, dv = op.sdpAttentionBwd(o, q, k, v, o, lse, isCausal=True)
    for needs in ((False, True, False), (False, False, True), (True, False, False)):
        part = op.sdpAttentionBwd(o, q, k, v, o, lse, isCausal=True, needs=needs)
        for want, g, n in zip((dq, dk, dv), part, needs):
            assert (g is not None) == n
            if n and want is not dq:
                assert torch.equal(g, want)
