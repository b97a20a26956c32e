"""GPU: the fp32 forward where the key tiles of a query tile are divided among the CTAs of a cluster (few query tiles), against
the CPU oracle: 2, 4 and 8 shares, shares without key tiles, sequences without keys, masks, ragged ends.
Tolerance: that of test_fwd_gpu.py for fp32."""
import numpy as np
import pytest
import torch

from conftest import rel_err
from gpu_util import TOL_REL_FP32, make, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,causal,lens,mask", [
    (1, 2, 1, 70, 256, False, None, False),             # 4 key tiles in 4 shares
    (1, 2, 2, 64, 1030, False, None, False),            # 17 in 8
    (2, 3, 3, 500, 500, True, None, False),             # 1 .. 8 tiles in 4 shares: early query tiles leave some empty
    (3, 2, 1, 100, 700, "bottom-right", (700, 30, 0), False),
    (2, 2, 1, 65, 600, False, (600, 1), True),
    (1, 3, 3, 200, 128, False, None, False),            # 2 in 2
    (16, 8, 4, 100, 300, False, None, False),           # 5 in 2 (D = 128: not divided)
    (1, 1, 1, 1, 65, False, None, False),               # 2 in 2
])
def test_divided_keys_fp32(oracle, D, B, Hq, Hkv, L, S, causal, lens, mask):
    from tinytorch_b200 import op
    q, qn = make((B, Hq, L, D), torch.float32, 61)
    k, kn = make((B, Hkv, S, D), torch.float32, 62)
    v, vn = make((B, Hkv, S, D), torch.float32, 63)
    ln = np.array(lens if lens else (S,) * B, dtype=np.int32)
    j, i = np.arange(S)[None, None, None, :], np.arange(L)[None, None, :, None]
    seen = j < ln[:, None, None, None]
    if causal:
        seen = seen & (j <= i + (ln[:, None, None, None] - L if causal == "bottom-right" else 0))
    seen = np.broadcast_to(seen, (B, 1, L, S)).copy()
    t = None
    if mask:
        m = np.random.default_rng(64).random((B, 1, L, S)) < 0.5
        t = torch.from_numpy(m).cuda()
        seen &= m
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=torch.from_numpy(ln).cuda() if lens else None, attnMask=t)
    torch.cuda.synchronize()
    some = np.broadcast_to(seen.any(-1), (B, Hq, L))  # rows that see a key
    bias = np.where(seen, 0.0, -1e30).astype(np.float32)
    want_o, want_l = oracle.fwd(qn, kn, vn, bias=bias)
    got_o, got_l = to_np(o), to_np(lse)
    assert rel_err(got_o[some], want_o[some]) <= TOL_REL_FP32
    assert np.abs(got_l[some] - want_l[some]).max() <= 1e-4
    assert (got_o[~some] == 0).all() and np.isneginf(got_l[~some]).all()


def _median_us(f, n=40):
    for _ in range(5):
        f()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(n + 1)]
    ev[0].record()
    for e in ev[1:]:
        f()
        e.record()
    torch.cuda.synchronize()
    return sorted(a.elapsed_time(b) for a, b in zip(ev, ev[1:]))[n // 2] * 1e3


@pytest.mark.parametrize("fewer,more", [(15, 16), (33, 34)])  # query tiles in clusters of 8 and of 4, around what 132..148 SMs hold
def test_no_round_for_a_cluster_too_many(fewer, more):
    """Clusters that the GPCs have no room for, one to an SM, share SMs with others instead of waiting for all of them to end (which takes
    twice the time; sharing measured 1.4 times)."""
    from tinytorch_b200 import op
    us = []
    for heads in (fewer, more):
        q, k = torch.randn(1, heads, 64, 64, device="cuda"), torch.randn(1, heads, 4000, 64, device="cuda")
        us.append(min(_median_us(lambda: op.sdpAttentionFwd(q, k, k)) for _ in range(3)))
    assert us[1] <= 1.7 * us[0], us


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S", [1, 63, 64, 65, 128, 129, 192])  # either side of what counts as a short walk
@pytest.mark.parametrize("causal,lens", [(False, False), (True, False), ("bottom-right", True)])
def test_short_undivided_walks_fp32(D, S, causal, lens):
    """Against the composition in fp64; more query tiles than are ever divided."""
    from tinytorch_b200 import op
    B, Hq, Hkv, L = 10, 32, 8, 70
    gen = torch.Generator("cuda").manual_seed(S + D)
    q, k, v = (torch.randn(s, device="cuda", generator=gen) for s in ((B, Hq, L, D), (B, Hkv, S, D), (B, Hkv, S, D)))
    n = torch.randint(0, S + 1, (B,), dtype=torch.int32, device="cuda", generator=gen) if lens else None
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=n)
    rows = torch.full((B, 1, 1, 1), S, device="cuda") if n is None else n.view(B, 1, 1, 1).long()
    i, j = torch.arange(L, device="cuda").view(1, 1, L, 1), torch.arange(S, device="cuda")
    seen = (j < rows) & (j <= i + (rows - L if causal == "bottom-right" else 0) if causal else j >= 0)
    s = q.double() @ k.double().repeat_interleave(Hq // Hkv, 1).transpose(2, 3) * D ** -0.5
    s = s.masked_fill(~seen, float("-inf"))
    want = torch.nan_to_num(s.softmax(-1)) @ v.double().repeat_interleave(Hq // Hkv, 1)
    assert float((o.double() - want).abs().max()) <= TOL_REL_FP32 * max(1.0, float(want.abs().max()))
    some = seen.any(-1).expand(B, Hq, L)
    assert float((lse.double() - s.logsumexp(-1))[some].abs().max()) <= 1e-4 and bool(torch.isneginf(lse[~some]).all())
