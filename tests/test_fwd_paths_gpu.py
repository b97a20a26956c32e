"""GPU: the prefill forward where a query block's keys are divided between the halves of a CTA and among clusters (few
queries, many keys), beside the pairs of blocks that shorter walks get, and where the two query blocks of an item belong to
different heads, against the CPU oracle.  The comments say what plan_of takes on 148 SMs.  Tolerances: those of test_fwd_gpu.py."""
import numpy as np
import pytest
import torch

from gpu_util import TOL_ABS_16BIT, check_status, make, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,L,S,causal,lens", [
    (1, 2, 2, 128, 768, False, None),                 # halves, 6 key tiles
    (1, 3, 1, 100, 384, False, None),                 # pairs, 3 key tiles
    (2, 20, 20, 600, 600, True, None),                # pairs, 200 blocks
    (1, 2, 1, 64, 100, False, None),                  # pairs, one key tile
    (1, 4, 1, 129, 1537, "bottom-right", None),       # clusters of 8, a block of one row
    (2, 3, 1, 40, 3100, "bottom-right", (3100, 700)),  # clusters of 8, an odd number of blocks, CTAs without keys
    (2, 2, 2, 300, 3072, False, (1, 0)),              # clusters of 8: a sequence without keys, one with a single key
    (3, 8, 2, 64, 1100, False, (1100, 128, 129)),      # halves (D = 128: clusters of 4): one key tile, a half without any
    (1, 4, 4, 512, 900, True, None),                  # halves, 1 .. 4 key tiles
    (1, 2, 1, 1024, 1024, True, None),                # halves (D = 128: clusters of 4): shares of a triangle
    (1, 4, 4, 64, 520, False, None),                  # halves, an odd number of key tiles
    (2, 40, 8, 129, 700, "bottom-right", (700, 131)),  # halves, 160 blocks: CTAs with a second item
    (2, 20, 20, 100, 1930, False, (1930, 60)),        # clusters of 2, one CTA of which has no keys
    (1, 20, 4, 64, 1700, False, None),                # clusters of 4
])
def test_keys_divided_among_a_cluster(oracle, dt, D, B, Hq, Hkv, L, S, causal, lens):
    from tinytorch_b200 import op
    dtype = {"bf16": torch.bfloat16, "f16": torch.float16}[dt]
    q, qn = make((B, Hq, L, D), dtype, 11)
    k, kn = make((B, Hkv, S, D), dtype, 12)
    v, vn = make((B, Hkv, S, D), dtype, 13)
    ln = None if lens is None else np.array(lens, dtype=np.int32)
    dl = None if ln is None else torch.from_numpy(ln).cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=dl, status=status)
    again, _ = op.sdpAttentionFwd(q, k, v, isCausal=causal, kvLens=dl)
    check_status(status)
    assert torch.equal(o, again)  # (each row is summed by one CTA, in a fixed order)
    if causal == "bottom-right":  # as an additive mask
        lim = np.arange(L)[None, :, None] + ((np.full(B, S) if ln is None else ln)[:, None, None] - L)
        bias = np.where(np.arange(S)[None, None, :] <= lim, 0.0, -1e30).astype(np.float32)[:, None]
        want, wl = oracle.fwd(qn, kn, vn, kv_lens=ln, bias=bias)
    else:
        want, wl = oracle.fwd(qn, kn, vn, causal=causal, kv_lens=ln)
    if ln is not None:
        want[ln == 0] = 0.0  # a row without keys gives 0 (the reference: NaN)
    assert np.abs(to_np(o) - want).max() <= TOL_ABS_16BIT
    got = lse.cpu().numpy()
    fin = np.isfinite(wl)
    assert np.array_equal(fin, np.isfinite(got))
    assert np.abs(got[fin] - wl[fin]).max() <= 2e-3


@pytest.mark.parametrize("Hq,Hkv,L", [(6, 2, 130), (5, 1, 257), (7, 7, 383)])
def test_blocks_of_different_heads_share_an_item(oracle, Hq, Hkv, L):
    from tinytorch_b200 import op
    q, qn = make((2, Hq, L, 128), torch.bfloat16, 21)
    k, kn = make((2, Hkv, L, 128), torch.bfloat16, 22)
    v, vn = make((2, Hkv, L, 128), torch.bfloat16, 23)
    o, lse = op.sdpAttentionFwd(q, k, v, isCausal=True)
    want, wl = oracle.fwd(qn, kn, vn, causal=True)
    assert np.abs(to_np(o) - want).max() <= TOL_ABS_16BIT
    assert np.abs(lse.cpu().numpy() - wl).max() <= 2e-3
