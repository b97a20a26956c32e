"""GPU: how the tensor-core kernels read masks, against the CPU oracle.  Full masks: rows at every alignment (odd lengths, a
view that starts inside a row), ragged last tiles, one and several key tiles.  Boolean masks that are the same for all heads
and rows: padding of every kind of length, with and without holes, and a sequence with no key at all.
Tolerance: that of test_mask_gpu.py."""
import numpy as np
import pytest
import torch

from gpu_util import TOL_ABS_16BIT, make, to_np

pytestmark = pytest.mark.gpu

NEG = np.float32(-np.inf)
TYPES = {"bf16": torch.bfloat16, "f16": torch.float16}


def _run(oracle, dt, D, B, Hq, Hkv, L, S, mask, bias, keep=None):
    from tinytorch_b200 import op
    q, qn = make((B, Hq, L, D), TYPES[dt], 51)
    k, kn = make((B, Hkv, S, D), TYPES[dt], 52)
    v, vn = make((B, Hkv, S, D), TYPES[dt], 53)
    do, don = make((B, Hq, L, D), TYPES[dt], 54)
    o, lse = op.sdpAttentionFwd(q, k, v, attnMask=mask)
    got = [o] + list(op.sdpAttentionBwd(do, q, k, v, o, lse, attnMask=mask))
    torch.cuda.synchronize()
    keep = list(range(B)) if keep is None else keep  # the sequences that have keys
    bias = np.broadcast_to(bias, (B,) + bias.shape[1:])[keep]
    want_o, want_l = oracle.fwd(qn[keep], kn[keep], vn[keep], bias=bias)
    want = [want_o] + list(oracle.bwd(qn[keep], kn[keep], vn[keep], don[keep], bias=bias))
    assert np.abs(to_np(lse)[keep] - want_l).max() <= 2e-2
    for g, w in zip(got, want):
        assert np.abs(to_np(g)[keep] - w).max() <= TOL_ABS_16BIT * max(1.0, np.abs(w).max())
    for b in set(range(B)) - set(keep):
        assert torch.isinf(lse[b]).all() and all((g[b] == 0).all() for g in got)


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["bool", "same", "f32"])
@pytest.mark.parametrize("L,S,skip", [(129, 131, 0), (257, 515, 0), (40, 390, 0), (300, 261, 3), (1, 130, 1), (128, 256, 0)])
def test_full_masks_at_every_alignment(oracle, dt, D, kind, L, S, skip):
    B, Hq, Hkv = 1, 4, 2
    rng = np.random.default_rng(55)
    if kind == "bool":
        m = rng.random((1, Hq, L, S + skip)) < 0.7
        m[..., skip] = True
        mask = torch.from_numpy(m).cuda()
        bias = np.where(m, np.float32(0), NEG)
    else:
        mask = torch.from_numpy(rng.standard_normal((1, Hq, L, S + skip)).astype(np.float32))
        mask = (mask if kind == "f32" else mask.to(TYPES[dt])).cuda()
        bias = mask.float().cpu().numpy()
    _run(oracle, dt, D, B, Hq, Hkv, L, S, mask[..., skip:], np.ascontiguousarray(bias[..., skip:]))


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("holes", [False, True])
@pytest.mark.parametrize("L,S", [(130, 389), (260, 128)])
def test_padding_masks(oracle, dt, D, holes, L, S):
    lens = (S, 0, 1, S - 1, 127, 128)
    m = np.arange(S)[None, :] < np.array(lens)[:, None]
    if holes:
        m[3, 0] = m[3, 5] = m[4, 126] = m[5, 60:100] = False
    mask = torch.from_numpy(m[:, None, None, :]).cuda()
    bias = np.broadcast_to(np.where(m, np.float32(0), NEG)[:, None, None, :], (len(lens), 1, L, S))
    _run(oracle, dt, D, len(lens), 2, 1, L, S, mask, bias, keep=[b for b in range(len(lens)) if m[b].any()])


@pytest.mark.parametrize("kind", ["bool", "add"])
def test_masks_that_start_at_any_byte(oracle, kind):
    """Views of one mask that start at every byte (bool) or element (16 bit) of a 16-byte piece, with rows and keys beyond the
    last tile: copies of nothing, too, come from an aligned address."""
    L, S = 33, 130
    rng = np.random.default_rng(56)
    for skip in range(16 if kind == "bool" else 8):
        if kind == "bool":
            m = rng.random((1, 2, L, S + skip)) < 0.7
            m[..., skip] = True
            mask, bias = torch.from_numpy(m).cuda(), np.where(m, np.float32(0), NEG)
        else:
            mask = torch.from_numpy(rng.standard_normal((1, 2, L, S + skip)).astype(np.float32)).bfloat16().cuda()
            bias = mask.float().cpu().numpy()
        _run(oracle, "bf16", 64, 1, 2, 2, L, S, mask[..., skip:], np.ascontiguousarray(bias[..., skip:]))
