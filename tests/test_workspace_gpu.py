"""GPU: a scratch buffer sized for the largest batch serves every smaller one.

Small batches are divided further than large ones (more shares, more partial results); where a caller's buffer does not
hold them, a call takes the large batch's division instead of refusing.  Reference: the same call with scratch memory of
its own, which is compared with the oracle elsewhere; another division changes the order of fp32 sums and, in the
16-bit types, at most a rounding of the result (2 ulp of its magnitude)."""
import ctypes as C

import pytest
import torch

from gpu_util import ULP, make

pytestmark = pytest.mark.gpu


def _close(got, want, dtype):
    eps = 1e-5 if dtype == torch.float32 else 2 * ULP[dtype]
    assert bool(((got.double() - want.double()).abs() <= eps * want.abs().double().clamp_min(float(want.abs().mean()))).all())


# (dtype, Hq, Hkv, D, capacity, largest batch)
DECODE = [(torch.bfloat16, 8, 8, 128, 4096, 3), (torch.float32, 4, 2, 64, 3000, 16), (torch.bfloat16, 16, 4, 128, 3000, 27),
          (torch.float16, 8, 2, 64, 5000, 60)]


@pytest.mark.parametrize("dt,Hq,Hkv,D,cap,most", DECODE)
def test_decode_buffer_of_the_largest_batch(dt, Hq, Hkv, D, cap, most):
    from tinytorch_b200 import _capi, op
    need = [op.workspaceBytes(_capi.KIND_DECODE, dt, b, Hq, Hkv, 1, cap, D) for b in range(1, most + 1)]
    assert max(need) > need[-1]  # (what makes this a test: some smaller batch would like more)
    q, k, v = (make(s, dt, i)[0] for i, s in ((81, (most, Hq, 1, D)), (82, (most, Hkv, cap, D)), (83, (most, Hkv, cap, D))))
    lens = torch.arange(most, device="cuda", dtype=torch.int32) * (cap // most) + cap // most
    ws = torch.empty(need[-1] + 64, dtype=torch.uint8, device="cuda").fill_(171)
    for b in range(1, most + 1):
        o, _ = op.sdpAttentionDecode(q[:b], k[:b], v[:b], lens[:b], workspace=ws[:need[-1]])
        _close(o, op.sdpAttentionDecode(q[:b], k[:b], v[:b], lens[:b])[0], dt)
    assert bool((ws[need[-1]:] == 171).all())


def _append(q, kn, vn, kc, vc, lens, ws):
    from tinytorch_b200 import _capi
    B, Hq, _, D = q.shape
    o, new = torch.empty_like(q), torch.empty_like(lens)
    p = _capi.DecodeAppendParams()
    p.struct_size, p.dtype = C.sizeof(p), {torch.bfloat16: _capi.BF16, torch.float16: _capi.F16, torch.float32: _capi.F32}[q.dtype]
    p.B, p.Hq, p.Hkv, p.capacity, p.D = B, Hq, kc.shape[1], kc.shape[2], D
    for n, t in (("q", q), ("k_new", kn), ("v_new", vn), ("k_cache", kc), ("v_cache", vc), ("o", o)):
        setattr(p, n, t.data_ptr())
    for n, t in (("q", q), ("k_new", kn), ("v_new", vn), ("k", kc), ("v", vc), ("o", o)):
        setattr(p, n + "_strides", _capi.Strides(t.stride(0), t.stride(1), t.stride(2)))
    p.scale, p.kv_lens, p.new_lens = D ** -0.5, lens.data_ptr(), new.data_ptr()
    p.device, p.stream = torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    _capi.check(_capi.lib().tt_attn_decode_append(C.byref(p)))
    return o, new


@pytest.mark.parametrize("dt,Hq,Hkv,D,cap,most", DECODE)
def test_decode_append_buffer_of_the_largest_batch(dt, Hq, Hkv, D, cap, most):
    from tinytorch_b200 import _capi, op
    need = op.workspaceBytes(_capi.KIND_DECODE_APPEND, dt, most, Hq, Hkv, 1, cap, D)
    q, kc, vc, kn, vn = (make(s, dt, 84 + i)[0] for i, s in enumerate(
        ((most, Hq, 1, D), (most, Hkv, cap, D), (most, Hkv, cap, D), (most, Hkv, 1, D), (most, Hkv, 1, D))))
    lens = torch.arange(most, device="cuda", dtype=torch.int32) * (cap // most) + 1
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    for b in sorted({1, 2, most // 2, most - 1, most}):
        o, new = _append(q[:b], kn[:b], vn[:b], kc[:b], vc[:b], lens[:b], ws)
        want, _, wn = op.sdpAttentionDecodeAppend(q[:b], kn[:b], vn[:b], kc[:b], vc[:b], lens[:b])
        _close(o, want, dt)
        assert torch.equal(new, wn)


def test_static_scratch_takes_every_batch_below_its_largest():
    """256 query heads on one kv head: a batch of three would be divided into more than the fixed array holds."""
    from tinytorch_b200 import _capi, op
    Hq, cap, D = 256, 4096, 128
    for B in (1, 3, 4, 5):
        q, k, v = (make(s, torch.float32, 91 + i)[0] for i, s in enumerate(((B, Hq, 1, D), (B, 1, cap, D), (B, 1, cap, D))))
        got = torch.empty_like(q)
        p = _capi.DecodeParams()
        p.struct_size, p.dtype = C.sizeof(p), _capi.F32
        p.B, p.Hq, p.Hkv, p.capacity, p.D = B, Hq, 1, cap, D
        p.q, p.k, p.v, p.o = q.data_ptr(), k.data_ptr(), v.data_ptr(), got.data_ptr()
        p.scale, p.device, p.stream = D ** -0.5, torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
        _capi.check(_capi.lib().tt_attn_decode_static(C.byref(p)))
        _close(got, op.sdpAttentionDecode(q, k, v)[0], torch.float32)


def _prefill(name, cls, q, k, v, o, ws, causal=0, mask=None, **ptrs):
    """tt_attn_fwd / tt_attn_bwd with a scratch buffer of the caller's."""
    from tinytorch_b200 import _capi
    p = cls()
    p.struct_size, p.dtype = C.sizeof(p), {torch.bfloat16: _capi.BF16, torch.float16: _capi.F16}[q.dtype]
    p.B, p.Hq, p.Hkv, p.Lq, p.Skv, p.D = q.shape[0], q.shape[1], k.shape[1], q.shape[2], k.shape[2], q.shape[3]
    p.q, p.k, p.v, p.o = (t.data_ptr() for t in (q, k, v, o))
    for n, t in ptrs.items():
        setattr(p, n, t.data_ptr())
    p.is_causal, p.scale = causal, q.shape[3] ** -0.5
    p.device, p.stream = torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    if mask is not None:  # [B, 1, 1, S]
        p.mask, p.mask_kind = mask.data_ptr(), _capi.MASK_BOOL
        p.mask_strides[0] = mask.stride(0)
    _capi.check(getattr(_capi.lib(), name)(C.byref(p)))


def test_backward_buffer_of_the_largest_batch():
    from tinytorch_b200 import _capi, op
    H, L, D, most, dt = 8, 2048, 128, 2, torch.bfloat16
    need = [op.workspaceBytes(_capi.KIND_BWD, dt, b, H, H, L, L, D) for b in range(1, most + 1)]
    assert need[0] > need[1]
    q, k, v, do = (make((most, H, L, D), dt, 95 + i)[0] for i in range(4))
    ws = torch.empty(need[-1] + 64, dtype=torch.uint8, device="cuda").fill_(171)
    for b in (1, 2):
        o, lse = op.sdpAttentionFwd(q[:b], k[:b], v[:b], isCausal=True)
        grads = [torch.empty_like(q[:b]) for _ in range(3)]
        _prefill("tt_attn_bwd", _capi.BwdParams, q[:b], k[:b], v[:b], o, ws[:need[-1]], causal=1, lse=lse, d_o=do[:b],
                 dq=grads[0], dk=grads[1], dv=grads[2])
        for got, want in zip(grads, op.sdpAttentionBwd(do[:b], q[:b], k[:b], v[:b], o, lse, isCausal=True)):
            _close(got, want, dt)
    assert bool((ws[need[-1]:] == 171).all())


def test_work_counter_alone_is_enough_for_a_large_batch():
    """256 bytes (and the backward's accumulators), at a batch whose mask lengths take more: with a padding mask and without."""
    from tinytorch_b200 import _capi, op
    B, H, L, D, dt = 40, 2, 130, 64, torch.float16
    q, k, v, do = (make((B, H, L, D), dt, 61 + i)[0] for i in range(4))
    n = torch.arange(B, device="cuda") * 3 + 5
    mask = (torch.arange(L, device="cuda")[None] < n[:, None])[:, None, None]
    lse = torch.empty((B, H, L), device="cuda")
    base = sum((B * H * L * 4 * x + 255) // 256 * 256 for x in (1, D))
    for m in (None, mask):
        o, grads = torch.empty_like(q), [torch.empty_like(q) for _ in range(3)]
        _prefill("tt_attn_fwd", _capi.FwdParams, q, k, v, o, torch.empty(256, dtype=torch.uint8, device="cuda"), mask=m, lse=lse)
        want, wl = op.sdpAttentionFwd(q, k, v, attnMask=m)
        _close(o, want, dt)
        assert float((lse - wl).abs().max()) <= 1e-4
        _prefill("tt_attn_bwd", _capi.BwdParams, q, k, v, want, torch.empty(base + 256, dtype=torch.uint8, device="cuda"), mask=m,
                 lse=wl, d_o=do, dq=grads[0], dk=grads[1], dv=grads[2])
        for got, w in zip(grads, op.sdpAttentionBwd(do, q, k, v, want, wl, attnMask=m)):
            _close(got, w, dt)
