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
