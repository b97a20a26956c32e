"""CPU: arguments that do not belong together are refused before anything is launched.

The tensors are fake CUDA tensors (no memory behind them), so a call that is let through fails on the missing driver, with
another error than the ValueError asked for here."""
import os

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from conftest import ROOT
from tinytorch_b200 import fused, function, op


@pytest.fixture(autouse=True)
def fake():
    if not os.path.exists(os.path.join(ROOT, "tinytorch_b200", "lib", "_native.so")):
        from tinytorch_b200.build import build, build_native
        build()
        build_native()
    with FakeTensorMode():
        yield


def t(*shape, dtype=torch.bfloat16, device="cuda"):
    return torch.empty(shape, dtype=dtype, device=device)


Q, KV, CACHE, NEW = (3, 8, 40, 64), (3, 4, 50, 64), (3, 4, 128, 64), (3, 4, 1, 64)
SMALLER = [dict(k=(2, 4, 50, 64)), dict(v=(2, 4, 50, 64)), dict(v=(3, 2, 50, 64)), dict(v=(3, 4, 49, 64)), dict(v=(3, 4, 50, 32)),
           dict(k=(3, 4, 50, 32))]


@pytest.mark.parametrize("wrong", SMALLER)
def test_keys_and_values_smaller_than_what_is_read(wrong):
    args = [t(*Q), t(*wrong.get("k", KV)), t(*wrong.get("v", KV))]
    for call in (op.sdpAttentionFwd, function.sdpAttention):
        with pytest.raises(ValueError):
            call(*args)


@pytest.mark.parametrize("wrong", [dict(k=(4, 4, 50, 64)), dict(v=(4, 4, 50, 64)), dict(v=(3, 5, 50, 64)), dict(v=(3, 4, 51, 64))] + SMALLER)
def test_gradients_of_keys_and_values_of_other_shapes(wrong):
    """Larger ones too: the kernels would leave a part of the gradient unwritten."""
    q, k, v = (x.requires_grad_() for x in (t(*Q), t(*wrong.get("k", KV)), t(*wrong.get("v", KV))))
    with pytest.raises(ValueError):
        function.sdpAttention(q, k, v)
    with pytest.raises(ValueError):
        op.sdpAttentionBwd(t(*Q), q.detach(), k.detach(), v.detach(), t(*Q), t(*Q[:3], dtype=torch.float32))


@pytest.mark.parametrize("name,x", [
    ("dO", dict(shape=(3, 8, 39, 64))), ("dO", dict(shape=Q, dtype=torch.float16)), ("o", dict(shape=(3, 7, 40, 64))),
    ("o", dict(shape=Q, dtype=torch.float32)), ("lse", dict(shape=(3, 8, 39), dtype=torch.float32)),
    ("lse", dict(shape=(3, 8, 40), dtype=torch.bfloat16)), ("lse", dict(shape=(3, 8, 40), dtype=torch.float32, device="cpu")),
])
def test_backward_operands(name, x):
    args = dict(dO=t(*Q), q=t(*Q), k=t(*KV), v=t(*KV), o=t(*Q), lse=t(*Q[:3], dtype=torch.float32))
    shape = x.pop("shape")
    args[name] = t(*shape, **x)
    with pytest.raises(ValueError):
        op.sdpAttentionBwd(**args)


@pytest.mark.parametrize("wrong", [
    dict(k=((2, 4, 128, 64), torch.bfloat16)), dict(v=((3, 4, 127, 64), torch.bfloat16)), dict(v=((3, 3, 128, 64), torch.bfloat16)),
    dict(k=(CACHE, torch.float16)), dict(v=(CACHE, torch.float32)), dict(new=(NEW, torch.float16)),
])
def test_decode_caches(wrong):
    q = t(3, 8, 1, 64)
    k, v, new = (t(*wrong.get(n, (s, torch.bfloat16))[0], dtype=wrong.get(n, (s, torch.bfloat16))[1])
                 for n, s in (("k", CACHE), ("v", CACHE), ("new", NEW)))
    lens = t(3, dtype=torch.int32)
    if "new" not in wrong:
        with pytest.raises(ValueError):
            op.sdpAttentionDecode(q, k, v, lens)
    with pytest.raises(ValueError):
        op.sdpAttentionDecodeAppend(q, new, t(*NEW), k, v, lens)


@pytest.mark.parametrize("lens", [dict(dtype=torch.int64), dict(n=2), dict(dtype=torch.float32), dict(step=2), dict(device="cpu")])
def test_lengths(lens):
    """An int64 tensor would be read as pairs of int32 words, a strided or short one beyond its end."""
    n, step = lens.get("n", 3), lens.get("step", 1)
    x = t(n * step, dtype=lens.get("dtype", torch.int32), device=lens.get("device", "cuda"))[::step]
    q1, k, v, new = t(3, 8, 1, 64), t(*CACHE), t(*CACHE), t(*NEW)
    for call in (lambda: op.sdpAttentionFwd(t(*Q), k, v, kvLens=x), lambda: function.sdpAttention(t(*Q), k, v, kvLens=x),
                 lambda: op.sdpAttentionBwd(t(*Q), t(*Q), k, v, t(*Q), t(*Q[:3], dtype=torch.float32), kvLens=x),
                 lambda: op.sdpAttentionDecode(q1, k, v, x), lambda: op.sdpAttentionDecodeAppend(q1, new, new, k, v, x)):
        with pytest.raises(ValueError):
            call()


def test_status_word_workspace_and_rotary_tables():
    q1, k, v, new, lens = t(3, 8, 1, 64), t(*CACHE), t(*CACHE), t(*NEW), t(3, dtype=torch.int32)
    for status in (t(1, dtype=torch.int64), t(0, dtype=torch.int32), t(1, dtype=torch.int32, device="cpu")):
        with pytest.raises(ValueError):
            op.sdpAttentionFwd(t(*Q), k, v, status=status)
        with pytest.raises(ValueError):
            op.sdpAttentionDecodeAppend(q1, new, new, k, v, lens, status=status)
    for ws in (t(4096, dtype=torch.uint8, device="cpu"), t(64, 64, dtype=torch.uint8)[:, :32]):
        with pytest.raises(ValueError):
            op.sdpAttentionDecode(q1, k, v, lens, workspace=ws)
    table = t(128, 32, dtype=torch.float32)
    for cos, sin in ((table, t(128, 32, dtype=torch.float64)), (table, t(128, 32, dtype=torch.float32, device="cpu")),
                     (t(128, 32, dtype=torch.float32, device="cpu"), table)):
        with pytest.raises(ValueError):
            op.sdpAttentionDecodeAppend(q1, new, new, k, v, lens, cos, sin)


def test_projection_operands():
    x, w = t(6, 64), t(16, 64)
    for call in (fused.linear, fused._linear_raw):
        with pytest.raises(ValueError):
            call(x, w, t(16, device="cpu"))
        with pytest.raises(AssertionError):
            call(x, w, t(8))
    for a, b in ((t(2, 6, 64), w), (x, t(16, 32)), (x, t(16, 64, dtype=torch.float16)), (t(64, 6).t(), w), (x, t(16, 64, device="cpu"))):
        with pytest.raises(ValueError):
            fused._linear_raw(a, b, None)
    with pytest.raises(ValueError):
        fused._linear_raw(x, w, None, t(1, dtype=torch.int64))


def test_norm_operands_on_another_device():
    with pytest.raises(ValueError):
        fused.fusedAddRmsNorm(t(4, 64), t(4, 64), t(64, device="cuda:1"), 1e-5)
