"""GPU: the projection kernel's tile shapes between 256 x 256 pairs and the divided contraction: single CTAs with 128 x 64..256 tiles
and pairs with 256 x 192.  Through the public functions at sizes where a row tile, a column tile, a block of 32 or 64 columns or the
contraction is ragged; every shape with every way its operands can be stored, asked for by itself; and that the planner takes each.

Reference and bound as in test_linear_paths_gpu.py."""
import ctypes as C
import math
import random

import pytest
import torch

from test_linear_paths_gpu import _check

pytestmark = pytest.mark.gpu


# What forward, dX and dW take on a chip with 148 SMs: the columns of a tile of single CTAs, p: of pairs, 0: the divided contraction.
SHAPES = [(129, 1024, 3016),    # 0, 0, 192
          (300, 1000, 3000),    # 64 (K tail), 0, 192
          (512, 1032, 4096),    # 128, 0, 0
          (1455, 520, 3624),    # p192 (two models 0.05 % apart: 160), 0, 128
          (3000, 1024, 1032),   # 192, 192, 0
          (349, 2096, 9704),    # 224, 0, p256
          (786, 3304, 3304),    # p192, p256, p256
          (1030, 72, 4104),     # 160 (one block and a part of the contraction), 0, 0
          (2049, 64, 1160),     # 0, 0, 0
          (1269, 64, 1000),     # 96, 0, 0
          (1689, 72, 2480),     # 256, 0, 0
          (696, 72, 128),       # 0, 64, 0
          (912, 1400, 136),     # 0, 128, 0
          (1207, 2976, 136),    # 0, 256, 0
          (167, 200, 9808)]     # 0, 0, 256


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N", SHAPES)
def test_tile_shapes(dtype, M, K, N):
    from tinytorch_b200 import fused
    g = torch.Generator("cuda").manual_seed(M + K + N)
    x, w, b, dy = (torch.randn(s, device="cuda", generator=g).to(dtype) for s in ((M, K), (N, K), (N,), (M, N)))
    for t in (x, w, b):
        t.requires_grad_()
    y = fused.linear(x, w, b)
    dx, dw, db = torch.autograd.grad(y, (x, w, b), dy, retain_graph=True)
    xd, wd, bd, dyd = (t.detach().double() for t in (x, w, b, dy))
    _check(y, xd, wd.t(), bd, dtype)
    _check(dx, dyd, wd, None, dtype)
    _check(dw, dyd.t(), xd, None, dtype)
    _check(db[:, None], dyd.t(), torch.ones(M, 1, device="cuda", dtype=torch.float64), None, dtype)
    # the same bits again, also where the tiles of an SM follow one another
    for _ in range(5):
        assert torch.equal(fused.linear(x, w, b), y)
        assert all(torch.equal(p, q) for p, q in zip(torch.autograd.grad(y, (x, w), dy, retain_graph=True), (dx, dw)))


def _params(dtype, M, N, K, x_t, w_t):
    from tinytorch_b200 import _capi
    f = _capi.lib().tt_linear_selftest
    f.argtypes, f.restype = [C.POINTER(_capi.LinearParams), C.c_int32, C.POINTER(C.c_int32)], C.c_int
    p = _capi.LinearParams()
    p.struct_size, p.dtype = C.sizeof(p), _capi.BF16 if dtype == torch.bfloat16 else _capi.F16
    p.M, p.N, p.K, p.x_t, p.w_t = M, N, K, x_t, w_t
    p.device, p.stream = torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream
    return f, p


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("x_t,w_t", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("shape", [64, 96, 128, 160, 192, 224, 256, -192])
def test_every_shape_with_every_operand_layout(dtype, shape, x_t, w_t):
    """x as [M, K] or [K, M], w as [N, K] or [K, N] (blocks of 64 columns, single CTAs only)."""
    if w_t and (shape < 0 or shape % 64):
        pytest.skip("there is no such tile")
    from tinytorch_b200 import _capi
    gen = torch.Generator("cuda").manual_seed(abs(shape) + 2 * x_t + w_t)
    for M, K, N in [(200, 136, 520),     # a tile or two, the last of each kind ragged, a K tail
                    (8, 8, 8),           # one block of everything
                    (264, 1096, 264),    # the ring goes round
                    (2408, 72, 2056),    # more tiles than SMs or pairs of them: both accumulators, several times
                    (128, 64, 12288)]:
        x, w, b = (torch.randn(s, device="cuda", generator=gen).to(dtype) for s in ((M, K), (N, K), (N,)))
        xs, ws = x.t().contiguous() if x_t else x, w.t().contiguous() if w_t else w
        y, status = torch.full((M, N), float("nan"), dtype=dtype, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        f, p = _params(dtype, M, N, K, x_t, w_t)
        p.x, p.w, p.bias, p.y, p.status = xs.data_ptr(), ws.data_ptr(), b.data_ptr(), y.data_ptr(), status.data_ptr()
        _capi.check(f(C.byref(p), shape, None))
        _check(y, x.double(), w.double().t(), b.double(), dtype)
        assert int(status) == 0


def test_every_shape_is_planned():
    """Each shape is what the planner takes for some ordinary size (nothing is launched)."""
    buf = torch.zeros(8, device="cuda")
    rng, seen = random.Random(4), {}
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    for _ in range(4000):
        M, K, N = log(129, 6000), 8 * log(8, 600), 8 * log(16, 1300)
        for kind, size, x_t, w_t in (("y", (M, N, K), 0, 0), ("dx", (M, K, N), 0, 1), ("dw", (N, K, M), 1, 1)):
            f, p = _params(torch.bfloat16, *size, x_t, w_t)
            p.x = p.w = p.y = buf.data_ptr()
            planned = C.c_int32(1)
            assert f(C.byref(p), 0, C.byref(planned)) == 0
            seen.setdefault(kind, set()).add(planned.value)
    assert seen["y"] == {0, 64, 96, 128, 160, 192, 224, 256, -192, -256}
    assert seen["dx"] == seen["dw"] == {0, 64, 128, 192, 256, -256}
