"""GPU: the projection kernel's tile shapes between 256 x 256 pairs and the divided contraction: single CTAs with 128 x 64..256 tiles
and pairs with 256 x 192, at sizes where a row tile, a column tile, a block of 32 or 64 columns or the contraction is ragged.

Reference and bound as in test_linear_paths_gpu.py."""
import pytest
import torch

from test_linear_paths_gpu import _check

pytestmark = pytest.mark.gpu


# (columns of the tile that the product takes)
SHAPES = [(129, 1024, 3016),    # 64, the second row tile holds one row
          (300, 1000, 3000),    # 64, K tail
          (512, 1032, 4096),    # 128
          (1455, 520, 3624),    # 160: the last block of 32 columns is partly beyond N
          (3000, 1024, 1032),   # 192
          (349, 2096, 9704),    # 224
          (786, 3304, 3304),    # pairs, 192
          (1030, 72, 4104),     # one block and a part of the contraction
          (2049, 64, 1160)]


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
