"""GPU: the projection kernels and their gradient products at the edges of their tiles and dispatch rules.

linear_split.cu takes outputs with few tiles (any M up to 128, and where it is expected to be the fastest), linear_tc.cu those with two
rounds of 256 x 256 tiles, linear_tile.cu (test_linear_tiles_gpu.py) what lies between; all read operands stored with the
contraction slow or fast.  Reference: the
same sums in fp64.  Bound per element: half a unit in the last place of the tensor dtype for the one rounding, plus
fp32 accumulation in any order: (terms + 2) * 2^-24 * sum of |products|.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

HALF_ULP = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # relative to the value's binade, from below
TINY = {torch.bfloat16: 1e-30, torch.float16: 2.0 ** -25}          # spacing of fp16 subnormals


def _check(got, a, b, bias, dtype):  # got ~ a b (+ bias), a [m, k], b [k, n] in fp64
    want, terms, size = a @ b, a.shape[1] + (bias is not None), a.abs() @ b.abs()
    if bias is not None:
        want, size = want + bias, size + bias.abs()
    bound = HALF_ULP[dtype] * want.abs() * 1.01 + (terms + 2) * 2.0 ** -24 * size + TINY[dtype]
    err = (got.double() - want).abs()
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N", [
    (1, 8, 8), (16, 64, 128), (17, 72, 136), (3, 4096, 264),                 # one tile of x; clusters of 1 .. 8
    (128, 520, 1024), (129, 1032, 4096), (255, 64, 4096), (300, 1024, 3000),  # several tiles of x, K tails; dW: tiles made to measure
    (511, 192, 264), (257, 4160, 512),
    (1100, 72, 9736), (2050, 456, 4872), (4000, 64, 2568),                    # forward: the persistent pairs, ragged on every side
])
def test_projection_and_gradients_at_tile_edges(dtype, M, K, N):
    from tinytorch_b200 import fused
    g = torch.Generator("cuda").manual_seed(M + 3 * K + 7 * N)
    x, w, b, dy = (torch.randn(s, device="cuda", generator=g).to(dtype) for s in ((M, K), (N, K), (N,), (M, N)))
    for t in (x, w, b):
        t.requires_grad_()
    y = fused.linear(x, w, b)
    dx, dw, db = torch.autograd.grad(y, (x, w, b), dy)
    xd, wd, bd, dyd = (t.detach().double() for t in (x, w, b, dy))
    _check(y, xd, wd.t(), bd, dtype)
    _check(dx, dyd, wd, None, dtype)
    _check(dw, dyd.t(), xd, None, dtype)
    _check(db[:, None], dyd.t(), torch.ones(M, 1, device="cuda", dtype=torch.float64), None, dtype)


def test_strided_rows_and_repeat():
    """Row-strided operands, the same answer twice (the sums over a cluster are in rank order)."""
    from tinytorch_b200 import fused
    g = torch.Generator("cuda").manual_seed(5)
    big = torch.randn(40, 2048 + 64, device="cuda", generator=g).bfloat16()
    w = torch.randn(1024, 2048 + 8, device="cuda", generator=g).bfloat16()[:, :2048]
    x = big[::2, 64:]
    y1, y2 = fused.linear(x, w), fused.linear(x, w)
    assert torch.equal(y1, y2)
    _check(y1, x.double(), w.double().t(), None, torch.bfloat16)


@pytest.mark.parametrize("M,N", [
    (2309, 4608),   # the lower half of the last row of tiles lies wholly beyond M
    (2560, 4616),   # of the last column of tiles only the first block of 64 columns exists
    (2560, 4744),   # ... the first two and a part of the third
    (2309, 4744),
])
def test_blocks_beyond_the_edge_between_full_tiles(M, N):
    """The persistent pairs with tiles of which some blocks store nothing, followed by tiles of which all do, and a
    contraction so short that the next tile is complete before a store has left shared memory: every element, and the
    same bits each time."""
    from tinytorch_b200 import fused
    g = torch.Generator("cuda").manual_seed(M + N)
    for K in (8, 64):
        x, w = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((M, K), (N, K)))
        y = fused.linear(x, w)
        _check(y, x.double(), w.double().t(), None, torch.bfloat16)
        for _ in range(20):
            assert torch.equal(fused.linear(x, w), y)


@pytest.mark.parametrize("first,width", [(3, 264), (0, 267), (8, 272), (1, 272)])
def test_gradients_that_are_parts_of_larger_ones(first, width):
    """dY at any offset and row stride, for every choice of gradients."""
    from tinytorch_b200 import fused
    g = torch.Generator("cuda").manual_seed(9)
    M, K, N = 33, 72, 256
    x, w, b = (torch.randn(s, device="cuda", generator=g).bfloat16().requires_grad_() for s in ((M, K), (N, K), (N,)))
    dy = torch.randn(M, width, device="cuda", generator=g).bfloat16()[:, first:first + N]
    y = fused.linear(x, w, b)
    want = torch.autograd.grad(y, (x, w, b), dy.contiguous(), retain_graph=True)
    for pick in ((0, 1, 2), (0,), (1,), (2,), (1, 2)):
        got = torch.autograd.grad(y, [(x, w, b)[i] for i in pick], dy, retain_graph=True)
        assert all(torch.equal(a, want[i]) for a, i in zip(got, pick))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N", [(1, 8), (2, 128), (63, 136), (129, 256), (4097, 1000)])
def test_bias_gradient_alone(dtype, M, N):
    """The column sums without a product beside them: the same sums as with one, every row counted."""
    from tinytorch_b200 import fused
    g = torch.Generator("cuda").manual_seed(M + N)
    x, w = (torch.randn(s, device="cuda", generator=g).to(dtype) for s in ((M, 64), (N, 64)))
    b = torch.randn(N, device="cuda", generator=g).to(dtype).requires_grad_()
    dy = torch.randn(M, N, device="cuda", generator=g).to(dtype)
    db, = torch.autograd.grad(fused.linear(x, w, b), b, dy)
    _check(db[:, None], dy.double().t(), torch.ones(M, 1, device="cuda", dtype=torch.float64), None, dtype)
    w.requires_grad_()
    assert torch.equal(db, torch.autograd.grad(fused.linear(x, w, b), (w, b), dy)[1])


def test_gradients_of_no_rows():
    from tinytorch_b200 import fused
    x, w, b = (torch.randn(s, device="cuda").bfloat16().requires_grad_() for s in ((3, 0, 64), (40, 64), (40,)))
    for pick in ((x, w, b), (b,)):
        y = fused.linear(x, w, b)
        assert y.shape == (3, 0, 40)
        for t, d in zip(pick, torch.autograd.grad(y, pick, torch.empty_like(y))):
            assert d.shape == t.shape and not bool(d.any())
