"""GPU: the differentiable operators in torch's autograd: traces, forward mode, functorch, and the native nodes' corners."""
import warnings

import pytest
import torch
import torch.autograd.forward_ad as fwad

from gpu_util import make

pytestmark = pytest.mark.gpu


def _attention(seed=0, dtype=torch.bfloat16):
    return [make((2, 4, 130, 64), dtype, 300 + seed + i)[0] for i in range(3)]


def _projection(seed=0):
    return [make(s, torch.bfloat16, 310 + seed + i)[0] for i, s in enumerate(((48, 64), (40, 64), (40,)))]


def _ops():
    from tinytorch_b200 import function, fused
    return [(lambda q, k, v: function.sdpAttention(q, k, v, isCausal=True), _attention), (fused.linear, _projection)]


@pytest.mark.parametrize("which", [0, 1])
def test_a_trace_records_the_operator(which):
    f, inputs = _ops()[which]
    a, b = inputs(0), inputs(40)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        traced = torch.jit.trace(lambda *x: f(*x) * 2, a, check_trace=False)
    assert torch.equal(traced(*b), f(*b) * 2) and not torch.equal(traced(*b), traced(*a))


@pytest.mark.parametrize("which", [0, 1])
def test_forward_mode_is_refused(which):
    """Not taken for a call without a tangent."""
    f, inputs = _ops()[which]
    x = inputs()
    with fwad.dual_level():
        for i in range(3):
            d = [fwad.make_dual(t, torch.ones_like(t)) if i == j else t for j, t in enumerate(x)]
            with pytest.raises((NotImplementedError, RuntimeError)):
                f(*d)
    f(*x)


@pytest.mark.parametrize("which", [0, 1])
def test_functorch_is_refused(which):
    f, inputs = _ops()[which]
    x = inputs()
    for call in (lambda: torch.func.grad(lambda t: f(t, *x[1:]).float().sum())(x[0]),
                 lambda: torch.vmap(lambda t: f(t, *x[1:]))(torch.stack([x[0], x[0]]))):
        with pytest.raises(RuntimeError, match="autograd.Function"):
            call()


@pytest.mark.parametrize("which", [0, 1])
def test_python_function_and_native_node_agree(which):
    from tinytorch_b200 import function, fused
    f, inputs = _ops()[which]
    x = [t.requires_grad_() for t in inputs()]
    y = f(*x)
    z = fused.FuncLinear.apply(*x) if which else function.FuncSDPAttention.apply(*x, True, None, 64 ** -0.5)
    g = torch.randn_like(y)
    assert torch.equal(y, z)
    # (two key tiles: dQ is a sum of two shares, whose order does not matter)
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, x, g), torch.autograd.grad(z, x, g)))


def test_saved_tensors_pass_through_hooks():
    """q, k, v, O and the row statistics: what a hook packs (here: to host memory) is what the backward pass uses."""
    f, inputs = _ops()[0]
    x = [t.requires_grad_() for t in inputs()]
    g = torch.randn_like(x[0])
    want = torch.autograd.grad(f(*x), x, g)
    packed = []

    def pack(t):
        packed.append((t.dtype, tuple(t.shape)))
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        y = f(*x)
    assert len(packed) == 5 and (torch.float32, (2, 4, 130)) in packed
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, x, g), want))


@pytest.mark.parametrize("kind", ["bool", "add"])
def test_mask_and_lengths_pointed_elsewhere_before_the_backward(kind):
    from tinytorch_b200 import function
    x = [t.requires_grad_() for t in _attention()]
    g = torch.randn_like(x[0])
    mask = torch.rand(130, 130, device="cuda").lt(0.7) if kind == "bool" else torch.randn(130, 130, device="cuda").bfloat16()
    lens = torch.tensor([130, 77], dtype=torch.int32, device="cuda")
    call = lambda m, n: function.sdpAttention(*x, attnMask=m, kvLens=n)
    want = torch.autograd.grad(call(mask.clone(), lens.clone()), x, g)
    y = call(mask, lens)
    mask.set_(torch.empty(1, dtype=mask.dtype, device="cuda"))
    lens.set_(torch.empty(2, dtype=torch.int32, device="cuda").fill_(1))
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, x, g), want))


@pytest.mark.parametrize("which", [0, 1])
def test_no_gradient_from_what_follows_is_a_gradient_of_zeros(which):
    class Drop(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.clone()

        @staticmethod
        def backward(ctx, grad):
            return None

    f, inputs = _ops()[which]
    x = [t.requires_grad_() for t in inputs()]
    Drop.apply(f(*x)).float().sum().backward()
    for t in x:
        assert t.grad is not None and not bool(t.grad.any())


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("pick", [(2,), (1, 2), (0, 1, 2)])
def test_the_bias_gradient_can_be_differentiated_again(native, pick):
    from tinytorch_b200 import fused
    x = [t.requires_grad_() for t in _projection()]
    y = (fused.linear if native else fused.FuncLinear.apply)(*x)
    dy, c = torch.randn_like(y).requires_grad_(), torch.randn_like(x[2])
    got = torch.autograd.grad(y, [x[i] for i in pick], dy, create_graph=True)
    assert torch.equal(torch.autograd.grad(got[-1], dy, c)[0], c.expand_as(dy))
    assert all(torch.equal(a, b) for a, b in zip(got, torch.autograd.grad(fused.linear(*x), [x[i] for i in pick], dy.detach())))
