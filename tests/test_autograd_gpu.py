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
