"""The reference's two hand-fused transformer-block operators on B200, with the
reference's names, argument meaning and in-place behaviour:

  siluMul(x)                                   op::siluMul, function::siluMul
      (src/Operation/OpFused.h:19, src/Function/FuncFused.h:14-19,31)
  fusedAddRmsNorm(input, residual, weight, eps)  op::fusedAddRmsNorm, function::fusedAddRmsNorm
      (src/Operation/OpFused.h:22, src/Function/FuncFused.h:21-28,33-35)

  linear(input, weight, bias=None)            function::linear
      (src/Function/FuncNNLayer.h:14-35,270-272): input [..., K] x weight [N, K]^T + bias [N];
      float16 / bfloat16 on the tensor cores (float32 stays on the library gemm and is refused here),
      with the reference's backward (dX = dY W, dW = dY^T X, db = sum dY) through the same kernel

All go through the C ABI of libtt_attn.so (include/tt_fused.h) and launch on the
current CUDA stream of the tensors' device.  None has a CPU implementation here, and - as
in the reference (FuncFused.h:18,27) - siluMul and fusedAddRmsNorm have no backward.
"""
import torch

from . import _capi


def siluMul(x):
    """x [..., 2d] -> silu(x[..., :d]) * x[..., d:], a new tensor [..., d]."""
    return _capi.native().silu_mul(x)


def fusedAddRmsNorm(input, residual, weight, eps):
    """In place: residual += input; input = rmsnorm(residual) * weight.  Returns None, like the reference."""
    _capi.native().add_rms_norm(input, residual, weight, eps)


def _linear_raw(x2, w, bias, status=None):
    """x2 [M, K] @ w [N, K]^T (+ bias [N]) -> [M, N]; rows may be strided, columns are contiguous."""
    return _capi.native().linear_raw(x2, w, bias, status)


class FuncLinear(torch.autograd.Function):
    """function::FuncLinear (src/Function/FuncNNLayer.h:14-35) on the tcgen05 kernels as a Python autograd function, for what
    the native node (LinearBackward in csrc/binding.cpp) does not do; see function.FuncSDPAttention."""

    @staticmethod
    def forward(ctx, input, weight, bias):
        x2 = input.reshape(-1, input.shape[-1])
        if x2.stride(1) != 1:
            x2 = x2.contiguous()
        w = weight if weight.stride(1) == 1 else weight.contiguous()
        ctx.save_for_backward(x2, w)
        ctx.in_shape = input.shape
        return _linear_raw(x2, w, bias).reshape(input.shape[:-1] + (weight.shape[0],))

    @staticmethod
    def backward(ctx, grad):
        x2, w = ctx.saved_tensors
        need_dx, need_dw, need_db = ctx.needs_input_grad
        again = need_db and torch.is_grad_enabled() and grad.requires_grad  # create_graph: db can be differentiated again
        dx, dw, db = _capi.native().linear_bwd(grad, x2, w, need_dx, need_dw, need_db and not again)
        if again:
            db = grad.reshape(-1, grad.shape[-1]).float().sum(0).to(grad.dtype)
        return dx if dx is None else dx.reshape(ctx.in_shape), dw, db


def linear(input, weight, bias=None):
    """Drop-in for function::linear (src/Function/FuncNNLayer.h:270-272)."""
    y = _capi.native().linear(input, weight, bias)
    return FuncLinear.apply(input, weight, bias) if y is NotImplemented else y
