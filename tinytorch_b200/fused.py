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


class FuncLinear:
    """function::FuncLinear (src/Function/FuncNNLayer.h:14-35) on the tcgen05 kernel; its node is LinearBackward in
    csrc/binding.cpp."""

    @staticmethod
    def apply(input, weight, bias):
        return _capi.native().linear(input, weight, bias)


def linear(input, weight, bias=None):
    """Drop-in for function::linear (src/Function/FuncNNLayer.h:270-272)."""
    return _capi.native().linear(input, weight, bias)
