/*
 * tt_fused.h - C ABI of the operators that sit either side of attention in a
 * transformer block, exported by libtt_attn.so for NVIDIA B200 (sm_100a): the two
 * fused element-wise / row operators (HBM-bound streaming kernels) and the
 * projection y = x w^T + bias (tensor cores).
 *
 *   tt_fused_add_rms_norm  replaces fusedAddRmsNormOpCudaImpl
 *                          (src/Operation/OpFusedCuda.cuh:103-142; CPU form
 *                          src/Operation/OpFusedCpu.h:42-72)
 *   tt_silu_mul            replaces siluMulOpCudaImpl
 *                          (src/Operation/OpFusedCuda.cuh:16-101; CPU form
 *                          src/Operation/OpFusedCpu.h:14-39)
 *   tt_linear              replaces the library gemm behind function::linear =
 *                          op::matmul(input, weight, false, true, bias) for 16-bit
 *                          tensors (src/Function/FuncNNLayer.h:14-19,
 *                          src/Operation/OpLinalg.cpp:243-269,
 *                          src/Operation/OpLinalgCuda.cuh:141-215; CPU form
 *                          src/Operation/OpLinalgCpu.h:118-151)
 *
 * dtype uses the reference's enum values (src/Tensor/DType.h:20-24): 0 = Float32,
 * 1 = Float16, 2 = BFloat16.  Arithmetic is fp32 with one rounding to the tensor
 * dtype per stored value, as in the reference's CUDA kernels.  Tensors are dense and
 * row-major with the normalised / gated dimension innermost.  Work is enqueued on
 * `stream` of `device`; nothing synchronises the host or allocates.  Return value: 0
 * or a negative tt_attn_status (tt_attn.h).
 */
#ifndef TT_FUSED_H_
#define TT_FUSED_H_

#include "tt_attn.h"

#ifdef __cplusplus
extern "C" {
#endif

/* In place, exactly as op::fusedAddRmsNorm(input, residual, weight, eps):
 *   residual <- T(input + residual)                         (fp32 add, rounded to T)
 *   input    <- T(residual * rsqrt(mean(r^2) + eps) * weight)
 * where the mean runs over the unrounded fp32 sums r and the product uses the
 * rounded residual (src/Operation/OpFusedCuda.cuh:110-127). */
typedef struct tt_fused_add_rms_norm_params {
  uint32_t struct_size;
  int32_t dtype;
  int64_t rows, dim;
  void* input;        /* [rows, dim], read and overwritten */
  void* residual;     /* [rows, dim], read and overwritten */
  const void* weight; /* [dim] */
  float eps;
  int32_t device;
  void* stream;
} tt_fused_add_rms_norm_params;

/* out[r, j] = silu(x[r, j]) * x[r, d + j] for x [rows, 2d], silu(g) = g / (1 + exp(-g))
 * (src/Operation/OpFusedCuda.cuh:38-42). */
typedef struct tt_silu_mul_params {
  uint32_t struct_size;
  int32_t dtype;
  int64_t rows, d; /* d = half of x's last dimension */
  const void* x;   /* [rows, 2d] */
  void* out;       /* [rows, d] */
  int32_t device;
  void* stream;
} tt_silu_mul_params;

/* y[M,N] = x[M,K] w[N,K]^T + bias[N] (bias may be NULL), Float16 / BFloat16 only (Float32
 * stays on the library gemm: TT_ATTN_ERR_DTYPE).  fp32 accumulation, the bias is added in
 * fp32 before the single rounding to the tensor dtype.  ldx / ldw / ldy are the row strides
 * in elements (0 = dense); K, N and the strides must be multiples of 8 and the pointers
 * 16-byte aligned (TT_ATTN_ERR_ALIGN otherwise).  `status` (optional device word) receives a
 * non-zero value if a bounded device-side wait expired.
 * The gradient products of FuncLinear::backward (src/Function/FuncNNLayer.h:20-34) contract
 * over the rows of an operand; x_t / w_t (added to the end of the struct; a caller with the
 * shorter struct_size gets 0) say that the operand is stored with the contraction as its slow
 * dimension, so that no transposed copy is needed:
 *   dX[M,K] = dY W     x = dY, w = W (stored [contraction N, K]), w_t = 1
 *   dW[N,K] = dY^T X   x = dY (stored [contraction M, N]), w = X (stored [contraction M, K]),
 *                      x_t = w_t = 1; K (the contraction) may then be any size
 * x_sum (optional, with x_t): [M] receives the sums of x over the contraction, in the tensor
 * dtype (fp32 accumulation): db = sum of dY over its rows, beside dW; with w and y both NULL
 * the sums alone. */
typedef struct tt_linear_params {
  uint32_t struct_size;
  int32_t dtype;
  int64_t M, N, K;
  const void* x;    /* [M, K]; with x_t [K, M] */
  const void* w;    /* [N, K]; with w_t [K, N] */
  const void* bias; /* [N] or NULL */
  void* y;          /* [M, N] */
  int64_t ldx, ldw, ldy;
  int32_t device;
  void* stream;
  int32_t* status;
  int32_t x_t, w_t;
  void* x_sum; /* [M] or NULL */
} tt_linear_params;

TT_ATTN_API int tt_linear(const tt_linear_params* p);

/* For tests: the same projection with a tile of the caller's choice among those that tt_linear chooses
 * from.  `shape`: the columns of a tile of single CTAs (64 .. 256 in steps of 32, with w_t of 64), or -192
 * for pairs (not with w_t); TT_ATTN_ERR_SHAPE for any other.  0 launches nothing.  `planned` (host memory,
 * or NULL with a shape) receives what tt_linear takes: such a number, -256 for pairs of 256 x 256, 0 for
 * the contraction divided over a cluster.  x_sum is not written. */
TT_ATTN_API int tt_linear_selftest(const tt_linear_params* p, int32_t shape, int32_t* planned);
TT_ATTN_API int tt_fused_add_rms_norm(const tt_fused_add_rms_norm_params* p);
TT_ATTN_API int tt_silu_mul(const tt_silu_mul_params* p);

#ifdef __cplusplus
}
#endif
#endif /* TT_FUSED_H_ */
