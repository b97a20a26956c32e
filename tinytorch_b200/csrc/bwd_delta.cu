// The first step of every attention backward: delta[b,h,i] = sum_d dO[i,d] * O[i,d], which is the rowsum(P o dP) of
//   dS = P o (dP - rowsum(P o dP)) * scale
// in the chain linear -> mul -> add -> softmax -> linear (src/Function/FuncNNLayer.h:20-34, src/Function/FuncElemWise.h:77-87,113-123,
// src/Operation/OpNNLayerCpu.h:78-109) that defines the gradient which FuncSDPAttention::backward leaves out (FuncNNLayer.h:267).
#include "common.cuh"

namespace ttattn {
namespace {

constexpr int kThreads = 256;

// delta[b,h,i] = sum_d dO[i,d] * O[i,d].  Each thread reads 16 bytes of a row of
// O and of dO; the D*sizeof(T)/16 threads of a row reduce with shuffles.  For the
// tensor-core backward the same pass clears the fp32 dQ accumulator (its TMA
// reductions need zeros to start from), which saves a separate memset of that size.
template <typename T, int D>
__global__ void __launch_bounds__(kThreads) bwd_delta_kernel(const BwdArgs a) {
  // Launched early itself.  The main kernel may come up, and start on Q, K, V and dO without waiting for this grid, once
  // every CTA here has seen everything before it complete.
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  if (a.sched && blockIdx.x == 0 && threadIdx.x == 0) *a.sched = 0;  // the main kernel's work counter
  if (a.mask_pure) {  // ... and the lengths that a padding mask comes to
    int32_t* lens = a.mask_lens;
    for (int b = blockIdx.x; b < a.B; b += gridDim.x) masked_lens(a.mask, a.kv_lens, a.Skv, b, lens, lens + a.B);
  }
  constexpr int N = 16 / sizeof(T);  // elements per thread
  constexpr int TPR = D / N;         // threads per row (8, 16 or 32)
  // (a device holds fewer than 2^31 rows of 64 elements)
  const uint32_t row = blockIdx.x * (kThreads / TPR) + threadIdx.x / TPR;
  const int part = threadIdx.x % TPR;
  const uint32_t total = static_cast<uint32_t>(a.B) * a.Hq * a.Lq;
  float s = 0.f;
  if (row < total) {
    const uint32_t i = row % a.Lq, bh = row / a.Lq, h = bh % a.Hq, b = bh / a.Hq;
    const T* o = reinterpret_cast<const T*>(a.o) + b * a.os.b + h * a.os.h + static_cast<int64_t>(i) * a.os.s + part * N;
    const T* g =
        reinterpret_cast<const T*>(a.d_o) + b * a.dos.b + h * a.dos.h + static_cast<int64_t>(i) * a.dos.s + part * N;
    const uint4 ov = *reinterpret_cast<const uint4*>(o), gv = *reinterpret_cast<const uint4*>(g);
    const T* op = reinterpret_cast<const T*>(&ov);
    const T* gp = reinterpret_cast<const T*>(&gv);
#pragma unroll
    for (int e = 0; e < N; ++e) s = fmaf(to_f32<T>(op[e]), to_f32<T>(gp[e]), s);
    if (a.zero_dq_accum) {
      float4* z = reinterpret_cast<float4*>(a.dq_accum + static_cast<int64_t>(row) * D + part * N);
#pragma unroll
      for (int e = 0; e < N / 4; ++e) z[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll
  for (int of = TPR / 2; of >= 1; of >>= 1) s += __shfl_xor_sync(0xffffffffu, s, of);
  if (part == 0 && row < total) a.delta[row] = s;
}

template <typename T, int D>
cudaError_t launch_delta_t(const BwdArgs& a, cudaStream_t stream) {
  const int64_t rows = static_cast<int64_t>(a.B) * a.Hq * a.Lq;
  if (rows > 0x7fffffffll) return cudaErrorInvalidValue;
  return launch_early(bwd_delta_kernel<T, D>, dim3(static_cast<unsigned>((rows * (D * sizeof(T) / 16) + kThreads - 1) / kThreads)), dim3(kThreads), 0,
                      stream, 1, a);
}

}  // namespace

cudaError_t launch_bwd_delta(int dtype, int D, const BwdArgs& a, cudaStream_t stream) {
  if (dtype == TT_ATTN_F32) return D == 64 ? launch_delta_t<float, 64>(a, stream) : launch_delta_t<float, 128>(a, stream);
  if (dtype == TT_ATTN_F16)
    return D == 64 ? launch_delta_t<__half, 64>(a, stream) : launch_delta_t<__half, 128>(a, stream);
  return D == 64 ? launch_delta_t<__nv_bfloat16, 64>(a, stream) : launch_delta_t<__nv_bfloat16, 128>(a, stream);
}

}  // namespace ttattn
