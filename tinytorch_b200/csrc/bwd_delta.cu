// The first step of every attention backward: delta[b,h,i] = sum_d dO[i,d] * O[i,d], which is the rowsum(P o dP) of
//   dS = P o (dP - rowsum(P o dP)) * scale
// in the chain linear -> mul -> add -> softmax -> linear (src/Function/FuncNNLayer.h:20-34, src/Function/FuncElemWise.h:77-87,113-123,
// src/Operation/OpNNLayerCpu.h:78-109) that defines the gradient which FuncSDPAttention::backward leaves out (FuncNNLayer.h:267).
#include <type_traits>

#include "f32_pieces.cuh"

namespace ttattn {
namespace {

constexpr int kThreads = 256;

// Rows whose log-sum-exp is further from 0 than this are looked at again here (additive masks, fp32).  An lse of -1e9, of a query whose keys all have
// a mask of -1e9, say, has lost the logarithm of their number, and exponents with it, the difference of two large numbers, are off by whole units:
// 2^18 instead of 1 / 90, or infinite.  Such a row's maximum and sum are kept apart, in scratch memory.  (Below, the roundings of lse are less than
// twice those of a score and mask of its size; a row's threads take 13 us for 500 keys of 64 elements.)  A row whose dO is zero, as padded
// queries' are, gives nothing, whatever its probabilities: it gets none.
constexpr float kLargeLse = 4096.f;

// A row's maximum, negated, and the inverse of its sum, from its scores, masked as the forward's kernels do it: by TPR neighbouring threads, `lanes` of
// their warp, thread `part` the keys part, part + TPR, ...  The main kernel's products differ in their last bits, and a sum that is rounded up there must
// not be beyond the maximum (by 128 at 1e9): scores are taken at the upper end of what they may be.
template <int D, int TPR>
__device__ __forceinline__ float2 scan_row(const BwdArgs& a, int b, int h, int i, int kv_len, int part, uint32_t lanes) {
  const int hk = h / (a.Hq / a.Hkv), seen = a.causal ? min(kv_len, i + causal_shift(a.causal, kv_len, a.Lq) + 1) : kv_len;
  const float4* q = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.q) + b * a.qs.b + h * a.qs.h + static_cast<int64_t>(i) * a.qs.s);
  const float* k = reinterpret_cast<const float*>(a.k) + b * a.ks.b + hk * a.ks.h;
  const float* mask = reinterpret_cast<const float*>(a.mask.ptr) + b * a.mask.sb + h * a.mask.sh + i * a.mask.sl;
  const float c = a.scale * kLog2e;
  float m = -INFINITY, l = 0.f;
  for (int key = part; key < seen; key += TPR) {
    const float4* row = reinterpret_cast<const float4*>(k + static_cast<int64_t>(key) * a.ks.s);
    float s = 0.f, size = 0.f;
#pragma unroll 8
    for (int d = 0; d < D / 4; ++d) {
      const float4 x = __ldg(q + d), y = __ldg(row + d);
      s = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, s))));
      size += fabsf(x.x * y.x) + fabsf(x.y * y.y) + fabsf(x.z * y.z) + fabsf(x.w * y.w);
    }
    // (a chain of D additions, and the other's, are off by D 2^-24 of the products' sizes at most)
    const float t = fmaf(mask[key], kLog2e, fmaf(size, fabsf(c) * (D * 0x1p-23f), s * c)), top = fmaxf(m, t);
    if (t != -INFINITY) l = fmaf(l, exp2f(m - top), exp2f(t - top));
    m = top;
  }
#pragma unroll
  for (int of = TPR / 2; of >= 1; of >>= 1) {
    const float m2 = __shfl_xor_sync(lanes, m, of), l2 = __shfl_xor_sync(lanes, l, of), top = fmaxf(m, m2);
    if (top != -INFINITY) l = l * exp2f(m - top) + l2 * exp2f(m2 - top);
    m = top;
  }
  return make_float2(-m, 1.f / l);
}

// delta[b,h,i] = sum_d dO[i,d] * O[i,d].  Each thread reads 16 bytes of a row of
// O and of dO; the D*sizeof(T)/16 threads of a row reduce with shuffles.  For the
// tensor-core backward the same pass clears the fp32 dQ accumulator (its TMA
// reductions need zeros to start from), which saves a separate memset of that size.
template <typename T, int D>
__global__ void __launch_bounds__(kThreads, 8) bwd_delta_kernel(const BwdArgs a) {
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
  const uint32_t i = row % a.Lq, bh = row / a.Lq, h = bh % a.Hq, b = bh / a.Hq;
  float s = 0.f;
  bool any = false;  // whether this part of dO is not all zero
  float lse = 0.f;
  if (row < total) {
    const T* o = reinterpret_cast<const T*>(a.o) + b * a.os.b + h * a.os.h + static_cast<int64_t>(i) * a.os.s + part * N;
    const T* g =
        reinterpret_cast<const T*>(a.d_o) + b * a.dos.b + h * a.dos.h + static_cast<int64_t>(i) * a.dos.s + part * N;
    const uint4 ov = *reinterpret_cast<const uint4*>(o), gv = *reinterpret_cast<const uint4*>(g);
    const T* op = reinterpret_cast<const T*>(&ov);
    const T* gp = reinterpret_cast<const T*>(&gv);
#pragma unroll
    for (int e = 0; e < N; ++e) s = fmaf(to_f32<T>(op[e]), to_f32<T>(gp[e]), s);
    if constexpr (std::is_same_v<T, float>) lse = a.row_stats ? a.lse[row] : 0.f, any = gp[0] != 0.f || gp[1] != 0.f || gp[2] != 0.f || gp[3] != 0.f;
    if (a.zero_dq_accum) {
      float4* z = reinterpret_cast<float4*>(a.dq_accum + static_cast<int64_t>(row) * D + part * N);
#pragma unroll
      for (int e = 0; e < N / 4; ++e) z[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll
  for (int of = TPR / 2; of >= 1; of >>= 1) s += __shfl_xor_sync(0xffffffffu, s, of);
  if (part == 0 && row < total) a.delta[row] = s;
  if constexpr (std::is_same_v<T, float>) {
    if (!a.row_stats) return;
    const uint32_t lanes = (TPR == 32 ? 0xffffffffu : (1u << TPR) - 1) << (threadIdx.x & 31 & ~(TPR - 1));
    const bool some = (__ballot_sync(0xffffffffu, any) & lanes) != 0;
    if (row >= total) return;
    int kv_len = a.Skv;
    if (a.kv_lens) kv_len = max(0, min(a.kv_lens[b], a.Skv));
    float2 stats = pieces::exponent_base(lse, kv_len);
    if (fabsf(lse) >= kLargeLse && fabsf(lse) != INFINITY) stats = some ? scan_row<D, TPR>(a, b, h, i, kv_len, part, lanes) : make_float2(-INFINITY, 1.f);
    if (part == 0) a.row_stats[row] = stats;
  }
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
