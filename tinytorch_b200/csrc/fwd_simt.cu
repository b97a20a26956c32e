// Prefill forward in full fp32 arithmetic (CUDA cores, FMA) for Float32 tensors.
//
// The reference's CUDA fp32 matmul runs in TF32 (src/Utils/CUDAUtils.cpp:148-155),
// which cannot meet a 1e-5 relative bound against its own CPU path
// (src/Operation/OpLinalgCpu.h:138-150); this kernel therefore keeps every
// product and sum in fp32.  Same fusion as the tensor-core kernel: one CTA owns a
// 64-row query tile of one (batch, head), streams 64-key tiles through shared
// memory, keeps an online softmax (warp-shuffle row max over the 16 lanes that
// share a row) and never writes scores to HBM.
//
// Bound by the FMA pipes (74 TFLOP/s at 1965 MHz).  128 threads, 8 x 4 scores and 8 x D/16 outputs per thread
// (simt_tile.cuh); the next K tile is copied in under the P V product and the next V tile under Q K^T; 3 CTAs of
// D = 64 and 2 of D = 128 share an SM.  B4 H16 S2048 D64 causal: 1587 -> 958 us (21.7 -> 35.9 TFLOP/s) against scalar
// shared-memory loads (eight per sixteen FMAs); ncu: FMA pipe 58 % busy, 2.7 warps per scheduler, the rest latency.
#include "simt_tile.cuh"

namespace ttattn {
namespace {

using namespace simt;
constexpr int kThreads = 128, TY = kThreads / 16, R = TS / TY;

template <int D>
constexpr int kSmemBytes = (3 * kTileFloats<D> + kScoreFloats) * static_cast<int>(sizeof(float));

template <int D, bool MASK>
__global__ void __launch_bounds__(kThreads, D == 64 && !MASK ? 3 : 2) fwd_simt_kernel(const FwdArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;
  float* Ks = Qs + kTileFloats<D>;
  float* Vs = Ks + kTileFloats<D>;
  float* Ps = Vs + kTileFloats<D>;

  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int mt = static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x);  // under a causal mask the last is longest
  const int h = blockIdx.y, b = blockIdx.z, hk = h / (a.Hq / a.Hkv);
  const int row0 = mt * TS;
  const float* q = reinterpret_cast<const float*>(a.q) + b * a.qs.b + h * a.qs.h;
  const float* k = reinterpret_cast<const float*>(a.k) + b * a.ks.b + hk * a.ks.h;
  const float* v = reinterpret_cast<const float*>(a.v) + b * a.vs.b + hk * a.vs.h;

  int kv_len = a.Skv;
  if (a.kv_lens) {
    int l = a.kv_lens[b];
    kv_len = l < 0 ? 0 : (l < a.Skv ? l : a.Skv);
  }
  const int shift = causal_shift(a.causal, kv_len, a.Lq);
  int kv_end = kv_len;
  if (a.causal && row0 + TS + shift < kv_end) kv_end = row0 + TS + shift > 0 ? row0 + TS + shift : 0;
  const int n_tiles = (kv_end + TS - 1) / TS;
  const float c = a.scale * kLog2e;
  const int64_t mask_base = b * a.mask.sb + h * a.mask.sh;

  if (n_tiles > 0) {
    load_tile<D, kThreads>(Qs, q, a.qs.s, row0, a.Lq, tid);
    load_tile<D, kThreads>(Ks, k, a.ks.s, 0, kv_len, tid);
    copies_commit();
    load_tile<D, kThreads>(Vs, v, a.vs.s, 0, kv_len, tid);
    copies_commit();
  }

  float m[R], l[R];
  float2 acc[R][D / 32];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    m[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
    for (int j = 0; j < D / 32; ++j) acc[i][j] = make_float2(0.f, 0.f);
  }

  for (int t = 0; t < n_tiles; ++t) {
    const int col0 = t * TS;
    copies_wait<1>();  // Q and K of this tile; V may still be on its way
    __syncthreads();
    float bias[MASK ? R : 1][4];
    if constexpr (MASK) {
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int row = row0 + ty + TY * i, col = col0 + tx + 16 * j;
          bias[i][j] = row < a.Lq && col < kv_len ? mask_bias2<float>(a.mask, mask_base + row * a.mask.sl + col) : 0.f;
        }
    }
    float s[R][4];
    product_nt<D, TY>(Qs, Ks, ty, tx, s);
    __syncthreads();  // K of this tile has been read
    if (t + 1 < n_tiles) load_tile<D, kThreads>(Ks, k, a.ks.s, col0 + TS, kv_len, tid);
    copies_commit();
    const bool edge = col0 + TS > kv_len || (a.causal && col0 + TS - 1 > row0 + shift);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = row0 + ty + TY * i;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] *= c;
        if constexpr (MASK) s[i][j] += bias[i][j];
        const int col = col0 + tx + 16 * j;
        if (edge && !(col < kv_len && (!a.causal || col <= row + shift))) s[i][j] = -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o >= 1; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m[i], mx);
      // a row that has seen no participating key yet keeps m = -inf; its
      // exponentials are taken against 0 and are all 0
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float alpha = exp2f(m[i] - m_use);
      m[i] = m_new;
      l[i] *= alpha;
      const float2 alpha2 = make_float2(alpha, alpha);
#pragma unroll
      for (int j = 0; j < D / 32; ++j) acc[i][j] = ptx::mul2(acc[i][j], alpha2);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = exp2f(s[i][j] - m_use);
        l[i] += p;
        Ps[(ty + TY * i) * LP + tx + 16 * j] = p;
      }
    }
    copies_wait<1>();  // V of this tile
    __syncthreads();
    product_nn<D, TY>(Ps, Vs, ty, tx, acc);
    __syncthreads();  // V and P have been read
    if (t + 1 < n_tiles) load_tile<D, kThreads>(Vs, v, a.vs.s, col0 + TS, kv_len, tid);
    copies_commit();
  }

  float* o = reinterpret_cast<float*>(a.o) + b * a.os.b + h * a.os.h;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    float ls = l[i];
#pragma unroll
    for (int of = 8; of >= 1; of >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, of);
    const int row = row0 + ty + TY * i;
    if (row >= a.Lq) continue;
    const float inv = ls > 0.f ? 1.f / ls : 0.f;
#pragma unroll
    for (int j = 0; j < D / 64; ++j)
      *reinterpret_cast<float4*>(o + static_cast<int64_t>(row) * a.os.s + tx * 4 + j * 64) =
          make_float4(acc[i][2 * j].x * inv, acc[i][2 * j].y * inv, acc[i][2 * j + 1].x * inv, acc[i][2 * j + 1].y * inv);
    if (a.lse && tx == 0)
      a.lse[(static_cast<int64_t>(b) * a.Hq + h) * a.Lq + row] = ls > 0.f ? (m[i] + log2f(ls)) * kLn2 : -INFINITY;
  }
}

template <int D, bool MASK>
cudaError_t launch_t(const FwdArgs& a, cudaStream_t stream) {
  auto kern = fwd_simt_kernel<D, MASK>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes<D>);
  if (e != cudaSuccess) return e;
  dim3 grid((a.Lq + TS - 1) / TS, a.Hq, a.B);
  kern<<<grid, kThreads, kSmemBytes<D>, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_fwd_simt(int dtype, int D, const FwdArgs& a, cudaStream_t stream) {
  if (dtype != TT_ATTN_F32) return cudaErrorInvalidValue;
  const bool mask = a.mask.ptr != nullptr;
  if (D == 64) return mask ? launch_t<64, true>(a, stream) : launch_t<64, false>(a, stream);
  if (D == 128) return mask ? launch_t<128, true>(a, stream) : launch_t<128, false>(a, stream);
  return cudaErrorInvalidValue;
}

}  // namespace ttattn
