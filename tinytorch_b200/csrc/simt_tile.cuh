// Building blocks of the fp32 attention kernels (fwd_simt.cu, bwd_simt.cu): 64-row tiles in shared memory and the two
// forms of product on them, on CUDA cores with packed fp32 FMAs.
//
// A thread grid of 16 columns (tx) x TY rows (ty) works on a tile; a thread owns R = 64 / TY rows.  Every operand
// comes from shared memory as 16-byte vectors: with R = 8 one vector feeds ten FMAs (the scalar loads these replace:
// two), and a warp's vectors fall on at most two wavefronts.  Row strides carry 4 floats of padding, which puts eight
// consecutive rows on different banks.  Sums run as fma.rn.f32x2: two fp32 FMAs per issued instruction, each rounded
// as the scalar one.  (Unrolling the vector loops 4 / 4 / 8 times: 3-5 % over 2 / 2 / 4; whole or not at all: slower.)
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace ttattn {
namespace simt {

constexpr int TS = 64;        // rows (queries or keys) of a tile
constexpr int LP = TS + 4;    // row stride of a 64 x 64 score tile
template <int D>
constexpr int kLd = D + 4;    // row stride of a [64, D] tile
template <int D>
constexpr int kTileFloats = TS * kLd<D>;
constexpr int kScoreFloats = TS * LP;

// rows [row0, row0 + 64) of src into dst[64][kLd<D>] by asynchronous 16-byte copies; rows at or beyond `valid` are zero
template <int D, int NT>
__device__ __forceinline__ void load_tile(float* dst, const float* src, int64_t row_stride, int row0, int valid, int tid) {
  const uint32_t base = ptx::smem_u32(dst);
#pragma unroll
  for (int i = 0; i < TS * (D / 4) / NT; ++i) {
    const int idx = tid + i * NT, r = idx / (D / 4), c4 = (idx % (D / 4)) * 4;
    const bool in = row0 + r < valid;
    const float* p = src + static_cast<int64_t>(in ? row0 + r : 0) * row_stride + c4;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + (r * kLd<D> + c4) * 4), "l"(p), "r"(in ? 16 : 0)
                 : "memory");
  }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {  // all but the last N committed groups have arrived
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// out[i][j] = sum_d A[ty + TY i][d] * B[tx + 16 j][d]
template <int D, int TY>
__device__ __forceinline__ void product_nt(const float* A, const float* B, int ty, int tx, float (&out)[TS / TY][4]) {
  constexpr int R = TS / TY;
  float2 acc[R][4];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  const float* ap = A + ty * kLd<D>;
  const float* bp = B + tx * kLd<D>;
#pragma unroll 4
  for (int d = 0; d < D; d += 4) {
    float4 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(bp + j * 16 * kLd<D> + d);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(ap + i * TY * kLd<D> + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = ptx::fma2(lo2(a), lo2(b[j]), acc[i][j]);
        acc[i][j] = ptx::fma2(hi2(a), hi2(b[j]), acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) out[i][j] = acc[i][j].x + acc[i][j].y;
}

// acc[i][.] += sum_k P[ty + TY i][k] * V[k][tx * 4 + 64 c ..]   (acc holds pairs of columns: 2 per group c of 4)
template <int D, int TY>
__device__ __forceinline__ void product_nn(const float* P, const float* V, int ty, int tx, float2 (&acc)[TS / TY][D / 32]) {
  constexpr int R = TS / TY, DC = D / 64;
  const float* pp = P + ty * LP;
#pragma unroll 4
  for (int k = 0; k < TS; k += 4) {
    float4 v[4][DC];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < DC; ++c) v[q][c] = *reinterpret_cast<const float4*>(V + (k + q) * kLd<D> + tx * 4 + c * 64);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 p4 = *reinterpret_cast<const float4*>(pp + i * TY * LP + k);
      const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < DC; ++c) {
          const float2 pq = make_float2(p[q], p[q]);
          acc[i][2 * c] = ptx::fma2(pq, lo2(v[q][c]), acc[i][2 * c]);
          acc[i][2 * c + 1] = ptx::fma2(pq, hi2(v[q][c]), acc[i][2 * c + 1]);
        }
    }
  }
}

// acc[i][.] += sum_k P[k][ty * R + i] * X[k][tx * 4 + 64 c ..]: the score tile transposed
template <int D, int TY>
__device__ __forceinline__ void product_tn(const float* P, const float* X, int ty, int tx, float2 (&acc)[TS / TY][D / 32]) {
  constexpr int R = TS / TY, DC = D / 64;
#pragma unroll 8
  for (int k = 0; k < TS; ++k) {
    float p[R];
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 p4 = *reinterpret_cast<const float4*>(P + k * LP + ty * R + i);
      p[i] = p4.x, p[i + 1] = p4.y, p[i + 2] = p4.z, p[i + 3] = p4.w;
    }
#pragma unroll
    for (int c = 0; c < DC; ++c) {
      const float4 x = *reinterpret_cast<const float4*>(X + k * kLd<D> + tx * 4 + c * 64);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float2 pi = make_float2(p[i], p[i]);
        acc[i][2 * c] = ptx::fma2(pi, lo2(x), acc[i][2 * c]);
        acc[i][2 * c + 1] = ptx::fma2(pi, hi2(x), acc[i][2 * c + 1]);
      }
    }
  }
}

// The mask elements (times log2 e) of this thread's scores: rows row, row + TY, .., columns col, col + 16, ..; 0 outside.
template <int TY, int R>
__device__ __forceinline__ void load_mask(const MaskArgs& m, int64_t base, int row, int n_rows, int col, int n_cols,
                                          float (&bias)[R][4]) {
  auto load = [&](auto* p, auto value) {  // (one loop per kind: nothing is decided per element)
    p += base + row * m.sl + col;
#pragma unroll
    for (int i = 0; i < R; ++i, p += TY * m.sl)
#pragma unroll
      for (int j = 0; j < 4; ++j) bias[i][j] = row + TY * i < n_rows && col + 16 * j < n_cols ? value(p[16 * j]) : 0.f;
  };
  if (m.kind == TT_ATTN_MASK_BOOL) load(reinterpret_cast<const uint8_t*>(m.ptr), [](uint8_t x) { return x ? 0.f : -INFINITY; });
  else load(reinterpret_cast<const float*>(m.ptr), [](float x) { return x * kLog2e; });
}

}  // namespace simt
}  // namespace ttattn
