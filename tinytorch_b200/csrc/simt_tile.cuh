// Building blocks of the fp32 backward kernels (bwd_simt.cu): 64-row tiles in shared memory and the two
// forms of product on them, on CUDA cores with packed fp32 FMAs.
//
// A thread grid of 16 columns (tx) x TY rows (ty) works on a tile; a thread owns R = 64 / TY rows.  Every operand
// comes from shared memory as 16-byte vectors: with R = 8 one vector feeds ten FMAs (the scalar loads these replace:
// two), and a warp's vectors fall on at most two wavefronts.  Row strides carry 4 floats of padding, which puts eight
// consecutive rows on different banks.  An operand of which a warp reads two consecutive rows at a time (the first of a
// product) can do without: kSwap exchanges neighbouring pieces of the odd rows instead.  Sums run as fma.rn.f32x2: two fp32 FMAs per issued instruction, each rounded
// as the scalar one.  (Unrolling the vector loops 4 / 4 / 8 times: 3-5 % over 2 / 2 / 4; whole or not at all: slower.)
#pragma once
#include <atomic>

#include "common.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"

namespace ttattn {
namespace simt {

constexpr int TS = 64;        // rows (queries or keys) of a tile
constexpr int LP = TS + 4;    // row stride of a 64 x 64 score tile
template <int D>
constexpr int kLd = D + 4;    // row stride of a [64, D] tile
template <int D>
constexpr int kTileFloats = TS * kLd<D>;
constexpr int kScoreFloats = TS * LP;

// How a tile lies in shared memory: padded rows; rows as they are; rows as they are, with neighbouring vectors of the odd
// rows exchanged (of a score tile: neighbouring halves of 32 columns; kSwapHalves copies one in like that).
enum Layout { kPad, kPlain, kSwap, kSwapHalves };

// rows [row0, row0 + 64) of src into dst by asynchronous 16-byte copies; rows at or beyond `valid` are zero
template <int D, int NT, Layout LAY = kPad>
__device__ __forceinline__ void load_tile(float* dst, const float* src, int64_t row_stride, int row0, int valid, int tid) {
  const uint32_t base = ptx::smem_u32(dst);
#pragma unroll
  for (int i = 0; i < TS * (D / 4) / NT; ++i) {
    const int idx = tid + i * NT, r = idx / (D / 4), c4 = (idx % (D / 4)) * 4;
    const bool in = row0 + r < valid;
    const float* p = src + static_cast<int64_t>(in ? row0 + r : 0) * row_stride + c4;
    const int swap = LAY == kSwap ? 4 : (LAY == kSwapHalves ? 16 : 0), at = r * (LAY == kPad ? kLd<D> : D) + (c4 ^ (r & 1) * swap);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + at * 4), "l"(p), "r"(in ? 16 : 0)
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
template <int D, int TY, Layout LA = kPad>
__device__ __forceinline__ void product_nt(const float* A, const float* B, int ty, int tx, float (&out)[TS / TY][4]) {
  constexpr int R = TS / TY, LDA = LA == kPad ? kLd<D> : D;
  float2 acc[R][4];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  const int odd = LA == kSwap ? (ty & 1) * 4 : 0;  // (of all rows ty + TY i)
  const float* ap[2] = {A + ty * LDA + odd, A + ty * LDA - odd};
  const float* bp = B + tx * kLd<D>;
#pragma unroll 1
  for (int d0 = 0; d0 < D; d0 += 16) {
#pragma unroll
    for (int d = d0; d < d0 + 16; d += 4) {
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(bp + j * 16 * kLd<D> + d);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(ap[(d - d0) / 4 & 1] + i * TY * LDA + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = ptx::fma2(lo2(a), lo2(b[j]), acc[i][j]);
          acc[i][j] = ptx::fma2(hi2(a), hi2(b[j]), acc[i][j]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) out[i][j] = acc[i][j].x + acc[i][j].y;
}

// acc[i][.] += sum_k P[ty + TY i][k] * V[k][tx * 4 + 64 c ..]   (acc holds pairs of columns: 2 per group c of 4)
template <int D, int TY, Layout LPL = kPad, Layout LV = kPad>
__device__ __forceinline__ void product_nn(const float* P, const float* V, int ty, int tx, float2 (&acc)[TS / TY][D / 32]) {
  constexpr int R = TS / TY, DC = D / 64, LDP = LPL == kPad ? LP : TS, LDV = LV == kPad ? kLd<D> : D;
  const int odd = LPL == kSwap ? (ty & 1) * 16 : 0;
#pragma unroll 1
  for (int k0 = 0; k0 < TS; k0 += 16) {
    const float* pp = P + ty * LDP + (k0 ^ odd) - k0;
#pragma unroll
    for (int k = k0; k < k0 + 16; k += 4) {
      float4 v[4][DC];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < DC; ++c) v[q][c] = *reinterpret_cast<const float4*>(V + (k + q) * LDV + tx * 4 + c * 64);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float4 p4 = *reinterpret_cast<const float4*>(pp + i * TY * LDP + k);
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

constexpr int kByteRow = TS / 4 + 1;  // words that hold the 64 bytes of a row at any offset

// The mask of a tile's scores.  Where thread (ty, tx) will write its probabilities, [(ty + TY i) LD + tx + 16 j] (kSwap: + 16 (j ^
// (ty & 1))), the tile's shared memory holds before
//   an additive mask   the thread's own elements, copied asynchronously one by one: nobody else has to wait for them;
//   a boolean one      its bytes, a row in the first 68 bytes of a row (one row where all are the same): aligned words, copied by
//                      all threads together.  Every thread has to take its own (bits) before any writes a probability,
//                      unless they lie somewhere else (stage_bytes, apply).
// (All elements in registers, fetched ahead of the product that comes first, are 32 of them: a CTA fewer to an SM.)  4 x 8
// heads x 500 with an additive mask, D = 128: forward 172 -> 125 us, without a mask 119; D = 64: backward 221 -> 202, 186.
template <int D, int TY, int NT, Layout LAY>
struct MaskTile {
  static constexpr int R = TS / TY, LD = LAY == kPad ? LP : TS;
  const MaskArgs& m;
  float* tile;
  int64_t base;  // of (batch, head)
  int ty, tx, tid;

  __device__ __forceinline__ bool additive() const { return m.kind != TT_ATTN_MASK_BOOL; }
  __device__ __forceinline__ float* mine() const { return tile + ty * LD + tx; }
  __device__ __forceinline__ int at(int i, int j) const { return i * TY * LD + (LAY == kSwap ? j ^ (ty & 1) : j) * 16; }

  // copies of the tile at (row0, col0) on their way; outside: 0 (added), anything (boolean)
  __device__ __forceinline__ void stage(int row0, int n_rows, int col0, int n_cols) const {
    if (additive())
      stage_added(row0, n_rows, col0, n_cols);
    else
      stage_bytes<LD>(tile, row0, n_rows, col0, n_cols);
  }
  __device__ __forceinline__ void stage_added(int row0, int n_rows, int col0, int n_cols) const {
    const int row = row0 + ty, col = col0 + tx;
    const float* p = reinterpret_cast<const float*>(m.ptr) + base + row * m.sl + col;
    const uint32_t dst = ptx::smem_u32(mine());
#pragma unroll
    for (int i = 0; i < R; ++i, p += TY * m.sl)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool in = row + TY * i < n_rows && col + 16 * j < n_cols;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + at(i, j) * 4),
                     "l"(in ? p + 16 * j : reinterpret_cast<const float*>(m.ptr)), "r"(in ? 4 : 0)
                     : "memory");
      }
  }
  template <int WORDS>  // of a row at `dst`
  __device__ __forceinline__ void stage_bytes(float* dst, int row0, int n_rows, int col0, int n_cols) const {
    const uint8_t* any = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(m.ptr) & ~uintptr_t(3));
    for (int e = tid; e < (m.sl == 0 ? kByteRow : TS * kByteRow); e += NT) {
      const int r = e / kByteRow, w = e - r * kByteRow;
      const uint8_t* p = reinterpret_cast<const uint8_t*>(m.ptr) + base + (row0 + r) * m.sl + col0;
      const int mis = static_cast<int>(reinterpret_cast<uintptr_t>(p) & 3);
      const bool in = row0 + r < n_rows && w * 4 - mis < n_cols - col0 && w * 4 - mis < TS;  // some byte of it is looked at
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(ptx::smem_u32(dst + r * WORDS + w)),
                   "l"(in ? p - mis + w * 4 : any), "r"(in ? 4 : 0)
                   : "memory");
    }
  }
  // boolean, bytes at `src`: scores of column col0 + tx + 16 j, scaled and masked
  template <int WORDS>
  __device__ __forceinline__ void apply(const float* src, int row0, int col0, float c, float (&s)[R][4]) const {
    const uint32_t off = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(m.ptr) + base + col0 + (row0 + ty) * m.sl);
    const uint8_t* p = reinterpret_cast<const uint8_t*>(src + ty * WORDS) + tx;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint8_t* q = p + i * TY * WORDS * 4 + ((off + i * TY * static_cast<uint32_t>(m.sl)) & 3);
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = q[16 * j] ? s[i][j] * c : -INFINITY;
    }
  }
  // boolean: bit 4 i + j: score (i, j) is hidden (or outside, where it does not count); the copies are complete and visible
  __device__ __forceinline__ uint32_t bits(int row0, int col0) const {
    const int first = m.sl == 0 ? 0 : ty, step = m.sl == 0 ? 0 : TY;
    const uint32_t off = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(m.ptr) + base + col0 + (row0 + first) * m.sl);
    const uint8_t* p = reinterpret_cast<const uint8_t*>(tile + first * LD) + tx;
    uint32_t b = 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const uint8_t* q = p + i * step * LD * 4 + ((off + i * step * static_cast<uint32_t>(m.sl)) & 3);
#pragma unroll
      for (int j = 0; j < 4; ++j) b |= q[16 * j] ? 0u : 1u << (4 * i + j);
    }
    return b;
  }
};

// the least a CTA can ask for so that no more than per_sm fit an SM
constexpr int least_smem(int per_sm) { return 228 * 1024 / (per_sm + 1) - 1024 + 128; }

// CTAs of clusters of this size that can be resident at once where shared memory leaves room for `per_sm` (1 or 2) on an SM: a
// cluster lives inside one GPC, and GPCs differ in size, from one chip to the next too.  Asked once per device.
static __global__ void room_kernel() {}
inline int cluster_room(int device, int cluster, int per_sm) {
  static std::atomic<int> known[64][3][2];
  if (device < 0 || device >= 64) return 0;
  if (cluster == 1) return per_sm * sm_count(device);
  std::atomic<int>& k = known[device][cluster == 2 ? 0 : (cluster == 4 ? 1 : 2)][per_sm - 1];
  int n = k.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(per_sm * sm_count(device) / cluster * cluster);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = least_smem(per_sm);
    cfg.attrs = attr, cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(room_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, room_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      clusters = 0;
    }
    n = clusters > 0 ? clusters * cluster : -1;
    k.store(n, std::memory_order_relaxed);
  }
  return n;
}

// Shared memory to ask for, so that no SM gets more CTAs than it has to, where all of them can be resident at once or two to an
// SM: CTAs are put on as few SMs as hold them, and some then work two or three to an SM beside idle ones (D = 128, 8 heads x 512:
// 61 us instead of 39; single CTAs, D = 64, 6 x 8 x 333: 72 instead of 53).  The launch attribute that asks for clusters to be
// spread changes nothing.  The price: two such calls on two streams do not share an SM either (D = 64, 2 heads x 1024, alone 43 ->
// 29 us, two at a time 47 -> 56; 8 heads x 512 29 -> 22 and 34 -> 37), and a successor that is launched early finds no room before
// the CTAs of this grid end.
// Clusters do not fill every GPC, so how many fit is asked of the device: one cluster more than that would wait for a whole round (16
// clusters of 8 where 15 fit, 512 queries x 2 heads on 4000 keys, D = 64: 105 us; as it is 73, without the request 74).
inline int spread_smem(int need, long long ctas, int cluster, int device) {
  for (int per_sm = 1; per_sm <= 2; ++per_sm)
    if (ctas <= cluster_room(device, cluster, per_sm)) {
      const int least = least_smem(per_sm);
      return need > least ? need : least;
    }
  return need;
}

}  // namespace simt
}  // namespace ttattn
