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
// shared-memory loads (eight per sixteen FMAs); ncu: FMA pipe 58 % busy, 2.7 warps per scheduler, the rest latency.  The mask of
// a tile comes through shared memory (MaskTile); one that is the same for all rows (MaskRow), and the bytes of a boolean one where
// there is room for them (D = 64), as part of the K tile's copies, so that no barrier and no wait is spent on them.
// Measured, us, elements loaded into registers -> now (all masks through MaskTile): 6 x 8 heads x 333, D = 64, padding 55.1 -> 53.6
// (57.8), boolean 60.4 -> 55.9 (61.4), additive 60.3 -> 57.6 (59.3); 2 x 16/4 heads x 1100, D = 64, padding 295 -> 280 (301), boolean
// 347 -> 295 (325); 4 x 8 heads x 500, D = 128, padding 159 -> 121 (126), boolean 184 -> 128 (132), additive 172 -> 125 (128).
//
// Few query tiles leave most SMs idle for the time of the longest walk over the keys, 4 us (D = 64) or 8 us per key tile.
// The key tiles are then divided among the CTAs of a cluster (SPLIT); their unnormalised O, maxima and sums meet in
// distributed shared memory and every CTA writes a share of the rows.  3 heads x 890 D128 causal: 116 -> 44 us; 2 x 3
// heads x 2221 D64 causal: 295 -> 156.
#include <algorithm>

#include "simt_tile.cuh"

namespace ttattn {
namespace {

using namespace simt;
enum MaskForm { kNoMask, kRowMask, kBoolMask, kAddMask };  // kRowMask: the same for all rows, of either kind
constexpr int kThreads = 128, TY = kThreads / 16, R = TS / TY;

// TIGHT: only K is padded, so that two CTAs of D = 128 fit an SM, to the byte (4 x 8 heads x 500: 136 -> 119 us).  Where there are too
// few for two the padded tiles are the faster (8 heads x 512, divided: 39 us instead of 42).  Three CTAs of D = 64 fit either way: tight
// tiles are the faster but for walks of one or two key tiles without a mask (kShortWalk), whose start the kernel's spills weigh on:
// padded and tight, 11 x 32/8 heads x 22 14.7 and 15.2 us, 40 x 8 x 60 16.5 and 17.0, 16 x 12 x 128 27.3 and 27.7; 12 x 4 x 250 29.9 and
// 29.4, 4 x 8 x 500 73.0 and 72.4.
constexpr int kShortWalk = 2;
template <int D, bool TIGHT>
struct Lay {
  static constexpr bool kTight = TIGHT;
  static constexpr Layout Q = kTight ? kSwap : kPad, V = kTight ? kPlain : kPad, P = kTight ? kSwap : kPad;
  static constexpr int kQ = kTight ? TS * D : kTileFloats<D>, kV = kQ, kP = kTight ? TS * TS : kScoreFloats;
  static constexpr bool kApart = D == 64;  // a boolean mask's bytes have a place of their own, for two tiles
  static constexpr int smem_bytes(MaskForm mask) {
    return (kQ + kTileFloats<D> + kV + kP + (kApart && mask == kBoolMask ? 2 * TS * kByteRow : 0)) * static_cast<int>(sizeof(float));
  }
};
static_assert(2 * (Lay<128, true>::smem_bytes(kBoolMask) + 1024) <= 228 * 1024, "two CTAs of D = 128 to an SM");
static_assert(3 * (Lay<64, false>::smem_bytes(kNoMask) + 1024) <= 228 * 1024, "three CTAs of D = 64 to an SM");
static_assert(3 * (Lay<64, true>::smem_bytes(kBoolMask) + 1024) <= 228 * 1024, "three CTAs of D = 64 to an SM");

template <int D, MaskForm MASK, bool SPLIT, bool TIGHT>
__global__ void __launch_bounds__(kThreads, D == 64 ? 3 : 2) fwd_simt_kernel(const FwdArgs a, int cluster) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();  // launched early: everything below reads or writes global memory
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;
  using LY = Lay<D, TIGHT>;
  float* Ks = Qs + LY::kQ;
  float* Vs = Ks + kTileFloats<D>;
  float* Ps = Vs + LY::kV;

  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int n_mt = SPLIT ? gridDim.x / cluster : gridDim.x, rank = SPLIT ? blockIdx.x % cluster : 0;
  const int mt = n_mt - 1 - static_cast<int>(SPLIT ? blockIdx.x / cluster : blockIdx.x);  // under a causal mask the last is longest
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
  const int all_tiles = (kv_end + TS - 1) / TS;
  const int t0 = SPLIT ? all_tiles * rank / cluster : 0, n_tiles = SPLIT ? all_tiles * (rank + 1) / cluster : all_tiles;
  const float c = a.scale * kLog2e;
  const int64_t mask_base = b * a.mask.sb + h * a.mask.sh;

  MaskTile<D, TY, kThreads, LY::P> mask{a.mask, Ps, mask_base, ty, tx, tid};
  const MaskRow<D> mask_row{a.mask, Ks, mask_base, tx, tid};
  float* mine = mask.mine();  // where this thread's scores go
  // a tile's mask comes with its K, or (ASIDE) later, in a group of copies of its own, to where the scores go
  constexpr bool APART = MASK == kBoolMask && LY::kApart, ASIDE = MASK == kAddMask || (MASK == kBoolMask && !APART);
  auto apart = [&](int t) { return Ps + LY::kP + (t & 1) * TS * kByteRow; };
  auto mask_with_k = [&](int t) {
    if constexpr (MASK == kRowMask) mask_row.stage(t, kv_len);
    if constexpr (APART) mask.template stage_bytes<kByteRow>(apart(t), row0, a.Lq, t * TS, kv_len);
  };
  auto mask_aside = [&](int col0) {
    if constexpr (MASK == kBoolMask)
      mask.template stage_bytes<mask.LD>(Ps, row0, a.Lq, col0, kv_len);
    else  // (stage_added by itself: 124 bytes of spills instead of 40; 8 x 16 heads x 512, D = 64 256 us instead of 233)
      mask.stage(row0, a.Lq, col0, kv_len);
  };
  if (n_tiles > t0) {
    load_tile<D, kThreads, LY::Q>(Qs, q, a.qs.s, row0, a.Lq, tid);
    load_tile<D, kThreads>(Ks, k, a.ks.s, t0 * TS, kv_len, tid);
    mask_with_k(t0);
    copies_commit();
    if constexpr (ASIDE) {
      mask_aside(t0 * TS);
      copies_commit();
    }
    load_tile<D, kThreads, LY::V>(Vs, v, a.vs.s, t0 * TS, kv_len, tid);
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

  for (int t = t0; t < n_tiles; ++t) {
    const int col0 = t * TS;
    copies_wait<ASIDE ? 2 : 1>();  // Q and K of this tile; the mask and V may still be on their way
    __syncthreads();
    float s[R][4];
    product_nt<D, TY, LY::Q>(Qs, Ks, ty, tx, s);
    if (MASK == kBoolMask && ASIDE) copies_wait<1>();
    __syncthreads();  // K of this tile has been read
    if (t + 1 < n_tiles) {
      load_tile<D, kThreads>(Ks, k, a.ks.s, col0 + TS, kv_len, tid);
      mask_with_k(t + 1);
    }
    copies_commit();
    uint32_t hidden = 0;
    if constexpr (MASK == kRowMask) {
      mask_row.apply(t, c, s);
    } else if constexpr (MASK == kAddMask) {
      copies_wait<2>();  // (of a thread's own)
    } else if constexpr (APART) {
      mask.template apply<kByteRow>(apart(t), row0, col0, c, s);
    } else if constexpr (MASK == kBoolMask) {
      hidden = mask.bits(row0, col0);
      __syncthreads();
    }
    const bool edge = col0 + TS > kv_len || (a.causal && col0 + TS - 1 > row0 + shift);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = row0 + ty + TY * i;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (MASK == kNoMask || ASIDE) s[i][j] *= c;  // (the others have been)
        if constexpr (MASK == kAddMask) s[i][j] = fmaf(mine[mask.at(i, j)], kLog2e, s[i][j]);
        if (MASK == kBoolMask && ASIDE && (hidden >> (4 * i + j) & 1)) s[i][j] = -INFINITY;
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
        mine[mask.at(i, j)] = p;
      }
    }
    copies_wait<1>();  // V of this tile
    __syncthreads();
    product_nn<D, TY, LY::P, LY::V>(Ps, Vs, ty, tx, acc);
    __syncthreads();  // V and P have been read
    if constexpr (ASIDE) {
      if (t + 1 < n_tiles) mask_aside(col0 + TS);
      copies_commit();
    }
    if (t + 1 < n_tiles) load_tile<D, kThreads, LY::V>(Vs, v, a.vs.s, col0 + TS, kv_len, tid);
    copies_commit();
  }

  float* o = reinterpret_cast<float*>(a.o) + b * a.os.b + h * a.os.h;
  float* lse = a.lse ? a.lse + (static_cast<int64_t>(b) * a.Hq + h) * a.Lq : nullptr;
  if constexpr (SPLIT) {
    // this CTA's share, where the others find it: O over the Q tile, (maximum, sum) over the scores
    constexpr int kMost = 8;  // CTAs per cluster
    float* share = Ps;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float ls = l[i];
#pragma unroll
      for (int of = 8; of >= 1; of >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, of);
      const int r = ty + TY * i;
#pragma unroll
      for (int j = 0; j < D / 64; ++j)
        *reinterpret_cast<float4*>(Qs + r * D + tx * 4 + j * 64) = make_float4(acc[i][2 * j].x, acc[i][2 * j].y, acc[i][2 * j + 1].x, acc[i][2 * j + 1].y);
      if (tx == 0) share[2 * r] = m[i], share[2 * r + 1] = ls;
    }
    ptx::cluster_sync();
    const int rows = TS / cluster, first = rank * rows;
    float* weight = Ps + 2 * TS;  // [row][CTA]
    if (tid < rows) {
      float2 st[kMost];
      float mx = -INFINITY, ls = 0.f;
#pragma unroll
      for (int r = 0; r < kMost; ++r)
        if (r < cluster) {
          st[r] = ptx::ld_cluster_f2(ptx::map_rank(ptx::smem_u32(share + 2 * (first + tid)), r));
          mx = fmaxf(mx, st[r].x);
        }
      const float ref = mx == -INFINITY ? 0.f : mx;
#pragma unroll
      for (int r = 0; r < kMost; ++r)
        if (r < cluster) ls += st[r].y * exp2f(st[r].x - ref);
      const float inv = ls > 0.f ? 1.f / ls : 0.f;
#pragma unroll
      for (int r = 0; r < kMost; ++r)
        if (r < cluster) weight[tid * kMost + r] = exp2f(st[r].x - ref) * inv;
      if (lse && row0 + first + tid < a.Lq) lse[row0 + first + tid] = ls > 0.f ? (mx + log2f(ls)) * kLn2 : -INFINITY;
    }
    __syncthreads();
    for (int e = tid; e < rows * (D / 4); e += kThreads) {
      const int r = e / (D / 4), d = e % (D / 4) * 4;
      if (row0 + first + r >= a.Lq) break;
      float4 x[kMost], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int p = 0; p < kMost; ++p)
        if (p < cluster) x[p] = ptx::ld_cluster_f4(ptx::map_rank(ptx::smem_u32(Qs + (first + r) * D + d), p));
#pragma unroll
      for (int p = 0; p < kMost; ++p)
        if (p < cluster) {
          const float w = weight[r * kMost + p];
          sum.x = fmaf(x[p].x, w, sum.x), sum.y = fmaf(x[p].y, w, sum.y), sum.z = fmaf(x[p].z, w, sum.z), sum.w = fmaf(x[p].w, w, sum.w);
        }
      *reinterpret_cast<float4*>(o + static_cast<int64_t>(row0 + first + r) * a.os.s + d) = sum;
    }
    ptx::cluster_sync();  // no CTA leaves while another still reads its share
  } else {
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
      if (lse && tx == 0) lse[row] = ls > 0.f ? (m[i] + log2f(ls)) * kLn2 : -INFINITY;
    }
  }
}

// CTAs per cluster, by how many query tiles there are (under a causal mask half: their walks are half as long on average),
// and only while the longest walk gets shorter.  From a sweep of 24 shapes with 1, 2, 4 and 8 (within 5 % of the best of them for each).
// D = 64, where three CTAs share an SM, is divided further than D = 128, where one already takes most of what the SM gives.
// Measured, us, undivided -> chosen: D64, 64 rows on 4000 keys, 2 heads 330 -> 54; 1024, 4 heads 88 -> 52; causal 2048, 8
// heads 304 -> 164; 128, 2 x 4 heads 15.1 -> 11.6.  D128, 512, 8 heads 69 -> 40; causal 2048, 8 heads 382 -> 320.  One step
// further in these: -, 50, 174, 11.6, 45, 336.
int split_of(const FwdArgs& a, int D) {
  const int n_mt = (a.Lq + TS - 1) / TS, tiles = (a.Skv + TS - 1) / TS;
  const bool triangle = a.causal == TT_ATTN_CAUSAL_TOP_LEFT;
  const int longest = triangle ? std::min(tiles, n_mt) : tiles;
  const long long ctas = static_cast<long long>(n_mt) * a.Hq * a.B, full = triangle ? (ctas + 1) / 2 : ctas;
  const int at_most[3] = {D == 64 ? 256 : 128, D == 64 ? 128 : 32, D == 64 ? 18 : 16};  // for 2, 4, 8 CTAs
  int cluster = 1;
  auto walk = [&](int c) { return (longest + c - 1) / c; };
  for (int i = 0; i < 3 && full <= at_most[i] && walk(2 * cluster) < walk(cluster); ++i) cluster *= 2;
  return cluster;
}

template <int D, MaskForm MASK>
cudaError_t launch_t(const FwdArgs& a, int device, cudaStream_t stream) {
  const int cluster = split_of(a, D);
  constexpr bool SPLIT_TIGHT = D == 64;
  auto kern = cluster > 1 ? fwd_simt_kernel<D, MASK, true, SPLIT_TIGHT> : fwd_simt_kernel<D, MASK, false, true>;
  int smem = cluster > 1 ? Lay<D, SPLIT_TIGHT>::smem_bytes(MASK) : Lay<D, true>::smem_bytes(MASK);
  if constexpr (D == 64 && MASK == kNoMask)
    if (cluster == 1 && a.Skv <= kShortWalk * TS) kern = fwd_simt_kernel<D, MASK, false, false>, smem = Lay<D, false>::smem_bytes(MASK);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  const long long ctas = static_cast<long long>((a.Lq + TS - 1) / TS) * cluster * a.Hq * a.B;
  return launch_early(kern, dim3((a.Lq + TS - 1) / TS * cluster, a.Hq, a.B), dim3(kThreads),
                      spread_smem(smem, ctas, cluster, device), stream, cluster, a, cluster);
}

template <int D>
cudaError_t launch_d(const FwdArgs& a, int device, cudaStream_t stream) {
  if (!a.mask.ptr) return launch_t<D, kNoMask>(a, device, stream);
  if (a.mask.sl == 0) return launch_t<D, kRowMask>(a, device, stream);
  return a.mask.kind == TT_ATTN_MASK_BOOL ? launch_t<D, kBoolMask>(a, device, stream) : launch_t<D, kAddMask>(a, device, stream);
}

}  // namespace

cudaError_t launch_fwd_simt(int dtype, int D, const FwdArgs& a, int device, cudaStream_t stream) {
  if (dtype != TT_ATTN_F32) return cudaErrorInvalidValue;
  if (D == 64) return launch_d<64>(a, device, stream);
  if (D == 128) return launch_d<128>(a, device, stream);
  return cudaErrorInvalidValue;
}

}  // namespace ttattn
