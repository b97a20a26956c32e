// Attention backward on CUDA cores with fp32 arithmetic for Float32 tensors, and the delta pre-pass of both backwards.
//
// The reference's FuncSDPAttention::backward is unimplemented
// (src/Function/FuncNNLayer.h:267); its gradient is defined by the chain
// linear -> mul -> add -> softmax -> linear (src/Function/FuncNNLayer.h:20-34,
// src/Function/FuncElemWise.h:77-87,113-123, src/Operation/OpNNLayerCpu.h:78-109):
//   dV = P^T dO          dP = dO V^T
//   dS = P o (dP - rowsum(P o dP)) * scale,   rowsum(P o dP) = rowsum(dO o O) = delta
//   dQ = dS K            dK = dS^T Q
// P is recomputed from Q, K and the forward's log-sum-exp, so no [L,S] matrix is
// ever stored, but for small ones in fp32.  The kernels:
//   bwd_delta_kernel   delta[b,h,i] = sum_d dO[i,d] * O[i,d]           (fp32 workspace)
//   bwd_simt_kernel    CTAs of two kinds in one launch, so that a small problem pays one launch and both kinds fill
//                      the machine together:
//     key CTAs    one per 64-key tile: loop over the query tiles (and over the query heads of the group),
//                 accumulate dK, dV in registers -> deterministic, no atomics
//     query CTAs  one per 64-query tile: loop over the key tiles, accumulate dQ
//   bwd_dq_kernel      instead of the query CTAs where there is room for dS and work enough for one more launch (bwd_ds_bytes): the
//                      key CTAs leave their dS tiles (STORE), and dQ is one product of them and K
// Bound by the FMA pipes: five products, or seven where dQ recomputes P and dS (atomics, whose order is not
// deterministic, would do without dS in memory).  16 x TY threads per tile (simt_tile.cuh): 8 rows per thread for D = 64; 4 for D = 128, where 8
// would need more accumulators than there are registers.  B4 H16 S2048 D64 causal: 4986 -> 2807 us (24 -> 43 TFLOP/s),
// B2 H4 S128 D64: 63 -> 23 us; ncu: FMA pipe 63 % busy.  Where tiles are few, or a key tile's walk is long because several
// query heads share it, the CTAs of a cluster share a walk (SPLIT, split_of) and add their accumulators in rank order.
#include <algorithm>

#include "simt_tile.cuh"

namespace ttattn {
namespace {

using namespace simt;
constexpr int kThreads = 256;  // of the delta kernel

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

template <int D>
struct Cfg {
  static constexpr int TY = D == 64 ? 8 : 16, NT = 16 * TY, R = TS / TY;
  static constexpr int kSmemBytes = (4 * kTileFloats<D> + 2 * kScoreFloats + 2 * TS) * static_cast<int>(sizeof(float));
};

// The (query tile, key tile) pair in shared memory: P into Ps (if KEYS) and dS into dSs, [query][key] both.  With a mask, Ps
// holds its elements before (see MaskTile).  `shift` is the causal alignment (key j participates iff j <= i + shift).
template <int D, bool MASK, bool KEYS, bool STORE>
__device__ __forceinline__ void tile_p_ds(const BwdArgs& a, const float* Qs, const float* Ks, const float* Vs,
                                          const float* dOs, const float* lse2_s, const float* delta_s, float* Ps,
                                          float* dSs, float* ds_out, int row0, int col0, int kv_len, int shift,
                                          MaskTile<D, Cfg<D>::TY, Cfg<D>::NT, kPad>& mask) {
  constexpr int TY = Cfg<D>::TY, R = Cfg<D>::R;
  const float c = a.scale * kLog2e;
  const int ty = mask.ty, tx = mask.tx;
  uint32_t hidden = 0;
  if constexpr (MASK) {
    if (!mask.additive()) {
      hidden = mask.bits(row0, col0);
      if (KEYS) __syncthreads();  // (P goes to the same place)
    }
  }
  float p[R][4], dp[R][4];
  product_nt<D, TY>(Qs, Ks, ty, tx, p);
  const bool edge = row0 + TS > a.Lq || col0 + TS > kv_len || (a.causal && col0 + TS - 1 > row0 + shift);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = ty + TY * i, row = row0 + r;
    const float lse2 = lse2_s[r];  // lse * log2(e); +inf for a row without any participating key, whose P is 0
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float x = fmaf(p[i][j], c, -lse2);
      if constexpr (MASK) {
        if (mask.additive()) x = fmaf(Ps[r * LP + tx + 16 * j], kLog2e, x);
        if (hidden >> (4 * i + j) & 1) x = -INFINITY;
      }
      p[i][j] = exp2f(x);
      const int col = col0 + tx + 16 * j;
      if (edge && !(row < a.Lq && col < kv_len && (!a.causal || col <= row + shift))) p[i][j] = 0.f;
      if constexpr (KEYS) Ps[r * LP + tx + 16 * j] = p[i][j];
    }
  }
  product_nt<D, TY>(dOs, Vs, ty, tx, dp);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = ty + TY * i;
    const float dl = delta_s[r];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float ds = p[i][j] * (dp[i][j] - dl) * a.scale;
      dSs[r * LP + tx + 16 * j] = ds;
      if (STORE) ds_out[r * TS + tx + 16 * j] = ds;
    }
  }
}

// where dS of (query tile, key tile) waits for the dQ pass: [query][key] of a tile, tiles of a head by query tile
__device__ __forceinline__ float* ds_tile(const BwdArgs& a, int b, int h, int qt, int kt) {
  const int64_t q_tiles = (a.Lq + TS - 1) / TS, k_tiles = (a.Skv + TS - 1) / TS;
  return a.ds + (((static_cast<int64_t>(b) * a.Hq + h) * q_tiles + qt) * k_tiles + kt) * (TS * TS);
}

// lse (times log2 e, +inf where -inf) and delta of the 64 queries from row0 on
__device__ __forceinline__ void load_vectors(const BwdArgs& a, float* lse2_s, float* delta_s, int64_t base, int row0, int tid) {
  if (tid < TS) {
    const bool in = row0 + tid < a.Lq;
    const float l = in ? a.lse[base + row0 + tid] : 0.f;
    lse2_s[tid] = l == -INFINITY ? INFINITY : l * kLog2e;
    delta_s[tid] = in ? a.delta[base + row0 + tid] : 0.f;
  }
}

// SPLIT: the sum of the cluster's accumulators, in rank order; each CTA stores a share of the rows.  `share`: this CTA's own
// accumulator in shared memory, [TS][D], where the others find it (complete before the cluster barrier ahead of this).
template <int D, int R>
__device__ __forceinline__ void keep_rows(float* share, int step, int first, int tx, const float2 (&acc)[R][D / 32]) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < D / 64; ++c)
      *reinterpret_cast<float4*>(share + (first + step * i) * D + tx * 4 + c * 64) =
          make_float4(acc[i][2 * c].x, acc[i][2 * c].y, acc[i][2 * c + 1].x, acc[i][2 * c + 1].y);
}
template <int D, int NT>
__device__ __forceinline__ void sum_rows(float* out, const Str3& st, int row0, int n_rows, const float* share, int rank, int cluster,
                                         int tid) {
  constexpr int kMost = 8;
  const int rows = TS / cluster, first = rank * rows;
  for (int e = tid; e < rows * (D / 4); e += NT) {
    const int r = first + e / (D / 4), d = e % (D / 4) * 4;
    if (row0 + r >= n_rows) break;
    const uint32_t at = ptx::smem_u32(share + r * D + d);
    float4 x[kMost], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int p = 0; p < kMost; ++p)
      if (p < cluster) x[p] = ptx::ld_cluster_f4(ptx::map_rank(at, p));
#pragma unroll
    for (int p = 0; p < kMost; ++p)
      if (p < cluster) sum.x += x[p].x, sum.y += x[p].y, sum.z += x[p].z, sum.w += x[p].w;
    *reinterpret_cast<float4*>(out + static_cast<int64_t>(row0 + r) * st.s + d) = sum;
  }
}

template <int D, int R>
__device__ __forceinline__ void store_rows(float* out, const Str3& st, int row0, int step, int n_rows, int first, int tx,
                                           const float2 (&acc)[R][D / 32]) {
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = row0 + first + step * i;
    if (row >= n_rows) continue;
#pragma unroll
    for (int c = 0; c < D / 64; ++c)
      *reinterpret_cast<float4*>(out + static_cast<int64_t>(row) * st.s + tx * 4 + c * 64) =
          make_float4(acc[i][2 * c].x, acc[i][2 * c].y, acc[i][2 * c + 1].x, acc[i][2 * c + 1].y);
  }
}

template <int D, bool MASK, bool SPLIT, bool STORE>
__global__ void __launch_bounds__(Cfg<D>::NT, D == 64 ? 2 : 1) bwd_simt_kernel(const BwdArgs a, int key_tiles, int key_ctas,
                                                                               int cluster) {
  using C = Cfg<D>;
  constexpr int TY = C::TY, R = C::R, NT = C::NT;
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;
  float* dOs = Qs + kTileFloats<D>;
  float* Ks = dOs + kTileFloats<D>;
  float* Vs = Ks + kTileFloats<D>;
  float* Ps = Vs + kTileFloats<D>;
  float* dSs = Ps + kScoreFloats;
  float* lse2_s = dSs + kScoreFloats;
  float* delta_s = lse2_s + TS;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  if (STORE) ptx::grid_dep_launch();  // (the dQ pass waits for this grid)
  // SPLIT: the CTAs of a cluster share the walk of one tile
  const int item = SPLIT ? blockIdx.x / cluster : blockIdx.x, rank = SPLIT ? blockIdx.x % cluster : 0;
  const bool keys = STORE || item < key_ctas;
  const int group = a.Hq / a.Hkv;
  MaskTile<D, TY, NT, kPad> mask{a.mask, Ps, 0, ty, tx, tid};

  float2 acc0[R][D / 32], acc1[R][D / 32];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < D / 32; ++j) acc0[i][j] = make_float2(0.f, 0.f), acc1[i][j] = make_float2(0.f, 0.f);

  const float* qb = reinterpret_cast<const float*>(a.q);
  const float* kb = reinterpret_cast<const float*>(a.k);
  const float* vb = reinterpret_cast<const float*>(a.v);
  const float* gb = reinterpret_cast<const float*>(a.d_o);
  const int q_tiles = (a.Lq + TS - 1) / TS;

  if (keys) {
    // ------------------------------------------------------------- dK, dV of a key tile --
    const int nt = item % key_tiles, bh = item / key_tiles;  // (the first key tile is seen by most queries)
    const int hk = bh % a.Hkv, b = bh / a.Hkv, col0 = nt * TS;
    int kv_len = a.Skv;
    if (a.kv_lens) {
      int l = a.kv_lens[b];
      kv_len = l < 0 ? 0 : (l < a.Skv ? l : a.Skv);
    }
    const int shift = causal_shift(a.causal, kv_len, a.Lq);
    // first query tile with a row i such that col0 <= i + shift
    const int qt0 = a.causal ? (col0 - shift > 0 ? (col0 - shift) / TS : 0) : 0;
    load_tile<D, NT>(Ks, kb + b * a.ks.b + hk * a.ks.h, a.ks.s, col0, a.Skv, tid);
    load_tile<D, NT>(Vs, vb + b * a.vs.b + hk * a.vs.h, a.vs.s, col0, a.Skv, tid);
    bool first = true;
    // the walk: query tiles qt0.. of the group's heads, one after the other; this CTA's share of it
    const int per_head = col0 < kv_len && qt0 < q_tiles ? q_tiles - qt0 : 0, steps = per_head * group;
    int n = SPLIT ? steps * rank / cluster : 0;
    const int n_end = SPLIT ? steps * (rank + 1) / cluster : steps;
    while (n < n_end) {
      const int g = n / per_head, h = hk * group + g, end = min(n_end, (g + 1) * per_head);
      const float* q = qb + b * a.qs.b + h * a.qs.h;
      const float* dO = gb + b * a.dos.b + h * a.dos.h;
      const int64_t base = (static_cast<int64_t>(b) * a.Hq + h) * a.Lq;
      for (; n < end; ++n) {
        const int row0 = (qt0 + n - g * per_head) * TS;
        __syncthreads();  // the tiles of the step before have been read
        load_tile<D, NT>(Qs, q, a.qs.s, row0, a.Lq, tid);
        load_tile<D, NT>(dOs, dO, a.dos.s, row0, a.Lq, tid);
        mask.base = b * a.mask.sb + h * a.mask.sh;
        if constexpr (MASK) mask.stage(row0, a.Lq, col0, kv_len);
        copies_commit();
        if (first) ptx::grid_dep_wait();  // launched early behind the delta pre-pass
        first = false;
        load_vectors(a, lse2_s, delta_s, base, row0, tid);
        copies_wait<0>();
        __syncthreads();
        float* ds_out = STORE ? ds_tile(a, b, h, row0 / TS, nt) : nullptr;
        tile_p_ds<D, MASK, true, STORE>(a, Qs, Ks, Vs, dOs, lse2_s, delta_s, Ps, dSs, ds_out, row0, col0, kv_len, shift, mask);
        __syncthreads();
        product_tn<D, TY>(Ps, dOs, ty, tx, acc0);
        product_tn<D, TY>(dSs, Qs, ty, tx, acc1);
      }
    }
    copies_commit();
    copies_wait<0>();
    if (first) ptx::grid_dep_wait();
    if constexpr (SPLIT) {
      __syncthreads();  // the tiles have been read
      keep_rows<D, R>(Qs, 1, ty * R, tx, acc0);
      keep_rows<D, R>(Ks, 1, ty * R, tx, acc1);
      ptx::cluster_sync();
      if (a.dv) sum_rows<D, NT>(reinterpret_cast<float*>(a.dv) + b * a.dvs.b + hk * a.dvs.h, a.dvs, col0, a.Skv, Qs, rank, cluster, tid);
      if (a.dk) sum_rows<D, NT>(reinterpret_cast<float*>(a.dk) + b * a.dks.b + hk * a.dks.h, a.dks, col0, a.Skv, Ks, rank, cluster, tid);
      ptx::cluster_sync();  // no CTA leaves while another still reads its share
    } else {
      if (a.dv)
        store_rows<D, R>(reinterpret_cast<float*>(a.dv) + b * a.dvs.b + hk * a.dvs.h, a.dvs, col0, 1, a.Skv, ty * R, tx, acc0);
      if (a.dk)
        store_rows<D, R>(reinterpret_cast<float*>(a.dk) + b * a.dks.b + hk * a.dks.h, a.dks, col0, 1, a.Skv, ty * R, tx, acc1);
    }
  } else {
    // ----------------------------------------------------------------- dQ of a query tile --
    const int x = item - key_ctas;
    const int mt = q_tiles - 1 - x % q_tiles, bh = x / q_tiles;  // (under a causal mask the last tile is longest)
    const int h = bh % a.Hq, b = bh / a.Hq, hk = h / group, row0 = mt * TS;
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
    const float* k = kb + b * a.ks.b + hk * a.ks.h;
    const float* v = vb + b * a.vs.b + hk * a.vs.h;
    load_tile<D, NT>(Qs, qb + b * a.qs.b + h * a.qs.h, a.qs.s, row0, a.Lq, tid);
    load_tile<D, NT>(dOs, gb + b * a.dos.b + h * a.dos.h, a.dos.s, row0, a.Lq, tid);
    if (n_tiles > t0) {
      load_tile<D, NT>(Ks, k, a.ks.s, t0 * TS, a.Skv, tid);
      load_tile<D, NT>(Vs, v, a.vs.s, t0 * TS, a.Skv, tid);
    }
    mask.base = b * a.mask.sb + h * a.mask.sh;
    if (MASK && n_tiles > t0) mask.stage(row0, a.Lq, t0 * TS, kv_len);
    copies_commit();
    ptx::grid_dep_wait();  // launched early behind the delta pre-pass
    load_vectors(a, lse2_s, delta_s, (static_cast<int64_t>(b) * a.Hq + h) * a.Lq, row0, tid);
    for (int t = t0; t < n_tiles; ++t) {
      const int col0 = t * TS;
      copies_wait<0>();
      __syncthreads();
      tile_p_ds<D, MASK, false, false>(a, Qs, Ks, Vs, dOs, lse2_s, delta_s, Ps, dSs, nullptr, row0, col0, kv_len, shift, mask);
      __syncthreads();
      if (t + 1 < n_tiles) {
        load_tile<D, NT>(Vs, v, a.vs.s, col0 + TS, a.Skv, tid);
        if constexpr (MASK) mask.stage(row0, a.Lq, col0 + TS, kv_len);
      }
      product_nn<D, TY>(dSs, Ks, ty, tx, acc0);
      __syncthreads();
      if (t + 1 < n_tiles) load_tile<D, NT>(Ks, k, a.ks.s, col0 + TS, a.Skv, tid);
      copies_commit();
    }
    copies_wait<0>();
    float* dq = reinterpret_cast<float*>(a.dq) + b * a.dqs.b + h * a.dqs.h;
    if constexpr (SPLIT) {
      __syncthreads();
      keep_rows<D, R>(Ks, TY, ty, tx, acc0);
      ptx::cluster_sync();
      sum_rows<D, NT>(dq, a.dqs, row0, a.Lq, Ks, rank, cluster, tid);
      ptx::cluster_sync();
    } else {
      store_rows<D, R>(dq, a.dqs, row0, TY, a.Lq, ty, tx, acc0);
    }
  }
}

// dQ of a 64-query tile from the dS tiles that the key CTAs have left: dQ += dS K over the key tiles that the queries see.
// One product a step, the next step's tiles copied in under it; SPLIT as above.
template <int D, bool SPLIT>
__global__ void __launch_bounds__(128, D == 64 ? 3 : 2) bwd_dq_kernel(const BwdArgs a, int cluster) {
  constexpr int TY = 8, R = TS / TY, NT = 128;
  extern __shared__ __align__(16) float sm[];
  float* Ss = sm;                   // dS, two stages
  float* Ks = sm + 2 * TS * TS;     // K, two stages
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int item = SPLIT ? blockIdx.x / cluster : blockIdx.x, rank = SPLIT ? blockIdx.x % cluster : 0;
  const int q_tiles = (a.Lq + TS - 1) / TS;
  const int mt = q_tiles - 1 - item % q_tiles, bh = item / q_tiles;  // (under a causal mask the last tile is longest)
  const int h = bh % a.Hq, b = bh / a.Hq, hk = h / (a.Hq / a.Hkv), row0 = mt * TS;
  ptx::grid_dep_launch();
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
  const float* k = reinterpret_cast<const float*>(a.k) + b * a.ks.b + hk * a.ks.h;
  const float* ds = ds_tile(a, b, h, mt, 0);
  auto load_k = [&](int t) { load_tile<D, NT, kPlain>(Ks + (t & 1) * TS * D, k, a.ks.s, t * TS, a.Skv, tid); };
  auto load_ds = [&](int t) {
    load_tile<TS, NT, kSwapHalves>(Ss + (t & 1) * TS * TS, ds + static_cast<int64_t>(t) * TS * TS, TS, 0, TS, tid);
  };
  float2 acc[R][D / 32];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < D / 32; ++j) acc[i][j] = make_float2(0.f, 0.f);
  if (n_tiles > t0) load_k(t0);
  ptx::grid_dep_wait();  // launched early behind the key CTAs, which leave dS
  if (n_tiles > t0) load_ds(t0);
  copies_commit();
  for (int t = t0; t < n_tiles; ++t) {
    if (t + 1 < n_tiles) load_k(t + 1), load_ds(t + 1);
    copies_commit();
    copies_wait<1>();
    __syncthreads();
    // (a tile's sum by itself: chains of 64 terms, not of all keys)
    float2 part[R][D / 32];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < D / 32; ++j) part[i][j] = make_float2(0.f, 0.f);
    product_nn<D, TY, kSwap, kPlain>(Ss + (t & 1) * TS * TS, Ks + (t & 1) * TS * D, ty, tx, part);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < D / 32; ++j) acc[i][j] = ptx::add2(acc[i][j], part[i][j]);
    __syncthreads();  // the stage may be filled again
  }
  float* dq = reinterpret_cast<float*>(a.dq) + b * a.dqs.b + h * a.dqs.h;
  if constexpr (SPLIT) {
    keep_rows<D, R>(Ks, TY, ty, tx, acc);
    ptx::cluster_sync();
    sum_rows<D, NT>(dq, a.dqs, row0, a.Lq, Ks, rank, cluster, tid);
    ptx::cluster_sync();
  } else {
    store_rows<D, R>(dq, a.dqs, row0, TY, a.Lq, ty, tx, acc);
  }
}

template <typename T, int D>
cudaError_t launch_delta_t(const BwdArgs& a, cudaStream_t stream) {
  const int64_t rows = static_cast<int64_t>(a.B) * a.Hq * a.Lq;
  if (rows > 0x7fffffffll) return cudaErrorInvalidValue;
  return launch_early(bwd_delta_kernel<T, D>, dim3(static_cast<unsigned>((rows * (D * sizeof(T) / 16) + kThreads - 1) / kThreads)), dim3(kThreads), 0,
                      stream, 1, a);
}

// CTAs per cluster: with few tiles the longest walk sets the time, with many the SMs' throughput, and every CTA has its fixed
// part.  The cheapest of 1, 2, 4 and 8 by a model fitted to 22 shapes (what it picks is on average within 3 % of the best):
// a step 12.6 us (D = 64) or 14.7 in a CTA alone, 5 or 13.8 of an SM's throughput (a query tile's three products count three
// quarters), 6 or 14.6 us of an SM per CTA.  Measured, us, undivided -> chosen: causal, 2 query heads on one, 3000, D64 1224
// -> 246; 8/2 heads x 700, D128 634 -> 165; 4 heads x 1500, D64 327 -> 152; 2 x 4 heads x 128, D64 20.5 -> 15.2; undivided
// 4 x 16 heads x 512, D64 237 (two shares: 250).
int split_of(const BwdArgs& a, int D, bool store) {
  const double step = D == 64 ? 12.6 : 14.7, busy = D == 64 ? 5.0 : 13.8, fixed = D == 64 ? 6.0 : 14.6, tail = D == 64 ? 0.62 : 0.23;
  const double kt = (a.Skv + TS - 1) / TS, qt = (a.Lq + TS - 1) / TS, heads = static_cast<double>(a.B) * a.Hq;
  const int longest = a.Hq / a.Hkv * static_cast<int>(qt);
  const double seen = a.causal == TT_ATTN_CAUSAL_TOP_LEFT ? 0.5 * (kt + 1) / kt : 1.0;  // of all (query, key) tiles
  const double work = (store ? 1.0 : 1.75) * heads * kt * qt * seen * busy;
  const double ctas = (store ? 0.0 : heads * qt) + static_cast<double>(a.B) * a.Hkv * kt;
  int best = 1;
  double best_us = 1e30;
  for (int c = 1, lg = 0; c <= 8; c *= 2, ++lg) {
    const double walk = (longest + c - 1) / c * step;
    // (clusters of 8 do not fill every GPC)
    const double us = std::max(walk + 1.5 * lg, (work + ctas * c * fixed) / kSms * (c == 8 ? 1.1 : 1.0) + tail * walk);
    if (us < best_us) best = c, best_us = us;
  }
  return best;
}

template <int D>
constexpr int kDqSmemBytes = 2 * (TS * TS + TS * D) * static_cast<int>(sizeof(float));

template <int D>
cudaError_t launch_dq(const BwdArgs& a, int device, cudaStream_t stream) {
  const long long q_tiles = (a.Lq + TS - 1) / TS, items = q_tiles * a.Hq * a.B;
  const int k_tiles = (a.Skv + TS - 1) / TS;
  int cluster = 1;  // (steps of 2 us (D = 64) or 4 in a CTA alone)
  while (cluster < 8 && items * cluster * 2 <= (D == 64 ? 2 : 1) * kSms && k_tiles >= 4 * cluster) cluster *= 2;
  auto kern = cluster > 1 ? bwd_dq_kernel<D, true> : bwd_dq_kernel<D, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  if (items * cluster > 0x7fffffffll) return cudaErrorInvalidValue;
  return launch_early(kern, dim3(static_cast<unsigned>(items * cluster)), dim3(128), spread_smem(kDqSmemBytes<D>, items * cluster, cluster, device),
                      stream, cluster, a, cluster);
}

template <int D, bool MASK>
cudaError_t launch_t(const BwdArgs& a, int device, cudaStream_t stream) {
  cudaError_t e = launch_delta_t<float, D>(a, stream);
  if (e != cudaSuccess) return e;
  const bool store = a.ds != nullptr;
  const int cluster = split_of(a, D, store);
  auto kern = store ? (cluster > 1 ? bwd_simt_kernel<D, MASK, true, true> : bwd_simt_kernel<D, MASK, false, true>)
                    : (cluster > 1 ? bwd_simt_kernel<D, MASK, true, false> : bwd_simt_kernel<D, MASK, false, false>);
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  const long long key_tiles = (a.Skv + TS - 1) / TS, q_tiles = (a.Lq + TS - 1) / TS;
  const long long key_ctas = a.dk || a.dv ? key_tiles * a.Hkv * a.B : 0, q_ctas = a.dq && !store ? q_tiles * a.Hq * a.B : 0;
  if ((key_ctas + q_ctas) * cluster > 0x7fffffffll) return cudaErrorInvalidValue;
  e = launch_early(kern, dim3(static_cast<unsigned>((key_ctas + q_ctas) * cluster)), dim3(Cfg<D>::NT),
                   spread_smem(Cfg<D>::kSmemBytes, (key_ctas + q_ctas) * cluster, cluster, device), stream, cluster, a,
                   static_cast<int>(key_tiles), static_cast<int>(key_ctas), cluster);
  return e == cudaSuccess && store ? launch_dq<D>(a, device, stream) : e;
}

}  // namespace

cudaError_t launch_bwd_delta(int dtype, int D, const BwdArgs& a, cudaStream_t stream) {
  if (dtype == TT_ATTN_F32) return D == 64 ? launch_delta_t<float, 64>(a, stream) : launch_delta_t<float, 128>(a, stream);
  if (dtype == TT_ATTN_F16)
    return D == 64 ? launch_delta_t<__half, 64>(a, stream) : launch_delta_t<__half, 128>(a, stream);
  return D == 64 ? launch_delta_t<__nv_bfloat16, 64>(a, stream) : launch_delta_t<__nv_bfloat16, 128>(a, stream);
}

// Where there is room for dS, dQ is one product more instead of three, by a kernel of its own: 16 KB of scratch for a pair of 64-row
// tiles, written and read once.  Up to 192 MB of it; and from as many pairs on as make up for
// the launch (which the dQ CTAs, beside the key CTAs in one grid, do without).  Measured, us, three products -> one: D64, 4 x 8
// heads x 500 190 -> 160, 6 x 8 x 333 with a mask 186 -> 134; D128, 4 x 8 x 500 424 -> 295, 3 x 890 causal 113 -> 95, 14 x 6/3 x 162 causal 120 -> 110;
// below the line 2 x 2 x 232, D64 17 -> 23, 15 x 4 x 45, D128 18 -> 23.
size_t bwd_ds_bytes(int B, int Hq, int Hkv, int Lq, int Skv, int D) {
  if (B <= 0 || Hq <= 0 || Lq <= 0 || Skv <= 0) return 0;
  const double pairs = static_cast<double>(B) * Hq * ((Lq + TS - 1) / TS) * ((Skv + TS - 1) / TS), bytes = pairs * TS * TS * sizeof(float);
  return bytes <= 192e6 && pairs >= (D == 64 ? 600 : 300) ? static_cast<size_t>(bytes) : 0;
}

cudaError_t launch_bwd_simt(int dtype, int D, const BwdArgs& a, int device, cudaStream_t stream) {
  if (dtype != TT_ATTN_F32) return cudaErrorInvalidValue;
  const bool mask = a.mask.ptr != nullptr;
  if (D == 64) return mask ? launch_t<64, true>(a, device, stream) : launch_t<64, false>(a, device, stream);
  if (D == 128) return mask ? launch_t<128, true>(a, device, stream) : launch_t<128, false>(a, device, stream);
  return cudaErrorInvalidValue;
}

}  // namespace ttattn
