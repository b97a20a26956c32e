// Prefill forward for fp16 / bf16 on sm_100a tensor cores.
//
// Replaces the score-materialising composition of FuncSDPAttention::forward
// (reference: src/Function/FuncNNLayer.h:231-266) by one fused kernel that never
// writes the [L,S] score matrix to HBM.
//
// Persistent kernel, one CTA per SM, all 512 TMEM columns.  A work item is a pair
// of 128-row query blocks of one (batch, kv head), numbered query tile by query
// tile with the heads of the group together: where heads share keys, both blocks
// see the same ones, and short sequences fill both.  CTAs draw items from a global
// counter, heads in order and, within a head, the longest (latest causal) pair
// first, so that the CTAs running at any moment share few heads' K/V in L2 and
// the last items to be drawn are the shortest.
// KEYS: where latency counts, i.e. with so few items that the longest walk over the key tiles sets the time, an item
// is ONE query block and the two halves of the CTA take its key tiles alternately (even, odd): half the steps.  The two
// accumulators are in the same TMEM lanes, so both warpgroups read both, each for half of the columns, and only maxima
// and sums cross through shared memory.  With fewer blocks than SMs the key tiles are divided further among the CTAs of
// a cluster, one item per cluster; their unnormalised O, maxima and sums meet in distributed shared memory at the end and
// every CTA of the cluster writes a share of the rows.
//   warp 8   producer : draws items and publishes them to the other warps; TMA
//                       tiled loads (128-byte swizzle, one copy per CTA) of the item's
//                       two Q tiles and of each K and V tile into a 2-stage ring.
//                       It runs ahead: the next item's Q and first K/V tiles are
//                       requested while the current item is still being computed.
//   warp 9   issuer   : one thread issues tcgen05.mma; S_t = Q_t.K^T accumulates in
//                       TMEM columns [t*128, t*128+128), O_t += P_t.V in columns
//                       [256 + t*D, 256 + (t+1)*D).  The two tiles are interleaved
//                       (PV_0 QK_0' PV_1 QK_1') so that the tensor pipe computes for
//                       one tile while the other tile's warpgroup is in its softmax.
//   warps 0-3 / 4-7   : softmax warpgroup of tile 0 / 1.  Thread r owns query row r
//                       (= TMEM lane r): it reads the whole 128-column S row with
//                       tcgen05.ld, so the row max and row sum need no cross-thread
//                       reduction in this layout; exponentials run as packed fp32
//                       pairs (fma.rn.f32x2 + ex2); P is written as packed 16-bit
//                       pairs over the S columns with tcgen05.st; O is rescaled
//                       only when the row max grew by more than 2^8; the same
//                       warpgroup writes O and LSE while the issuer already starts
//                       the next item's first QK.
// P never leaves TMEM: the second MMA takes its A operand from TMEM.
// Every mbarrier wait is bounded; an expired wait sets the status word and makes
// the CTA unwind.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"

namespace ttattn {
namespace {

constexpr int BM = 128;      // rows of one query tile (= TMEM lanes)
constexpr int QT = 2;        // query tiles per item
constexpr int BN = 128;      // keys per tile
constexpr int NSTAGE = 2;    // K/V ring depth
constexpr int kThreads = 384;  // 2 softmax warpgroups + 1 warpgroup holding the producer and issuer warps
constexpr int kTmemCols = 512;
constexpr int kItemConsumers = 1 + QT * BM;  // issuer thread + every softmax thread
#ifndef TT_FWD_TAIL_WAVES
#define TT_FWD_TAIL_WAVES 2
#endif
constexpr int kTailWaves = TT_FWD_TAIL_WAVES;  // waves of work items at the end that are ordered longest first across heads

// One work item, decoded once by the producer.
struct Item {
  int b, hk, h[QT], row0[QT];  // head and first row of the two blocks
  int kv_len, shift;           // key j participates iff j <= i + shift (causal)
  int j0, nt[QT];              // first key tile, and how many each half walks from there (KEYS: in turn)
  int n_max;                   // the longer walk; -1: no more items
  int mask;                    // whether the mask has to be looked at
};

struct __align__(16) SmemCtl {
  uint64_t q_full[QT], q_empty[QT];  // per query tile: tile 0 of the next item is loaded while tile 1 still works
  uint64_t k_full[NSTAGE], k_empty[NSTAGE], v_full[NSTAGE], v_empty[NSTAGE];
  uint64_t s_full[QT], p_full[QT], o_full[QT];
  uint64_t item_full[2], item_empty[2];
  Item item[2];
  uint32_t tmem_base;
  int abort_flag;
};

template <int D>
constexpr int tile_bytes() {
  return BM * D * 2;
}
constexpr int kStageBytes = BM * 128;  // per warpgroup: one 64-column block of an O tile
// a second buffer for mask rows (see MaskRows), where there is room for it
template <int D, int GEN>
constexpr int kMaskExtra = D == 64 && GEN == 2 ? QT * kStageBytes : 0;
template <int D, int GEN>
constexpr int smem_bytes() {
  return (QT + 2 * NSTAGE) * tile_bytes<D>() + QT * kStageBytes + kMaskExtra<D, GEN> + 1024 /*alignment slack*/ + 512 /*SmemCtl*/;
}

// GEN: 1: the variant for a causal triangle that is not top-left aligned, 2: that and a mask; the fast variant (0) compiles
// all of that out.
// KEYS: `per_head` items (query blocks) per (batch, kv head), `rank` of `cluster` shares of the key tiles; else pairs.
template <int GEN, bool KEYS>
__device__ __forceinline__ Item decode_item(const FwdArgs& a, int w, int per_head, int rank = 0, int cluster = 1) {
  Item it;
  // Heads in order, the longest (latest causal) pair of a head first: the CTAs running at any moment share few
  // heads' K/V in L2.  Only the last items are ordered differently: over the final kTailWaves waves the pairs of
  // the remaining heads are taken longest first ACROSS those heads, so that what is drawn last is short and the
  // CTAs finish together (in head order the last head's longest pair, an eighth of a CTA's whole share of
  // 128 heads of 4096 rows, would be drawn when most CTAs are nearly done).  Those heads' K/V together fit L2.
  const int n_heads = a.B * a.Hkv, group = a.Hq / a.Hkv;
  int tail_heads = (kTailWaves * static_cast<int>(gridDim.x) + per_head - 1) / per_head;
  if (tail_heads > n_heads) tail_heads = n_heads;
  const int w0 = (n_heads - tail_heads) * per_head;
  int bh, mp;
  if (w < w0) {
    bh = w / per_head;
    mp = per_head - 1 - (w - bh * per_head);
  } else {
    const int x = w - w0, rank_in = x / tail_heads;
    bh = n_heads - tail_heads + (x - rank_in * tail_heads);
    mp = per_head - 1 - rank_in;
  }
  it.b = bh / a.Hkv;
  it.hk = bh - it.b * a.Hkv;
  int kv_len = a.Skv;
  if (a.kv_lens) {
    int l = a.kv_lens[it.b];
    kv_len = l < 0 ? 0 : (l < a.Skv ? l : a.Skv);
  }
  it.kv_len = kv_len;
  it.mask = GEN == 2 && !(a.mask_pure && a.mask_pure[it.b]);
  it.shift = GEN ? causal_shift(a.causal, kv_len, a.Lq) : 0;  // key j participates iff j <= i + shift
  const int x = KEYS ? mp : mp * QT, qt0 = x / group, qt1 = KEYS ? qt0 : (x + 1) / group;
  it.h[0] = it.hk * group + x - qt0 * group, it.h[1] = KEYS ? it.h[0] : it.hk * group + x + 1 - qt1 * group;
  it.row0[0] = qt0 * BM, it.row0[1] = qt1 * BM;
  // key tiles that a block sees (0 for one wholly beyond Lq)
  auto tiles = [&](int row0) {
    int e = kv_len;
    if (a.causal) {
      int c = row0 + BM + it.shift;
      if (GEN) c = c > 0 ? c : 0;
      if (c < e) e = c;
    }
    return row0 < a.Lq ? (e + BN - 1) / BN : 0;
  };
  it.j0 = 0;
  if constexpr (KEYS) {
    int n = tiles(it.row0[0]);
    if (cluster > 1) {
      it.j0 = n * rank / cluster;
      n = n * (rank + 1) / cluster - it.j0;
    }
    it.nt[0] = (n + 1) / 2, it.nt[1] = n / 2;
  } else {
    it.nt[0] = tiles(it.row0[0]), it.nt[1] = tiles(it.row0[1]);
  }
  it.n_max = it.nt[0] > it.nt[1] ? it.nt[0] : it.nt[1];
  return it;
}

// The mask of one warp's 32 query rows, 128 bytes of a row at a time (128 keys of a boolean mask, 64 of a 16-bit or 32 of
// an fp32 one) through 4 KB of shared memory.  A thread owns a whole row of scores, but 32 rows read by 32 threads are 32
// cache lines per load, and rows of an odd length are not even aligned: 13 times the time without a mask.  The warp copies
// row by row instead, the aligned 16-byte pieces that hold the segment, eight lanes a row (cp.async: nothing waits for them
// until the scores have arrived; the pieces of a row are rotated by its number against bank conflicts), and each thread
// reads its row back and shifts it into place; a ninth piece, of a row that is not aligned, waits in registers.  A mask that
// is the same for all rows is one row.  B5 H32/16 L1620 D64 with an additive bf16 mask: 2193 -> 394 us, without a
// mask 170.
template <typename T>
struct MaskRows {
  const uint8_t* base;  // the warp's first row
  int rows;             // rows that exist

  static __device__ __forceinline__ const uint8_t* down16(const uint8_t* p) {
    return reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(p) & ~uintptr_t(15));
  }

  __device__ __forceinline__ void stage(const FwdArgs& a, int esz, int lane, int at, uint32_t buf, uint4& tail) const {
    const int64_t pitch = a.mask.sl * esz;
    const int left = a.Skv * esz - at;  // bytes of a row that exist from there on
    const int piece = lane & 7, r0 = lane >> 3;
    const uint8_t* p = base + r0 * pitch + at;
    const uint32_t dst = buf + r0 * 128;
    if (rows >= 32 && left >= 128 + 15) {
#pragma unroll
      for (int i = 0; i < 32; i += 4, p += 4 * pitch)
        ptx::cp_async16(dst + i * 128 + (((piece + r0 + i) & 7) << 4), down16(p) + piece * 16, 16);
    } else {
      const uint8_t* any = down16(reinterpret_cast<const uint8_t*>(a.mask.ptr));  // valid and aligned, for copies of nothing
#pragma unroll 1
      for (int i = 0; i < 32; i += 4, p += 4 * pitch) {
        const uint8_t* src = down16(p) + piece * 16;
        const int n = r0 + i < rows ? static_cast<int>(p + left - src) : 0;
        if (pitch != 0 || r0 == 0) ptx::cp_async16(dst + i * 128 + (((piece + r0 + i) & 7) << 4), n > 0 ? src : any, n > 16 ? 16 : (n > 0 ? n : 0));
        if (pitch == 0) break;
      }
    }
    if (!a.mask.wide) {
      const uint8_t* mine = base + lane * pitch + at;
      const uint8_t* src = down16(mine) + 128;
      tail = make_uint4(0, 0, 0, 0);
      if ((lane < rows || pitch == 0) && src < mine + left && down16(mine) != mine) tail = *reinterpret_cast<const uint4*>(src);
    }
  }

  // this lane's segment, 8 words at a time: use(first word, words)
  template <typename F>
  __device__ __forceinline__ void read(const FwdArgs& a, int esz, int lane, uint32_t buf, const uint4& tail, F use) const {
    ptx::cp_async_wait();
    __syncwarp();
    const int64_t pitch = a.mask.sl * esz;
    uint32_t r = pitch == 0 ? 0 : lane;
    asm volatile("" : "+r"(r));  // (the addresses are computed here, not kept in registers)
    const uint32_t row = buf + r * 128;
    auto piece = [&](int i) { return ptx::ld_shared4(row + (((i + r) & 7) << 4)); };
    uint4 p[4];  // the pieces of a chunk and the next
    p[0] = piece(0), p[1] = piece(1);
    if (a.mask.wide) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 x = p[(c & 1) * 2], y = p[(c & 1) * 2 + 1];
        if (c < 3) p[(~c & 1) * 2] = piece(2 * c + 2), p[(~c & 1) * 2 + 1] = piece(2 * c + 3);
        const uint32_t w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        use(c * 8, w);
      }
    } else {
      const uint32_t mis = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(base) + lane * pitch) & 15;
      const bool by2 = mis & 8, by1 = mis & 4;
      const uint32_t sh = (mis & 3) * 8;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 x = p[(c & 1) * 2], y = p[(c & 1) * 2 + 1];
        if (c < 3) p[(~c & 1) * 2] = piece(2 * c + 2), p[(~c & 1) * 2 + 1] = piece(2 * c + 3);
        const uint4 z = c < 3 ? p[(~c & 1) * 2] : tail;
        uint32_t w[12] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w, z.x, z.y, z.z, z.w};
#pragma unroll
        for (int i = 0; i < 10; ++i) w[i] = by2 ? w[i + 2] : w[i];
#pragma unroll
        for (int i = 0; i < 9; ++i) w[i] = by1 ? w[i + 1] : w[i];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], sh);
        use(c * 8, w);
      }
    }
    __syncwarp();  // the buffer may be filled again
  }
};

// s[e] <- c * s[e] + mask for the keys of 8 words, the first of them key e0 of the tile
template <typename T, int KIND>
__device__ __forceinline__ void add_mask(uint32_t (&s)[BN], int e0, const uint32_t* w, float c) {
  const float2 c2 = make_float2(c, c);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if constexpr (KIND == TT_ATTN_MASK_BOOL) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = e0 + k * 4 + i;
        s[e] = (w[k] >> (8 * i)) & 0xffu ? __float_as_uint(__uint_as_float(s[e]) * c) : 0xff800000u;
      }
    } else if constexpr (KIND == TT_ATTN_MASK_ADD_F32) {
      s[e0 + k] = __float_as_uint(fmaf(__uint_as_float(s[e0 + k]), c, __uint_as_float(w[k])));
    } else {
      const int e = e0 + k * 2;
      const T* t = reinterpret_cast<const T*>(&w[k]);
      const float2 m = std::is_same<T, __nv_bfloat16>::value
                           ? make_float2(__uint_as_float(__byte_perm(w[k], 0, 0x1044)), __uint_as_float(w[k] & 0xffff0000u))
                           : make_float2(to_f32<T>(t[0]), to_f32<T>(t[1]));
      const float2 x = ptx::fma2(make_float2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), c2, m);
      s[e] = __float_as_uint(x.x), s[e + 1] = __float_as_uint(x.y);
    }
  }
}

// The 128 rows of an item over the CS CTAs of the cluster.  `stats`: (reference, sum) of every row, `xo`: its
// unnormalised O, at the same place in the shared memory of each CTA.  D / 4 lanes read a row (a warp's reads are whole
// 512-byte rows), 8 vectors are in flight per thread; this CTA's own share is read as ordinary shared memory.
template <int D, bool BF16, int CS>
__device__ __forceinline__ void combine_rows(const FwdArgs& a, const Item& it, int rank, int warp, int lane, uint32_t stats,
                                             uint32_t xo) {
  using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
  constexpr int kPer = 128 / D;  // rows that a warp reads at a time
  constexpr int kBatch = 8 / CS, kRows = BM / CS;
  const int c4 = lane % (D / 4);
  uint32_t pstats[CS], pxo[CS];  // this CTA's first, then the others in turn
#pragma unroll
  for (int r = 1; r < CS; ++r) pstats[r] = ptx::map_rank(stats, (rank + r) % CS), pxo[r] = ptx::map_rank(xo, (rank + r) % CS);
  pstats[0] = stats, pxo[0] = xo;
#pragma unroll 1
  for (int i = warp * kPer + lane / (D / 4); i < kRows; i += 8 * kPer * kBatch) {
    float4 x[kBatch][CS];
    float2 ml[kBatch][CS];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int rr = rank * kRows + i + u * 8 * kPer;
#pragma unroll
      for (int r = 0; r < CS; ++r) {
        const uint32_t sa = pstats[r] + rr * 8, xa = pxo[r] + rr * D * 4 + ((c4 ^ rr) & (D / 4 - 1)) * 16;
        ml[u][r] = r == 0 ? ptx::ld_shared_f2(sa) : ptx::ld_cluster_f2(sa);
        x[u][r] = r == 0 ? ptx::ld_shared_f4(xa) : ptx::ld_cluster_f4(xa);
      }
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int row = it.row0[0] + rank * kRows + i + u * 8 * kPer, head = it.h[0];
      float m = -INFINITY, l = 0.f;
#pragma unroll
      for (int r = 0; r < CS; ++r) m = fmaxf(m, ml[u][r].x);
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int r = 0; r < CS; ++r) {
        if (ml[u][r].x == -INFINITY) continue;  // (a CTA without key tiles for the row left no O)
        const float w = ptx::ex2(ml[u][r].x - m);
        l = fmaf(ml[u][r].y, w, l);
        v.x = fmaf(x[u][r].x, w, v.x), v.y = fmaf(x[u][r].y, w, v.y), v.z = fmaf(x[u][r].z, w, v.z), v.w = fmaf(x[u][r].w, w, v.w);
      }
      if (row >= a.Lq) continue;
      const float inv = l > 0.f ? 1.f / l : 0.f;
      *reinterpret_cast<uint2*>(reinterpret_cast<T*>(a.o) + it.b * a.os.b + head * a.os.h + static_cast<int64_t>(row) * a.os.s +
                                c4 * 4) = make_uint2(pack2<BF16>(v.x * inv, v.y * inv), pack2<BF16>(v.z * inv, v.w * inv));
      if (a.lse && c4 == 0)
        a.lse[(static_cast<int64_t>(it.b) * a.Hq + head) * a.Lq + row] = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
    }
  }
}

template <int D, bool BF16, int GEN, bool KEYS>
__global__ void __launch_bounds__(kThreads, 1)
    fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                  const FwdArgs a, int cluster) {
  extern __shared__ uint8_t smem_raw[];
  // 128-byte-swizzled tiles must start on a 1024-byte boundary.
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int TB = tile_bytes<D>();
  uint8_t* sQ = smem;                    // QT tiles
  uint8_t* sK = smem + QT * TB;          // NSTAGE tiles
  uint8_t* sV = sK + NSTAGE * TB;        // NSTAGE tiles
  uint8_t* sO = sV + NSTAGE * TB;        // QT staging blocks for the O stores
  SmemCtl* ctl = reinterpret_cast<SmemCtl*>(sO + QT * kStageBytes + kMaskExtra<D, GEN>);
  volatile int* abort_flag = &ctl->abort_flag;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int n_blocks = (a.Lq + BM - 1) / BM * (a.Hq / a.Hkv), per_head = KEYS ? n_blocks : (n_blocks + QT - 1) / QT;
  const int n_items = per_head * a.Hkv * a.B;
  const int rank = KEYS && cluster > 1 ? static_cast<int>(ptx::cluster_rank()) : 0;
  auto item_of = [&](int w) { return KEYS ? decode_item<GEN, true>(a, w, per_head, rank, cluster) : decode_item<GEN, false>(a, w, per_head); };

  constexpr int HALVES = D / 64;  // 64-element (128-byte) column blocks per row
  constexpr int HALF_BYTES = BM * 128;

  if (warp == 8 && lane == 0) {
#pragma unroll
    for (int t = 0; t < QT; ++t) {
      ptx::mbar_init(&ctl->q_full[t], 1);
      ptx::mbar_init(&ctl->q_empty[t], 1);
    }
#pragma unroll
    for (int i = 0; i < NSTAGE; ++i) {
      ptx::mbar_init(&ctl->k_full[i], 1);
      ptx::mbar_init(&ctl->k_empty[i], 1);
      ptx::mbar_init(&ctl->v_full[i], 1);
      ptx::mbar_init(&ctl->v_empty[i], 1);
    }
#pragma unroll
    for (int t = 0; t < QT; ++t) {
      ptx::mbar_init(&ctl->s_full[t], 1);
      ptx::mbar_init(&ctl->p_full[t], BM);
      ptx::mbar_init(&ctl->o_full[t], 1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&ctl->item_full[i], 1);
      ptx::mbar_init(&ctl->item_empty[i], kItemConsumers);
    }
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::tma_prefetch_desc(&tmQ);
    ptx::tma_prefetch_desc(&tmK);
    ptx::tma_prefetch_desc(&tmV);
    ptx::tma_prefetch_desc(&tmO);
  }
  if (warp == 9) {
    ptx::tmem_alloc(&ctl->tmem_base, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  ptx::grid_dep_launch();  // (the next kernel may come up: this grid has its TMEM)
  ptx::grid_dep_wait();    // (launched early: everything below reads or writes global memory)

  // Register budget: the softmax warpgroups hold a whole 128-column S row per
  // thread; the producer / issuer warpgroup needs little.
  if (warp >= 8) {
    // (D = 128: 224 + 224 + 56 registers per thread over the three warpgroups; D = 64, whose issuing loop
    // carries the look-ahead at item boundaries, and KEYS: 216 + 216 + 72.  Both add up to the 168 x 384 registers
    // the CTA was launched with, so the increase below can always be served.)
    ptx::setmaxnreg_dec<D == 128 && !KEYS ? 56 : 72>();
    if (warp == 8) {
      // ---------------------------------------------------------- producer --
      if (lane == 0) {
        uint32_t g = 0;             // K/V tiles requested so far (ring position)
        uint32_t qc0 = 0, qc1 = 0;  // items whose Q tile 0 / 1 was requested so far
        for (uint32_t i = 0;; ++i) {
          // the first item is the CTA's own number; the counter, where one is needed, hands out the rest
          int w;
          if (KEYS && cluster > 1)
            w = i == 0 ? static_cast<int>(blockIdx.x) / cluster : -1;
          else
            w = i == 0 ? static_cast<int>(blockIdx.x) : (a.sched ? static_cast<int>(gridDim.x) + atomicAdd(a.sched, 1) : -1);
          if (w >= n_items) w = -1;
          const int slot = i & 1;
          Item it{};
          it.n_max = -1;
          if (w >= 0) it = item_of(w);
          if (!ptx::mbar_wait(&ctl->item_empty[slot], ((i >> 1) & 1) ^ 1, abort_flag)) break;
          ctl->item[slot] = it;
          ptx::mbar_arrive(&ctl->item_full[slot]);
          if (w < 0) break;
          if (it.n_max == 0) continue;
          bool ok = true;
          // a Q tile is loaded only if it has key tiles to walk; tile 0 goes first and, with the first K tile,
          // ahead of tile 1: the issuer starts tile 0 of this item while tile 1 of the previous one still works
          auto load_q = [&](int t, uint32_t& qc) {
            if ((t == 0 ? it.nt[0] : it.nt[1]) == 0) return true;
            if (!ptx::mbar_wait(&ctl->q_empty[t], (qc & 1) ^ 1, abort_flag)) return false;
            ptx::mbar_arrive_expect_tx(&ctl->q_full[t], TB);
#pragma unroll
            for (int hf = 0; hf < HALVES; ++hf)
              ptx::tma_load_4d(sQ + t * TB + hf * HALF_BYTES, &tmQ, &ctl->q_full[t], hf * 64,
                              t == 0 ? it.row0[0] : it.row0[1], t == 0 ? it.h[0] : it.h[1], it.b);
            ++qc;
            return true;
          };
          if (!(ok = load_q(0, qc0))) break;
          if constexpr (KEYS) {
            // every tile goes to one half only; K a tile ahead of V, as the products consume them
            const int n = it.nt[0] + it.nt[1];
            auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* full, uint64_t* empty, int j) {
              const uint32_t gj = g + j;
              const int st = gj % NSTAGE;
              if (!ptx::mbar_wait(&empty[st], ((gj / NSTAGE) & 1) ^ 1, abort_flag)) return false;
              ptx::mbar_arrive_expect_tx(&full[st], TB);
#pragma unroll
              for (int hf = 0; hf < HALVES; ++hf)
                ptx::tma_load_4d(dst + st * TB + hf * HALF_BYTES, map, &full[st], hf * 64, (it.j0 + j) * BN, it.hk, it.b);
              return true;
            };
            ok = load(sK, &tmK, ctl->k_full, ctl->k_empty, 0);
            for (int j = 0; j < n && ok; ++j) {
              if (j + 1 < n) ok = load(sK, &tmK, ctl->k_full, ctl->k_empty, j + 1);
              if (ok) ok = load(sV, &tmV, ctl->v_full, ctl->v_empty, j);
            }
            if (!ok) break;
            g += n;
          } else {
            for (int j = 0; j < it.n_max; ++j, ++g) {
              const int st = g % NSTAGE;
              const uint32_t ph = (g / NSTAGE) & 1;
              if (!(ok = ptx::mbar_wait(&ctl->k_empty[st], ph ^ 1, abort_flag))) break;
              ptx::mbar_arrive_expect_tx(&ctl->k_full[st], TB);
#pragma unroll
              for (int hf = 0; hf < HALVES; ++hf)
                ptx::tma_load_4d(sK + st * TB + hf * HALF_BYTES, &tmK, &ctl->k_full[st], hf * 64, (it.j0 + j) * BN, it.hk, it.b);
              if (j == 0 && !(ok = load_q(1, qc1))) break;
              if (!(ok = ptx::mbar_wait(&ctl->v_empty[st], ph ^ 1, abort_flag))) break;
              ptx::mbar_arrive_expect_tx(&ctl->v_full[st], TB);
#pragma unroll
              for (int hf = 0; hf < HALVES; ++hf)
                ptx::tma_load_4d(sV + st * TB + hf * HALF_BYTES, &tmV, &ctl->v_full[st], hf * 64, (it.j0 + j) * BN, it.hk, it.b);
            }
          }
          if (!ok) break;
        }
      }
    } else if (warp == 9) {
      // ------------------------------------------------------------ issuer --
      // Order per key tile j:  PV(0,j)  QK(0,j+1)  PV(1,j)  QK(1,j+1).  MMAs of one
      // thread execute in issue order, so QK(t,j+1) overwriting S_t / P_t cannot
      // pass PV(t,j) that still reads P_t, and the first QK of the next item
      // cannot pass the last PV of this one.
      // The whole warp runs the loop (waits included, made uniform by a vote); one elected lane issues.
      {
        const bool leader = ptx::elect_one();
        auto uwait = [&](uint64_t* bar, uint32_t parity) {
          return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag)) != 0;
        };
        // A negative scale is folded into the sign of Q so that the softmax
        // always works with a non-negative multiplier.
        const uint32_t neg = a.scale < 0.f ? (1u << 13) : 0u;
        const uint32_t idesc_qk = ptx::make_idesc_f16(BM, BN, BF16 ? 1 : 0, 0, 0) | neg;
        const uint32_t idesc_pv = ptx::make_idesc_f16(BM, D, BF16 ? 1 : 0, 0, 1);
        // Descriptor words are prepared once; stepping to the next k-slice or ring
        // stage is a single 32-bit add, so that this thread keeps pace with the
        // tensor pipe (one 128x128x16 MMA per 64 cycles).
        constexpr uint32_t kHi = ptx::smem_desc_hi_sw128(1024);
        const uint32_t qlo = ptx::smem_desc_lo(ptx::smem_u32(sQ), 16);
        const uint32_t klo = ptx::smem_desc_lo(ptx::smem_u32(sK), 16);
        const uint32_t vlo = ptx::smem_desc_lo(ptx::smem_u32(sV), HALF_BYTES);

        uint32_t g0 = 0;        // ring position of the item's first key tile
        uint32_t c0 = 0, c1 = 0;  // softmax iterations completed per tile (p_full phases)
        uint32_t qc0 = 0, qc1 = 0;  // items whose Q tile 0 / 1 was used so far (q_full phases)
        bool ok = true;
        bool pre0 = false;      // the first QK of tile 0 of the coming item has been issued already

        auto wait_k = [&](uint32_t g) { return uwait(&ctl->k_full[g % NSTAGE], (g / NSTAGE) & 1); };
        auto issue_qk = [&](int t, uint32_t g) {
          const uint32_t a0 = qlo + (KEYS ? 0 : t * (TB >> 4)), b0 = klo + (g % NSTAGE) * (TB >> 4), d = tmem + t * 128;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            // K-major operands: 64-element halves HALF_BYTES apart, 32 bytes per k-step
            const uint32_t off = ((ks >> 2) * HALF_BYTES + (ks & 3) * 32) >> 4;
            if (leader) ptx::mma_ss2(d, a0 + off, kHi, b0 + off, kHi, idesc_qk, ks > 0 ? 1u : 0u);
          }
          if (leader) ptx::mma_commit(&ctl->s_full[t]);
        };
        auto issue_pv = [&](int t, uint32_t g, bool first) {
          const uint32_t b0 = vlo + (g % NSTAGE) * (TB >> 4), d = tmem + 256 + t * D, a0 = tmem + t * 128;
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks) {
            // V is N(=D)-contiguous: 16 keys per k-step = 2048 bytes; the two
            // 64-wide column blocks of D=128 are HALF_BYTES apart (LBO).
            if (leader) ptx::mma_ts2(d, a0 + ks * 8, b0 + ks * (2048 >> 4), kHi, idesc_pv, (!first || ks > 0) ? 1u : 0u);
          }
        };

        // first QK of tile t of an item whose first key tile sits at ring position g
        auto first_qk = [&](int t, uint32_t& qc, uint32_t g, int nt_t) {
          if (!uwait(&ctl->q_full[t], qc & 1)) return false;
          ++qc;
          if (!wait_k(g)) return false;
          ptx::tc_fence_after();
          issue_qk(t, g);
          if (leader && nt_t == 1) ptx::mma_commit(&ctl->q_empty[t]);  // the only QK of this tile
          return true;
        };
        // non-blocking probe, the same answer in every lane
        auto utest = [&](uint64_t* bar, uint32_t parity) {
          return __all_sync(0xffffffffu, ptx::mbar_test(bar, parity)) != 0;
        };

        for (uint32_t i = 0; ok; ++i) {
          const int slot = i & 1;
          if (!uwait(&ctl->item_full[slot], (i >> 1) & 1)) break;
          const int nt0 = ctl->item[slot].nt[0], nt1 = ctl->item[slot].nt[1], n_max = ctl->item[slot].n_max;
          __syncwarp();  // every lane has read the slot before it is handed back
          if (leader) ptx::mbar_arrive(&ctl->item_empty[slot]);
          if (n_max < 0) break;
          if (n_max == 0) continue;
          auto nt = [&](int t) { return t == 0 ? nt0 : nt1; };

          if constexpr (KEYS) {
            // half t takes the key tiles t, t + 2, ...: tile j of the item at ring position g0 + j, used once; the same
            // order PV(0) QK(0)' PV(1) QK(1)' as below
            const int n = nt0 + nt1;
            auto qk = [&](int t, int j) {
              issue_qk(t, g0 + j);
              if (leader) ptx::mma_commit(&ctl->k_empty[(g0 + j) % NSTAGE]);
              if (leader && j == n - 1) ptx::mma_commit(&ctl->q_empty[0]);
            };
            if (!(ok = uwait(&ctl->q_full[0], qc0 & 1))) break;
            ++qc0;
#pragma unroll
            for (int t = 0; t < QT; ++t) {
              if (t >= n) continue;
              if (!(ok = wait_k(g0 + t))) break;
              ptx::tc_fence_after();
              qk(t, t);
            }
            for (int i2 = 0; i2 < nt0 && ok; ++i2) {
#pragma unroll
              for (int t = 0; t < QT; ++t) {
                const int j = 2 * i2 + t;
                if (j >= n) continue;
                const uint32_t g = g0 + j;
                bool okb = ptx::mbar_wait(&ctl->v_full[g % NSTAGE], (g / NSTAGE) & 1, abort_flag);
                if (j + 2 < n && okb) okb = ptx::mbar_wait(&ctl->k_full[(g + 2) % NSTAGE], ((g + 2) / NSTAGE) & 1, abort_flag);
                if (okb) okb = ptx::mbar_wait(&ctl->p_full[t], ((t == 0 ? c0 : c1) + i2) & 1, abort_flag);
                if (!(ok = __all_sync(0xffffffffu, okb) != 0)) break;
                ptx::tc_fence_after();
                issue_pv(t, g, i2 == 0);
                if (leader && i2 == nt(t) - 1) ptx::mma_commit(&ctl->o_full[t]);
                if (leader) ptx::mma_commit(&ctl->v_empty[g % NSTAGE]);
                if (j + 2 < n) qk(t, j + 2);
              }
            }
            g0 += n;
            c0 += nt0;
            c1 += nt1;
            continue;
          }

          if (nt0 > 0 && !pre0 && !(ok = first_qk(0, qc0, g0, nt0))) break;
          pre0 = false;
          if (nt1 > 0 && !(ok = first_qk(1, qc1, g0, nt1))) break;
          if (leader) ptx::mma_commit(&ctl->k_empty[g0 % NSTAGE]);
          // Tile 0 is done and tile 1 still has key tiles to walk (the causal diagonal): if the next item is
          // known and its Q tile 0 and first K tile have landed, start its tile 0 now, so that warpgroup 0
          // does not sit idle for tile 1's last iteration.  Nothing here blocks.  (S_0 is free: its last P has
          // been consumed in issue order; O_0 is not written before warpgroup 0 delivers the next P, i.e.
          // after its epilogue.)
          auto try_pre0 = [&]() {
            if (pre0 || nt0 == 0) return;
            const int nslot = (i + 1) & 1;
            if (!utest(&ctl->item_full[nslot], ((i + 1) >> 1) & 1)) return;
            const int nt0n = ctl->item[nslot].n_max < 0 ? 0 : ctl->item[nslot].nt[0];
            const uint32_t gn = g0 + n_max;
            if (nt0n <= 0 || !utest(&ctl->q_full[0], qc0 & 1) || !utest(&ctl->k_full[gn % NSTAGE], (gn / NSTAGE) & 1))
              return;
            if (!(ok = first_qk(0, qc0, gn, nt0n))) return;
            pre0 = true;
          };

          for (int j = 0; j < n_max && ok; ++j) {
            const uint32_t g = g0 + j;
            const int last_pv = (j < nt1) ? 1 : 0;
            const int last_qk = (j + 1 < nt1) ? 1 : 0;
#pragma unroll
            for (int t = 0; t < QT; ++t) {
              const bool do_pv = j < nt(t), do_qk = j + 1 < nt(t);
              // all waits first, then the MMAs of this tile back to back; the wait for P comes last: it is
              // the one on the critical path (softmax -> PV -> next QK -> softmax), the tiles are long there
              // (one vote for the three: between them the lanes only poll)
              bool okb = true;
              if (do_pv) okb = ptx::mbar_wait(&ctl->v_full[g % NSTAGE], (g / NSTAGE) & 1, abort_flag);
              if (do_qk && okb) okb = ptx::mbar_wait(&ctl->k_full[(g + 1) % NSTAGE], ((g + 1) / NSTAGE) & 1, abort_flag);
              if (do_pv && okb) okb = ptx::mbar_wait(&ctl->p_full[t], ((t == 0 ? c0 : c1) + j) & 1, abort_flag);
              if (!(ok = __all_sync(0xffffffffu, okb) != 0)) break;
              ptx::tc_fence_after();
              if (do_pv) {
                issue_pv(t, g, j == 0);
                if (leader && j == nt(t) - 1) ptx::mma_commit(&ctl->o_full[t]);
                if (leader && t == last_pv) ptx::mma_commit(&ctl->v_empty[g % NSTAGE]);
              }
              if (do_qk) {
                issue_qk(t, g + 1);
                if (leader && j + 2 == nt(t)) ptx::mma_commit(&ctl->q_empty[t]);  // last QK of this tile: its Q may be replaced
                if (leader && t == last_qk) ptx::mma_commit(&ctl->k_empty[(g + 1) % NSTAGE]);
              }
            }
            if constexpr (D == 64) {
              if (ok && j >= nt0 - 1 && nt1 > nt0) try_pre0();
            }
          }
          g0 += n_max;
          c0 += nt0;
          c1 += nt1;
        }
      }
    }
  } else {
    ptx::setmaxnreg_inc<D == 128 && !KEYS ? 224 : 216>();
    // ------------------------------------------------------------- softmax --
    const int t = warp >> 2;          // query tile of this warpgroup
    const int r_in = tid & (BM - 1);  // row within the tile = TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + t * 128 + lane_addr;
    const uint32_t tO = tmem + 256 + t * D + lane_addr;
    // > 0 so that a masked (-inf) score stays -inf when it is scaled
    const float c = fmaxf(fabsf(a.scale) * kLog2e, 1e-30f), cs = fmaxf(fabsf(a.scale), 1e-30f);
    using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
    uint32_t cnt = 0;  // softmax iterations completed (s_full phase)
    uint32_t ec = 0, e1 = 0;  // items with work completed (o_full phase; KEYS: of tile 0, of tile 1)
    bool ok = true;
    uint32_t s[BN];

    // The warpgroup meets at named barriers in the epilogue, so its threads must
    // leave the loop together: an expired wait is voted on (twice per item) and
    // then every thread of the warpgroup unwinds.
    for (uint32_t i = 0;; ++i) {
      const int slot = i & 1;
      ok = ptx::mbar_wait(&ctl->item_full[slot], (i >> 1) & 1, abort_flag);
      // (KEYS: both warpgroups, which also meet after the walk)
      if (KEYS ? ptx::named_barrier_or(3, QT * BM, !ok) : ptx::named_barrier_or(1 + t, BM, !ok)) break;
      const volatile Item* pub = &ctl->item[slot];
      const int b = pub->b, kv_len = pub->kv_len, shift = pub->shift, j0 = pub->j0, n_max = pub->n_max;
      const int n_t = pub->nt[t], tile_row0 = pub->row0[t], head = pub->h[t];
      const bool use_mask = GEN == 2 && pub->mask;
      if (!KEYS) ptx::mbar_arrive(&ctl->item_empty[slot]);  // (KEYS: read again after the walk, and then handed back)
      if (n_max < 0) break;
      const int row = tile_row0 + r_in;  // global query row of this thread
      T* orow = reinterpret_cast<T*>(a.o) + b * a.os.b + head * a.os.h + static_cast<int64_t>(row) * a.os.s;
      float* lse_row = a.lse ? a.lse + (static_cast<int64_t>(b) * a.Hq + head) * a.Lq + row : nullptr;

      if (KEYS ? cluster == 1 && n_max == 0 : n_t == 0) {
        if (KEYS) ptx::mbar_arrive(&ctl->item_empty[slot]);
        // no participating key (or tile beyond Lq): O = 0, LSE = -inf
        if (row < a.Lq && (!KEYS || t == 0)) {
#pragma unroll
          for (int e = 0; e < D; e += 8) *reinterpret_cast<uint4*>(orow + e) = make_uint4(0, 0, 0, 0);
          if (lse_row) *lse_row = -INFINITY;
        }
        continue;
      }

      // with a mask the scores are scaled when the mask is added, and the rest of the loop multiplies by log2(e)
      const float cm = use_mask ? kLog2e : c;
      const float2 c2 = make_float2(cm, cm);
      MaskRows<T> mk = {};
      const int esz = a.mask.kind == TT_ATTN_MASK_BOOL ? 1 : (a.mask.kind == TT_ATTN_MASK_ADD_F32 ? 4 : 2);
      // segments of the tile alternate between the buffers, of which D = 128 has one
      constexpr int kBufs = kMaskExtra<D, GEN> > 0 ? 2 : 1;
      const uint32_t mbuf = ptx::smem_u32(sO + t * kStageBytes + (warp & 3) * 32 * 128);
      auto buffer = [&](int seg) { return mbuf + seg % kBufs * (QT * kStageBytes); };
      uint4 mtail[kBufs];
      auto stage_mask = [&](int j, int seg) {
        mk.stage(a, esz, lane, (j0 + (KEYS ? 2 * j + t : j)) * BN * esz + seg * 128, buffer(seg), mtail[seg % kBufs]);
      };
      if constexpr (GEN == 2) {
        if (use_mask && n_t > 0) {
          // (through this warp's rows of the staging block of O, out of which the item before may still be stored)
          const int row0 = tile_row0 + (warp & 3) * 32;
          mk.base = reinterpret_cast<const uint8_t*>(a.mask.ptr) + (b * a.mask.sb + head * a.mask.sh + row0 * a.mask.sl) * esz;
          mk.rows = a.mask.sl == 0 ? 1 : a.Lq - row0;
          if (r_in == 0) ptx::bulk_wait_read();
          ptx::named_barrier(1 + t, BM);
          stage_mask(0, 0);
          if (kBufs > 1 && esz > 1) stage_mask(0, 1);
        }
      }

      float m_ref = -INFINITY;  // reference max, in scaled log2 units
      float2 l2 = make_float2(0.f, 0.f);
      for (int j = 0; j < n_t && ok; ++j) {
        ok = ptx::mbar_wait(&ctl->s_full[t], (cnt + j) & 1, abort_flag);
        if (!ok) break;
        ptx::tc_fence_after();
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) ptx::tmem_ld32p(tS + cc * 32, s + cc * 32);
        ptx::tmem_wait_ld();

        const int col0 = (j0 + (KEYS ? 2 * j + t : j)) * BN;
        if constexpr (GEN == 2) {
          if (use_mask) {
            auto read = [&](int seg, auto use) {
              mk.read(a, esz, lane, buffer(seg), mtail[seg % kBufs], use);
              if (seg + kBufs < esz) stage_mask(j, seg + kBufs);
            };
            if (esz == 1) {
              read(0, [&](int k, const uint32_t* w) { add_mask<T, TT_ATTN_MASK_BOOL>(s, k * 4, w, cs); });
            } else if (esz == 2) {
              read(0, [&](int k, const uint32_t* w) { add_mask<T, TT_ATTN_MASK_ADD>(s, k * 2, w, cs); });
              read(1, [&](int k, const uint32_t* w) { add_mask<T, TT_ATTN_MASK_ADD>(s, 64 + k * 2, w, cs); });
            } else {
#pragma unroll
              for (int seg = 0; seg < 4; ++seg)
                read(seg, [&](int k, const uint32_t* w) { add_mask<T, TT_ATTN_MASK_ADD_F32>(s, seg * 32 + k, w, cs); });
            }
            if (j + 1 < n_t) {
              stage_mask(j + 1, 0);
              if (kBufs > 1 && esz > 1) stage_mask(j + 1, 1);
            }
          }
        }
        const bool mask_tile = (col0 + BN > kv_len) || (a.causal && col0 + BN - 1 > tile_row0 + shift);
        if (mask_tile) {
          // Highest valid column of this row within the tile.
          int lim = kv_len - 1 - col0;
          if (a.causal && row + shift - col0 < lim) lim = row + shift - col0;
#pragma unroll
          for (int e = 0; e < BN; ++e)
            if (e > lim) s[e] = 0xff800000u;  // -inf
        }
        // The row maximum is only a reference point for the exponentials, so it is
        // not recomputed for every tile: after the first tile the row keeps its
        // reference as long as the tile's exponentials stay small, which the tile's
        // own row sum shows (all terms are positive: sum <= 2^8 implies every term
        // <= 2^8).  Only when the sum is larger (or not finite) is the maximum of
        // the tile taken, O and the running sum rescaled, and the tile redone.
        bool need_max = (j == 0);
        for (;;) {
          if (need_max) {
            // eight independent 3-input max chains over the 128 columns
            float mx[8];
#pragma unroll
            for (int q = 0; q < 8; ++q)
              mx[q] = ptx::max3(__uint_as_float(s[q]), __uint_as_float(s[q + 8]), -INFINITY);
#pragma unroll
            for (int e = 16; e < BN; e += 16)
#pragma unroll
              for (int q = 0; q < 8; ++q)
                mx[q] = ptx::max3(mx[q], __uint_as_float(s[e + q]), __uint_as_float(s[e + q + 8]));
            const float x_max =
                ptx::max3(ptx::max3(mx[0], mx[1], mx[2]), ptx::max3(mx[3], mx[4], mx[5]), fmaxf(mx[6], mx[7])) * cm;
            if (j == 0) {
              m_ref = x_max;
            } else if (__any_sync(0xffffffffu, x_max > m_ref)) {
              // tcgen05.ld / .st are warp-collective: every lane takes part, lanes
              // whose maximum did not grow with alpha = 1
              const float m_new = fmaxf(m_ref, x_max);
              const float alpha = (GEN && m_new == -INFINITY) ? 1.f : ptx::ex2(m_ref - m_new);
              uint32_t r[32];
#pragma unroll
              for (int cc = 0; cc < D / 32; ++cc) {
                ptx::tmem_ld32(tO + cc * 32, r);
                ptx::tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
                ptx::tmem_st32(tO + cc * 32, r);
              }
              l2.x *= alpha, l2.y *= alpha;
              m_ref = m_new;
            }
          }
          // P = 2^(c*s - m_ref) in packed fp32 pairs; two halves of 64 columns so that
          // the packed 16-bit P of the first half is stored while the second is computed.
          // (general variant) a row that has seen no participating key yet keeps
          // m_ref = -inf; its exponentials are taken against 0 and are all 0
          const float m_use = (GEN && m_ref == -INFINITY) ? 0.f : m_ref;
          const float2 nm2 = make_float2(-m_use, -m_use);
          float2 lt = make_float2(0.f, 0.f);
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t pk[32];
#pragma unroll
            for (int e2 = 0; e2 < 64; e2 += 2) {
              const int e = hf * 64 + e2;
              float2 x = ptx::fma2(make_float2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), c2, nm2);
              // (D = 64, where the exponentials and not the MMAs set the pace: one in sixteen on the FMA pipe)
              const float2 p = make_float2(ptx::ex2(x.x), (D == 64 && (e2 & 15) == 0) ? ptx::ex2_fma(x.y) : ptx::ex2(x.y));
              lt = ptx::add2(lt, p);
              pk[e2 >> 1] = pack2<BF16>(p.x, p.y);
            }
            ptx::tmem_st32(tS + hf * 32, pk);
          }
          const float tile_sum = lt.x + lt.y;
          // redo with a fresh maximum if any row of the warp needs it (tcgen05.ld /
          // .st are warp-collective, so the warp decides together)
          // ... and such a row takes the maximum of every tile until it has one
          const bool redo = !need_max && (!(tile_sum <= 256.f) || (GEN && m_ref == -INFINITY));
          if (!__any_sync(0xffffffffu, redo)) {
            l2 = ptx::add2(l2, lt);
            break;
          }
          need_max = true;
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive(&ctl->p_full[t]);
      }
      cnt += n_t;

      if constexpr (KEYS) {
        // Both halves of the walk: wait for both accumulators (tile 0's phase ec, tile 1's e1), exchange references and
        // sums (over the unused second Q tile), then warpgroup t puts columns [64 t, 64 t + 64) together (D = 64:
        // warpgroup 0 all of them).
        const int nt0 = pub->nt[0], nt1 = pub->nt[1];
        ptx::mbar_arrive(&ctl->item_empty[slot]);
        if (ok && nt0 > 0) ok = ptx::mbar_wait(&ctl->o_full[0], ec & 1, abort_flag);
        if (ok && nt1 > 0) ok = ptx::mbar_wait(&ctl->o_full[1], e1 & 1, abort_flag);
        ec += nt0 > 0, e1 += nt1 > 0;
        float2* stat = reinterpret_cast<float2*>(sQ + TB);
        stat[t * BM + r_in] = make_float2(n_t > 0 ? m_ref : -INFINITY, l2.x + l2.y);
        if (ptx::named_barrier_or(3, QT * BM, !ok)) break;
        ptx::tc_fence_after();
        const float2 sa = stat[r_in], sb = stat[BM + r_in];
        const float m = fmaxf(sa.x, sb.x);
        // (a half without key tiles, or a row that none of its keys takes part in, has reference -inf)
        const float wa = sa.x == -INFINITY ? 0.f : ptx::ex2(sa.x - m), wb = sb.x == -INFINITY ? 0.f : ptx::ex2(sb.x - m);
        const float l = sa.y * wa + sb.y * wb;
        const bool mine = D == 128 || t == 0;
        const int c0 = D == 128 ? t * 64 : 0;
        uint8_t* stage = sO + t * kStageBytes;
        if (mine) {
          if (cluster == 1) {
            if (r_in == 0) ptx::bulk_wait_read();  // previous store out of this block has been read
            ptx::named_barrier(1 + t, BM);
          }
          const float inv = cluster > 1 ? 1.f : (l > 0.f ? 1.f / l : 0.f);
          const float ua = wa * inv, ub = wb * inv;
          const uint32_t ta = tmem + 256 + lane_addr + c0;
#pragma unroll 1
          for (int cc = 0; cc < 2; ++cc) {  // 32 columns at a time
            if (nt0 > 0) ptx::tmem_ld32p(ta + cc * 32, s);
            if (nt1 > 0) ptx::tmem_ld32p(ta + D + cc * 32, s + 32);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              const float x = nt0 > 0 ? __uint_as_float(s[e]) * ua : 0.f;
              s[e] = __float_as_uint(nt1 > 0 ? fmaf(__uint_as_float(s[32 + e]), ub, x) : x);
            }
            if (cluster == 1) {
#pragma unroll
              for (int ch = 0; ch < 4; ++ch) {
                uint4 wv;
                wv.x = pack2<BF16>(__uint_as_float(s[ch * 8 + 0]), __uint_as_float(s[ch * 8 + 1]));
                wv.y = pack2<BF16>(__uint_as_float(s[ch * 8 + 2]), __uint_as_float(s[ch * 8 + 3]));
                wv.z = pack2<BF16>(__uint_as_float(s[ch * 8 + 4]), __uint_as_float(s[ch * 8 + 5]));
                wv.w = pack2<BF16>(__uint_as_float(s[ch * 8 + 6]), __uint_as_float(s[ch * 8 + 7]));
                *reinterpret_cast<uint4*>(stage + r_in * 128 + (((cc * 4 + ch) ^ (r_in & 7)) << 4)) = wv;
              }
            } else {
              // unnormalised O for the other CTAs, over the K / V stages (every MMA of the CTA is complete)
              float* xo = reinterpret_cast<float*>(sK) + r_in * D;
#pragma unroll
              for (int ch = 0; ch < 8; ++ch)  // (16-byte pieces of a row permuted by the row: no bank conflicts)
                *reinterpret_cast<uint4*>(xo + (((c0 >> 2) + cc * 8 + ch) ^ (r_in & (D / 4 - 1))) * 4) =
                    make_uint4(s[ch * 4], s[ch * 4 + 1], s[ch * 4 + 2], s[ch * 4 + 3]);
            }
          }
        }
        ptx::tc_fence_before();
        ptx::named_barrier(3, QT * BM);  // both accumulators and the statistics have been read
        if (cluster > 1) {
          if (t == 0) stat[2 * BM + r_in] = make_float2(m, l);
          break;
        }
        if (mine) {
          ptx::fence_proxy_async_smem();
          ptx::named_barrier(1 + t, BM);
          if (r_in == 0) {
            ptx::tma_store_4d(&tmO, stage, c0, tile_row0, head, b);
            ptx::bulk_commit();
          }
        }
        if (t == 0 && row < a.Lq && lse_row) *lse_row = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
        continue;
      }

      // epilogue: O / l -> global, LSE.  The issuer may already be computing the
      // next item's first S_t; its first PV waits for this warpgroup's next P.
      if (ok) ok = ptx::mbar_wait(&ctl->o_full[t], ec & 1, abort_flag);
      ++ec;
      if (ptx::named_barrier_or(1 + t, BM, !ok)) break;
      ptx::tc_fence_after();
#pragma unroll
      for (int cc = 0; cc < D / 32; ++cc) ptx::tmem_ld32p(tO + cc * 32, s + cc * 32);
      ptx::tmem_wait_ld();
      const float l = l2.x + l2.y;
      const float inv = l > 0.f ? 1.f / l : 0.f;
      // O leaves through shared memory and TMA stores (coalesced; rows beyond Lq
      // are clipped by the tensor map): one 64-column block at a time, written in
      // the 128-byte-swizzled layout the map expects.
      uint8_t* stage = sO + t * kStageBytes;
#pragma unroll
      for (int hf = 0; hf < HALVES; ++hf) {
        if (r_in == 0) ptx::bulk_wait_read();  // previous store out of this block has been read
        ptx::named_barrier(1 + t, BM);
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) {
          const int e = hf * 64 + ch * 8;
          uint4 wv;
          wv.x = pack2<BF16>(__uint_as_float(s[e + 0]) * inv, __uint_as_float(s[e + 1]) * inv);
          wv.y = pack2<BF16>(__uint_as_float(s[e + 2]) * inv, __uint_as_float(s[e + 3]) * inv);
          wv.z = pack2<BF16>(__uint_as_float(s[e + 4]) * inv, __uint_as_float(s[e + 5]) * inv);
          wv.w = pack2<BF16>(__uint_as_float(s[e + 6]) * inv, __uint_as_float(s[e + 7]) * inv);
          *reinterpret_cast<uint4*>(stage + r_in * 128 + ((ch ^ (r_in & 7)) << 4)) = wv;
        }
        ptx::fence_proxy_async_smem();
        ptx::named_barrier(1 + t, BM);
        if (r_in == 0 && ok) {
          ptx::tma_store_4d(&tmO, stage, hf * 64, tile_row0, head, b);
          ptx::bulk_commit();
        }
      }
      if (ok && row < a.Lq && lse_row) *lse_row = l > 0.f ? (m_ref + log2f(l)) * kLn2 : -INFINITY;
    }
    if (r_in == 0) ptx::bulk_wait_all();
  }

  if (KEYS && cluster > 1) {
    __syncwarp();
    ptx::cluster_sync();
    if (warp < 8 && *abort_flag == 0) {
      const Item it = item_of(blockIdx.x / cluster);
      const uint32_t stats = ptx::smem_u32(sQ + TB) + 2 * BM * 8, xo = ptx::smem_u32(sK);
      if (cluster == 2)
        combine_rows<D, BF16, 2>(a, it, rank, warp, lane, stats, xo);
      else if (cluster == 4)
        combine_rows<D, BF16, 4>(a, it, rank, warp, lane, stats, xo);
      else
        combine_rows<D, BF16, 8>(a, it, rank, warp, lane, stats, xo);
    }
    __syncwarp();
    ptx::cluster_sync();  // no CTA leaves while another still reads its shared memory
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
  if (tid == 0 && ctl->abort_flag && a.status) atomicOr(a.status, kStatusWaitExpired);
}

// ------------------------------------------------------------------ host ----
template <int D, bool BF16, int GEN, bool KEYS>
cudaError_t launch_k(const FwdArgs& a, int dtype, int grid, int cluster, cudaStream_t stream) {
  CUtensorMap tq, tk, tv, to;
  if (!make_map(&tq, dtype, a.q, D, a.Lq, a.Hq, a.B, a.qs) || !make_map(&tk, dtype, a.k, D, a.Skv, a.Hkv, a.B, a.ks) ||
      !make_map(&tv, dtype, a.v, D, a.Skv, a.Hkv, a.B, a.vs) || !make_map(&to, dtype, a.o, D, a.Lq, a.Hq, a.B, a.os))
    return cudaErrorInvalidValue;
  auto kern = fwd_tc_kernel<D, BF16, GEN, KEYS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<D, GEN>());
  if (e != cudaSuccess) return e;
  return launch_early(kern, dim3(grid), dim3(kThreads), smem_bytes<D, GEN>(), stream, cluster, tq, tk, tv, to, a, cluster);
}

// CTAs of clusters of this size that can be resident at once, one to an SM (a cluster lives inside one GPC, and GPCs
// differ in size).  Asked once per device.
template <int D, bool BF16, int GEN>
int cluster_slots(int device, int cluster) {
  static std::atomic<int> known[64][3];
  if (device < 0 || device >= 64) return 0;
  std::atomic<int>& k = known[device][cluster == 2 ? 0 : (cluster == 4 ? 1 : 2)];
  int n = k.load(std::memory_order_relaxed);
  if (n == 0) {
    auto kern = fwd_tc_kernel<D, BF16, GEN, true>;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count(device) / cluster * cluster);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_bytes<D, GEN>();
    cfg.attrs = attr, cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<D, GEN>()) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      clusters = 0;
    }
    n = clusters > 0 ? clusters * cluster : -1;
    k.store(n, std::memory_order_relaxed);
  }
  return n;
}

// How the work is divided (see the head of the file): what is expected to take the least time, by a model fitted to a sweep
// of 20 shapes (what it picks is within 2 us of the best of pairs, blocks, and clusters of 2, 4 and 8 for each).  Pairs: 6.5
// us and the longest walk, or an SM's share of all walks, 4.5 us for every item besides its steps.  Single blocks: half the
// steps, a little longer ones, 9 us, and 7 us an item.  A cluster adds 5 us.  Measured, us, pairs -> chosen: 2 x 256 queries
// against 8192 keys, 32/8 heads 117 -> 66; 64 against 4096, 8/2 heads 64 -> 18; 32 against 15000, 8 heads D = 64 186 -> 22;
// causal 1024, 16 heads 20.4 -> 16.1; causal 4096, 8 heads 61 -> 41; causal 8 x 512, 32/8 heads 35 (blocks: 58).
struct Plan {
  bool keys;
  int cluster;
};
template <int D, bool BF16, int GEN>
Plan plan_of(const FwdArgs& a, int device) {
  const int group = a.Hq / a.Hkv, n_qt = (a.Lq + BM - 1) / BM, sms = sm_count(device);
  const long long heads = static_cast<long long>(a.B) * a.Hkv, blocks = heads * group * n_qt, pairs = heads * ((group * n_qt + 1) / 2);
  if (blocks > 8ll * sms) return Plan{false, 1};
  const int n_all = (a.Skv + BN - 1) / BN;
  auto tiles = [&](int qt) {  // key tiles of query tile qt, every cache row taken as valid
    if (!a.causal) return n_all;
    const long long c = (qt + 1ll) * BM + (a.causal == TT_ATTN_CAUSAL_BOTTOM_RIGHT ? a.Skv - a.Lq : 0);
    const long long t = c > 0 ? (c + BN - 1) / BN : 0;
    return t < n_all ? static_cast<int>(t) : n_all;
  };
  constexpr double kPairStep = D == 128 ? 1.65 : 1.35, kKeysStep = D == 128 ? 1.75 : 1.35, kPairItem = 4.5, kKeysItem = 7.0;
  double pair_all = kPairItem * pairs, keys_all = kKeysItem * blocks;
  for (int qt = 0; qt < n_qt; ++qt) {
    const int n = tiles(qt);
    keys_all += kKeysStep * heads * group * ((n + 1) / 2);
    pair_all += kPairStep * heads * 0.5 * group * n;
  }
  const int last = tiles(n_qt - 1);
  auto share = [&](double all, long long items, double one) {  // of an SM; walks of one length come in whole rounds
    return 2.0 + (a.causal ? all / sms : static_cast<double>((items + sms - 1) / sms) * one);
  };
  const double pair_one = 6.5 + kPairStep * last, keys_one = 9.0 + kKeysStep * ((last + 1) / 2);
  const double pair_us = std::max(pair_one, share(pair_all, pairs, kPairItem + kPairStep * last));
  const double keys_us = blocks <= sms ? keys_one
                                       : std::max(keys_one, share(keys_all, blocks, kKeysItem + kKeysStep * ((last + 1) / 2)));
  Plan best{keys_us < pair_us, 1};
  double best_us = std::min(keys_us, pair_us);
  for (int cs = 2; cs <= 8; cs *= 2) {
    if (blocks * cs > sms || blocks * cs > cluster_slots<D, BF16, GEN>(device, cs)) break;
    const double us = 14.0 + kKeysStep * (((last + cs - 1) / cs + 1) / 2);
    if (us < best_us) best = Plan{true, cs}, best_us = us;
  }
  return best;
}

// ahead of the main kernel: the lengths that a padding mask comes to, and the work counter
__global__ void __launch_bounds__(256) lens_kernel(const FwdArgs a, int* sched, int32_t* lens, int32_t* pure) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) *sched = 0;
  masked_lens(a.mask, a.kv_lens, a.Skv, blockIdx.x, lens, pure);
}

template <int D, bool BF16, int GEN>
cudaError_t launch_t(FwdArgs a, int dtype, int device, cudaStream_t stream) {
  const long long n_blocks = (a.Lq + BM - 1ll) / BM * (a.Hq / a.Hkv), heads = static_cast<long long>(a.Hkv) * a.B;
  const Plan p = plan_of<D, BF16, GEN>(a, device);
  const long long n_items = (p.keys ? n_blocks : (n_blocks + QT - 1) / QT) * heads;
  if (n_items > 0x7fffffffll) return cudaErrorInvalidValue;
  const int sms = sm_count(device);
  const int grid = p.cluster > 1 ? static_cast<int>(n_items) * p.cluster : static_cast<int>(n_items < sms ? n_items : sms);
  const bool counter = p.cluster == 1 && n_items > grid;
  if (GEN == 2 && a.mask_lens) {
    int32_t* lens = a.mask_lens;
    cudaError_t e = launch_early(lens_kernel, dim3(a.B), dim3(256), 0, stream, 1, a, a.sched, lens, lens + a.B);
    if (e != cudaSuccess) return e;
    a.kv_lens = lens, a.mask_pure = lens + a.B;
  } else if (counter) {
    // the counter that hands out what comes after the CTAs' first items must start at zero for every launch
    cudaError_t e = launch_zero_word(a.sched, stream);
    if (e != cudaSuccess) return e;
  }
  if (!counter) a.sched = nullptr;
  return p.keys ? launch_k<D, BF16, GEN, true>(a, dtype, grid, p.cluster, stream)
                : launch_k<D, BF16, GEN, false>(a, dtype, grid, 1, stream);
}

}  // namespace

template <int GEN>
cudaError_t launch_g(int dtype, int D, const FwdArgs& a, int device, cudaStream_t stream) {
  const bool bf = dtype == TT_ATTN_BF16;
  if (D == 128)
    return bf ? launch_t<128, true, GEN>(a, dtype, device, stream) : launch_t<128, false, GEN>(a, dtype, device, stream);
  if (D == 64)
    return bf ? launch_t<64, true, GEN>(a, dtype, device, stream) : launch_t<64, false, GEN>(a, dtype, device, stream);
  return cudaErrorInvalidValue;
}

cudaError_t launch_fwd_tc(int dtype, int D, const FwdArgs& a, int device, cudaStream_t stream) {
  // the general variant only where it is needed: the fast one carries none of its code
  const bool general = a.causal == TT_ATTN_CAUSAL_BOTTOM_RIGHT;
  return a.mask.ptr ? launch_g<2>(dtype, D, a, device, stream)
         : general  ? launch_g<1>(dtype, D, a, device, stream)
                    : launch_g<0>(dtype, D, a, device, stream);
}

}  // namespace ttattn
