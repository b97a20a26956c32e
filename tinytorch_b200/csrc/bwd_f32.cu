// Attention backward for Float32 tensors on the tensor cores: fp32 products as sums of bf16 ones (f32_pieces.cuh).
//
// CTAs of two kinds in one launch, one walk for both.  A CTA owns 128 rows ("own") and walks tiles of 64 rows of the other side ("other"):
//   key CTAs    own: keys;     other: queries of all heads of the group, query by query; out: dV = P^T dO and dK = dS^T Q
//   query CTAs  own: queries of all heads of the group, query by query; other: keys;     out: dQ = dS K
// S and dP are made with the own side in the MMA's rows, so that a thread finds its row's scores in its TMEM lane and leaves P and
// dS there as the A operands of the products that follow.  K (Q) of the own side lies in TMEM, V (dO) in shared memory, the other side's
// two tiles in shared memory, all as three bf16 planes.  Every tile's product is read from TMEM and added to the sums in registers.
//   warps 0-7   two warpgroups, the halves of the 64 columns: P and dS; then the tile's products into the sums: key CTAs dV the
//               first, dK the second, query CTAs half the columns of dQ each
//   warps 8-15  the other side's tiles into their pieces, with what goes with their rows (log-sum-exp, delta); D = 64: the first operand (Q or
//               K) by one warpgroup, the second (dO or V) by the other; D = 128, where a tile waits for its one place: by both together.
//               The second warpgroup brings masks too
//   warp 16     issues the MMAs of S and dP: of the next tile as soon as what lies in their places has been used
//   warp 17     issues those of dV and dK (dQ)
// so that P is made under dK of the tile before and dP, and dS under dV.  (One warp for all four spends 1700 of 6100 clocks per tile in waits.)
// No atomics: every sum runs in one order.
//
// Where there is room for dS and work enough for one more launch (bwd_ds_bytes), the key CTAs leave theirs and bwd_f32_dq_kernel makes dQ
// of it: one product instead of the query CTAs' three.
//
// Bound by the tensor pipe and the waits around it; D = 128, where only one tile of the other side fits, by its two operands' conversion
// besides.  Against the same in fp32 FMAs on CUDA cores, us, with the delta pass: D = 64, 4 x 8 heads x 500 156 -> 58 (additive mask 170 -> 74),
// causal 8 x 8 x 1024 785 -> 245, 2 x 16/2 x 700 218 -> 86, but one tile of 4 x 16 x 57 12.5 -> 15.3; D = 128, 4 x 8 x 500 296 -> 110 (additive mask
// 304 -> 137), causal 4 x 8 x 1024 718 -> 203.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cluster_host.cuh"
#include "f32_pieces.cuh"

namespace ttattn {
namespace {

using namespace pieces;
enum MaskForm { kNoMask, kBoolMask, kAddMask };
constexpr int BM = 128, BN = 64;
constexpr int kThreads = 640, kWork = 256, kIssueWarp = 16;

struct Ctl {
  uint64_t a_full, b1_full[2], b1_free[2], b2_full[2], b2_free[2], s_full, dp_full, p_full, ds_full, t1_full, t2_full, t1_free, t2_free, m_full, m_free;
  uint64_t x_free, y_free;  // the places of S and P, dP and dS
  uint32_t tmem_base;
  int abort_flag, bad;
};

template <int D, MaskForm MASK>
struct Lay {
  using TA = Tile<BM, D, kWork>;
  static constexpr int kLoad = D == 64 ? 128 : 256;  // threads that bring a tile
  using TB = Tile<BN, D, kLoad>;
  static constexpr int kStages = D == 64 ? 2 : 1;  // of the other side's tiles
  static constexpr int kMaskBytes = MASK == kNoMask ? 0 : (MASK == kBoolMask ? BM * 8 : BM * BN * 4);
  static constexpr int kA2 = 0, kB1 = TA::kBytes, kB2 = kB1 + kStages * TB::kBytes, kM = kB2 + kStages * TB::kBytes;
  static constexpr int kVec = kM + kMaskBytes;  // [2][exponent base, factor, delta][64]
  static constexpr int kVecBytes = 3 * BN * 4;
  static constexpr int kCtl = kVec + 2 * kVecBytes;
  static constexpr int kBytes = kCtl + 256;
  static constexpr int kLdO = D + 4;  // floats a row of the sums on their way out
  // TMEM: planes of the own side's first operand | S, then P | dP, then dS | product of a tile.
  // kWide: products of 64 columns come as two sums (f32_pieces.cuh).  The planes of 16 columns
  // of P and dS lie over the scores that they are made of.  Without (TMEM is full), scores lie in columns 16..79 of a region and the
  // planes of 16 columns in 24 each: written first to last by the one warpgroup and last to first by the other, they come to lie over
  // scores that have been read.
  static constexpr bool kWide = D == 64;
  static constexpr uint32_t kRegion = kWide ? 2 * BN : 96, kScores = kWide ? 0 : 16;
  static __host__ __device__ constexpr uint32_t plane_at(uint32_t piece, uint32_t ks) {
    return kWide ? ks * 16 + (piece == 2 ? 64 : piece * 8) : ks * 24 + piece * 8;
  }
  static constexpr uint32_t kA1 = 0, kX = D / 2 * kPieces, kY = kX + kRegion, kT = kY + kRegion;
  static_assert(kT + (kWide ? 2 * D : D) <= 512, "TMEM");
  static constexpr int kWorkRegs = D == 64 ? 152 : 184, kLoadRegs = D == 64 ? 64 : 40, kIssueRegs = D == 64 ? 48 : 32;
  static_assert(2 * kWorkRegs + 2 * kLoadRegs + kIssueRegs <= 5 * 96, "registers of the launch");
  static_assert(2 * BM * kLdO * 4 <= kVec, "sums over the tiles");
};
static_assert(sizeof(Ctl) <= 256, "control block");
static_assert(Lay<128, kAddMask>::kBytes <= 227 * 1024, "shared memory");

// two neighbouring words of accumulators
__device__ __forceinline__ float2 floats2(const uint32_t (&x)[16], int i) { return make_float2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])); }
// where dS waits for the dQ pass: for each (batch, kv head) the queries' rows, in whole tiles, of keys, in whole tiles
__device__ __forceinline__ int ds_pitch(const BwdArgs& a) { return (a.Skv + BN - 1) / BN * BN; }
__device__ __forceinline__ int ds_rows(const BwdArgs& a) { return (a.Lq * (a.Hq / a.Hkv) + BN - 1) / BN * BN; }
__device__ __forceinline__ float* ds_of(const BwdArgs& a, int b, int hk) {
  return a.ds + (static_cast<int64_t>(b) * a.Hkv + hk) * ds_rows(a) * ds_pitch(a);
}

// Nothing follows where the roles' ways meet: a warp that has given registers back must not come to code that is compiled for more.
template <int D, bool KEYS, MaskForm MASK, bool SPLIT>
__device__ __forceinline__ void walk(const BwdArgs& a, uint8_t* smem, uint32_t base, Ctl* ctl, uint32_t tmem, int item, int rank, int cluster) {
  using LY = Lay<D, MASK>;
  using TA = typename LY::TA;
  using TB = typename LY::TB;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort_flag = &ctl->abort_flag;

  // ------------------------------------------------------------------------------------------------ what to do --
  const int group = a.Hq / a.Hkv, rows = a.Lq * group, heads = a.B * a.Hkv;
  const int own_tiles = KEYS ? (a.Skv + BM - 1) / BM : (rows + BM - 1) / BM;
  // longest walks first: under a causal mask those of the first keys and the last queries
  const int mt = KEYS ? item / heads : own_tiles - 1 - item / heads;
  const int hk = item % heads % a.Hkv, b = item % heads / a.Hkv, own0 = mt * BM;
  const Group rw(group, rows);
  const int head0 = hk * group;
  int kv_len = a.Skv;
  if (a.kv_lens) {
    const int l = a.kv_lens[b];
    kv_len = l < 0 ? 0 : (l < a.Skv ? l : a.Skv);
  }
  const int shift = causal_shift(a.causal, kv_len, a.Lq);
  // tiles of the other side: from `begin` on, `tiles` of them
  int begin = 0, tiles;
  if constexpr (KEYS) {
    const long long first = a.causal && own0 > shift ? static_cast<long long>(own0 - shift) * group : 0;  // row of the first query that sees a key
    const bool any = own0 < kv_len && first < rows;
    begin = any ? static_cast<int>(first) / BN : 0;
    tiles = any ? (rows + BN - 1) / BN - begin : 0;
  } else {
    const int last_q = rw.query(min(own0 + BM, rows) - 1);
    tiles = ((a.causal ? max(0, min(kv_len, last_q + shift + 1)) : kv_len) + BN - 1) / BN;
  }
  if (SPLIT) {
    const int t0 = tiles * rank / cluster, t1 = tiles * (rank + 1) / cluster;
    begin += t0, tiles = t1 - t0;
  }
  const int n = tiles;
  const float* qp = reinterpret_cast<const float*>(a.q) + b * a.qs.b;
  const float* gp = reinterpret_cast<const float*>(a.d_o) + b * a.dos.b;
  const float* kp = reinterpret_cast<const float*>(a.k) + b * a.ks.b + hk * a.ks.h;
  const float* vp = reinterpret_cast<const float*>(a.v) + b * a.vs.b + hk * a.vs.h;
  // The first or second operand's row r, of queries (Q, dO) or keys (K, V): row 0 stands in where there is none.
  auto query_row = [&](bool first, int r) {
    r = r < rows ? r : 0;
    const int64_t i = rw.query(r), h = head0 + rw.head(r);
    return first ? qp + h * a.qs.h + i * a.qs.s : gp + h * a.dos.h + i * a.dos.s;
  };
  auto key_row = [&](bool first, int r) {
    const int64_t i = r < kv_len ? r : 0;
    return first ? kp + i * a.ks.s : vp + i * a.vs.s;
  };
  auto own_row = [&](bool first, int r) { return KEYS ? key_row(first, own0 + r) : query_row(first, own0 + r); };
  const int own_rows = (KEYS ? kv_len : rows) - own0, other_rows = KEYS ? rows : kv_len;  // (own ones may be fewer than none)
  const int64_t stat_base = static_cast<int64_t>(b) * a.Hq * a.Lq;  // of lse and delta
  auto stat_at = [&](int r) { return stat_base + static_cast<int64_t>(head0 + rw.head(r)) * a.Lq + rw.query(r); };
  auto stats_of = [&](int r) {  // of the query in row r
    if (r >= rows) return make_float2(-INFINITY, 1.f);
    if (MASK == kAddMask && a.row_stats) return a.row_stats[stat_at(r)];
    const float lse = a.lse[stat_at(r)];
    // (too large for its exponents to be right within a few per cent, and no room for better: the row counts for nothing)
    return MASK == kAddMask && fabsf(lse) >= 0x1p18f ? make_float2(-INFINITY, 1.f) : exponent_base(lse, kv_len);
  };

  auto last_pass = [&](bool careful) {  // by all threads at the end of a pass
    ptx::named_barrier(1, kThreads);
    return !ctl->bad || careful || n == 0 || *abort_flag;
  };
  float* out_s = reinterpret_cast<float*>(smem);  // the sums on their way out: [one or two][row][kLdO]

  if (warp < 8) {
    // ------------------------------------------------------------------------------------------- P, dS and sums --
    ptx::setmaxnreg_inc<LY::kWorkRegs>();
    constexpr int kAcc = KEYS ? D / 2 : D / 4;
    const int wg = warp >> 2, r = tid & 127;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t x_at = tmem + LY::kX + lane_base, y_at = tmem + LY::kY + lane_base;
    float2 acc[kAcc];
    bool careful = false;
    for (int done = 0, pass = 0;; ++pass, done += n, careful = true) {
#pragma unroll
      for (int j = 0; j < kAcc; ++j) acc[j] = make_float2(0.f, 0.f);
      float2 odd = make_float2(0.f, 0.f);  // NaN once something is not finite
      if (n > 0) {
        // the own side: first operand into TMEM (a thread half a row), second into shared memory
        {
          const float* p = own_row(true, r);
#pragma unroll 1
          for (int j = wg * (D / 2); j < (wg + 1) * (D / 2); j += 16) {
            float4 x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = load4_or_zero(p + j + 4 * e, r < own_rows);
            uint32_t w[kPieces][8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (rare(careful)) {
                split2<true>(x[e].x, x[e].y, w[0][2 * e], w[1][2 * e], w[2][2 * e], odd);
                split2<true>(x[e].z, x[e].w, w[0][2 * e + 1], w[1][2 * e + 1], w[2][2 * e + 1], odd);
              } else {
                split2<false>(x[e].x, x[e].y, w[0][2 * e], w[1][2 * e], w[2][2 * e], odd);
                split2<false>(x[e].z, x[e].w, w[0][2 * e + 1], w[1][2 * e + 1], w[2][2 * e + 1], odd);
              }
            }
#pragma unroll
            for (int i = 0; i < kPieces; ++i) ptx::tmem_st8(tmem + LY::kA1 + lane_base + i * (D / 2) + j / 2, w[i]);
          }
          ptx::tmem_wait_st();
          ptx::tc_fence_before();
        }
#pragma unroll 1
        for (int i0 = 0; i0 < TA::kChunks; i0 += 4) {
          float4 x[4][2];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = TA::row(tid, i0 + i);
            const float* p = own_row(false, row) + TA::col(tid);
            x[i][0] = load4_or_zero(p, row < own_rows), x[i][1] = load4_or_zero(p + 4, row < own_rows);
          }
#pragma unroll
          for (int i = 0; i < 4; i += 2) TA::put(base + LY::kA2, tid, i0 + i, reinterpret_cast<const float4(&)[2][2]>(x[i]), careful, odd);
        }
        ptx::fence_proxy_async_smem();
        ptx::mbar_arrive(&ctl->a_full);
      }
      const float c = a.scale * kLog2e;
      // what the row takes part in: other rows lo .. hi - 1
      int lo = 0, hi;
      float2 stats = make_float2(0.f, 1.f);  // query CTAs: the row's
      float delta = 0.f;
      int all_lo = 0, all_hi;         // what every row of the CTA takes part in
      if constexpr (KEYS) {
        const int key = own0 + r;
        const long long from = a.causal ? static_cast<long long>(key - shift) * group : 0;
        lo = key >= kv_len || from >= rows ? 0x7fffffff : max(0, static_cast<int>(from));
        hi = rows;
        const long long last = a.causal ? static_cast<long long>(own0 + BM - 1 - shift) * group : 0;
        all_lo = own0 + BM > kv_len || last >= rows ? 0x7fffffff : max(0, static_cast<int>(last));
        all_hi = rows;
      } else {
        const int i_q = rw.query(own0 + r);
        hi = own0 + r < rows ? (a.causal ? min(kv_len, i_q + shift + 1) : kv_len) : 0;
        all_hi = a.causal ? min(kv_len, rw.query(own0) + shift + 1) : kv_len;
        stats = stats_of(own0 + r);
        delta = own0 + r < rows ? a.delta[stat_at(own0 + r)] : 0.f;
      }
      // a tile's product into the sums
      const uint32_t from = tmem + lane_base + LY::kT + (KEYS ? 0 : wg * (D / 2));
      auto take = [&](uint64_t* full, uint64_t* free, uint32_t at) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(full, at & 1, abort_flag))) return false;
        ptx::tc_fence_after();
#pragma unroll
        for (int j = 0; j < kAcc; j += 8) {
          uint32_t o[16], o2[16];
          ptx::tmem_ld16(from + 2 * j, o);
          if (LY::kWide) ptx::tmem_ld16(from + D + 2 * j, o2);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e)
            acc[j + e] = ptx::add2(acc[j + e], LY::kWide ? ptx::add2(floats2(o, 2 * e), floats2(o2, 2 * e)) : floats2(o, 2 * e));
        }
        ptx::tc_fence_before();
        ptx::mbar_arrive(free);
        return true;
      };
      for (int t = 0; t < n; ++t) {
        const uint32_t at = done + t, par = at & 1;
        const int col0 = (begin + t) * BN;
        const uint32_t vec = base + LY::kVec + par * LY::kVecBytes;  // key CTAs: of the columns
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctl->s_full, par, abort_flag))) break;
        if constexpr (MASK != kNoMask)
          if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctl->m_full, par, abort_flag))) break;
        ptx::tc_fence_after();
        float p[32];  // in the order of the blocks
        auto planes = [&](uint32_t at, const float* x) {  // pieces of a block's 16 columns
          uint32_t w[kPieces][8];
          if (rare(careful)) {
#pragma unroll
            for (int e = 0; e < 8; ++e) split2<true>(x[2 * e], x[2 * e + 1], w[0][e], w[1][e], w[2][e], odd);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) split2<false>(x[2 * e], x[2 * e + 1], w[0][e], w[1][e], w[2][e], odd);
          }
#pragma unroll
          for (int i = 0; i < kPieces; ++i) ptx::tmem_st8(at + LY::plane_at(i, 0), w[i]);
        };
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          const int j0 = wg * 32 + (blk ^ wg) * 16;  // the block's first column
          float* pb = p + blk * 16;
          uint32_t s[16], s2[16];
          ptx::tmem_ld16(x_at + LY::kScores + j0, s);
          if (LY::kWide) ptx::tmem_ld16(x_at + BN + j0, s2);
          uint32_t seen = 0xffffffffu;  // a boolean mask's bits
          if constexpr (MASK == kBoolMask) {
            if constexpr (KEYS) {  // words of 32 keys, one per column
              seen = 0;
#pragma unroll
              for (int j = 0; j < 16; j += 4) {
                const uint4 w = ptx::ld_shared4(base + LY::kM + ((warp & 3) * BN + j0 + j) * 4);
                seen |= (w.x >> lane & 1) << j | (w.y >> lane & 1) << (j + 1) | (w.z >> lane & 1) << (j + 2) | (w.w >> lane & 1) << (j + 3);
              }
            } else {  // two words a row
              asm volatile("ld.shared.u32 %0, [%1];" : "=r"(seen) : "r"(base + LY::kM + r * 8 + wg * 4) : "memory");
              seen >>= j0 & 31;
            }
          }
          ptx::tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            float l4[4] = {stats.x, stats.x, stats.x, stats.x}, w4[4] = {stats.y, stats.y, stats.y, stats.y};
            if constexpr (KEYS) {
              const float4 v = ptx::ld_shared_f4(vec + (j0 + j) * 4), w = ptx::ld_shared_f4(vec + (BN + j0 + j) * 4);
              l4[0] = v.x, l4[1] = v.y, l4[2] = v.z, l4[3] = v.w;
              w4[0] = w.x, w4[1] = w.y, w4[2] = w.z, w4[3] = w.w;
            }
            float mk[4];
            if constexpr (MASK == kAddMask) {
              if constexpr (KEYS) {
#pragma unroll
                for (int e = 0; e < 4; ++e) mk[e] = *reinterpret_cast<const float*>(smem + LY::kM + ((j0 + j + e) * BM + r) * 4);
              } else {
                const float4 v = ptx::ld_shared_f4(base + LY::kM + r * BN * 4 + (((j0 + j) / 4 ^ (r & 7)) << 4));
                mk[0] = v.x, mk[1] = v.y, mk[2] = v.z, mk[3] = v.w;
              }
            }
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              const float2 c2 = make_float2(c, c), l2 = make_float2(l4[e], l4[e + 1]);
              float2 x = LY::kWide ? ptx::add2(floats2(s, j + e), floats2(s2, j + e)) : floats2(s, j + e);
              if constexpr (MASK == kAddMask)  // (the forward's sum, with its roundings)
                x = ptx::add2(ptx::fma2(make_float2(mk[e], mk[e + 1]), make_float2(kLog2e, kLog2e), ptx::mul2(x, c2)), l2);
              else
                x = ptx::fma2(x, c2, l2);
              x = ptx::mul2(make_float2(ptx::ex2(x.x), ptx::ex2(x.y)), make_float2(w4[e], w4[e + 1]));
              pb[j + e] = x.x, pb[j + e + 1] = x.y;
            }
          }
          const bool edge = col0 + j0 < all_lo || col0 + j0 + 16 > all_hi;
          if (edge || MASK == kBoolMask) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (col0 + j0 + j < lo || col0 + j0 + j >= hi || !(seen >> j & 1)) pb[j] = 0.f;
          }
          if constexpr (KEYS) planes(x_at + LY::plane_at(0, j0 / 16), pb);
        }
        if constexpr (MASK != kNoMask) ptx::mbar_arrive(&ctl->m_free);
        if constexpr (KEYS) ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive(KEYS ? &ctl->p_full : &ctl->x_free);  // (query CTAs: S has been read)
        if (!(KEYS && wg == 0) && t > 0 && !take(&ctl->t2_full, &ctl->t2_free, at - 1)) break;
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctl->dp_full, par, abort_flag))) break;
        ptx::tc_fence_after();
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          const int j0 = wg * 32 + (blk ^ wg) * 16;
          float* pb = p + blk * 16;
          uint32_t s[16], s2[16];
          ptx::tmem_ld16(y_at + LY::kScores + j0, s);
          if (LY::kWide) ptx::tmem_ld16(y_at + BN + j0, s2);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            float d4[4] = {delta, delta, delta, delta};
            if constexpr (KEYS) {
              const float4 v = ptx::ld_shared_f4(vec + 2 * BN * 4 + (j0 + j) * 4);
              d4[0] = v.x, d4[1] = v.y, d4[2] = v.z, d4[3] = v.w;
            }
#pragma unroll
            for (int e = 0; e < 4; e += 2) {  // dS, without the scale
              const float2 dp = LY::kWide ? ptx::add2(floats2(s, j + e), floats2(s2, j + e)) : floats2(s, j + e);
              const float2 x = ptx::mul2(make_float2(pb[j + e], pb[j + e + 1]), ptx::add2(dp, make_float2(-d4[e], -d4[e + 1])));
              pb[j + e] = x.x, pb[j + e + 1] = x.y;
            }
          }
          planes(y_at + LY::plane_at(0, j0 / 16), pb);
          if (KEYS && a.ds && own0 + r < ds_pitch(a)) {
            float* p = ds_of(a, b, hk) + static_cast<int64_t>(col0 + j0) * ds_pitch(a) + own0 + r;
#pragma unroll
            for (int j = 0; j < 16; ++j, p += ds_pitch(a)) *p = pb[j];
          }
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive(&ctl->ds_full);
        if (KEYS && wg == 0 && !take(&ctl->t1_full, &ctl->t1_free, at)) break;
      }
      if (!(KEYS && wg == 0) && n > 0 && !__any_sync(0xffffffffu, *abort_flag != 0)) take(&ctl->t2_full, &ctl->t2_free, done + n - 1);
      if (was_odd(odd)) ctl->bad = 1;
      if (last_pass(careful)) break;
    }
    // dK and dQ still want the scale
    const float f = KEYS && wg == 0 ? 1.f : a.scale;
    float* dst = out_s + (KEYS ? (wg * BM + r) * LY::kLdO : r * LY::kLdO + wg * (D / 2));
#pragma unroll
    for (int j = 0; j < kAcc; j += 2)
      *reinterpret_cast<float4*>(dst + 2 * j) = make_float4(acc[j].x * f, acc[j].y * f, acc[j + 1].x * f, acc[j + 1].y * f);
    auto store = [&](int which, int r, int d, const float4& x) {  // of dV (0) or dK (1), or of dQ
      if constexpr (KEYS) {
        float* p = reinterpret_cast<float*>(which == 0 ? a.dv : a.dk);
        const int64_t st_b = which == 0 ? a.dvs.b : a.dks.b, st_h = which == 0 ? a.dvs.h : a.dks.h, st_s = which == 0 ? a.dvs.s : a.dks.s;
        if (p && own0 + r < a.Skv) *reinterpret_cast<float4*>(p + b * st_b + hk * st_h + (own0 + r) * st_s + d) = x;
      } else if (own0 + r < rows) {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.dq) + b * a.dqs.b + (head0 + rw.head(own0 + r)) * a.dqs.h + rw.query(own0 + r) * a.dqs.s + d) = x;
      }
    };
    constexpr int kOuts = KEYS ? 2 : 1;
    const int d = tid % (D / 4) * 4;
    if constexpr (SPLIT) {
      ptx::cluster_sync();
      // the shares of the cluster's CTAs, added in rank order; every CTA stores a share of the rows
      constexpr int kMost = 8;
      const int share = (BM + cluster - 1) / cluster;
#pragma unroll 1
      for (int e = tid / (D / 4); e < kOuts * share; e += kWork / (D / 4)) {
        const int which = e / share, row = rank * share + e % share;
        if (row >= BM) continue;
        const uint32_t at = ptx::smem_u32(out_s + (which * BM + row) * LY::kLdO + d);
        float4 x[kMost], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kMost; ++i)
          if (i < cluster) x[i] = ptx::ld_cluster_f4(ptx::map_rank(at, i));
#pragma unroll
        for (int i = 0; i < kMost; ++i)
          if (i < cluster) sum.x += x[i].x, sum.y += x[i].y, sum.z += x[i].z, sum.w += x[i].w;
        store(which, row, d, sum);
      }
      ptx::cluster_sync();  // no CTA leaves while another still reads its share
    } else {
      ptx::named_barrier(2, kWork);
#pragma unroll 4
      for (int e = tid / (D / 4); e < kOuts * BM; e += kWork / (D / 4))
        store(e / BM, e % BM, d, *reinterpret_cast<const float4*>(out_s + e * LY::kLdO + d));
    }
    if (tid == 0 && *abort_flag && a.status) atomicOr(a.status, kStatusWaitExpired);
  } else if (warp < kIssueWarp) {
    // ---------------------------------------------------------------------------- the other side's tiles, masks --
    ptx::setmaxnreg_dec<LY::kLoadRegs>();
    const int lt = tid & (LY::kLoad - 1);
    constexpr int kHeld = D == 64 ? 4 : 2;  // chunks in flight
    float4 raw[kHeld][2];
    // (D = 64: which of the operands is a number of the warp's, and the code for both is one: as two copies it is 15 % slower)
    struct Operand {
      const float* rows;
      int64_t st_s, st_h;
    };
    auto operand = [&](bool first) {
      return Operand{(KEYS ? (first ? qp + head0 * a.qs.h : gp + head0 * a.dos.h) : (first ? kp : vp)) + TB::col(lt),
                     KEYS ? (first ? a.qs.s : a.dos.s) : (first ? a.ks.s : a.vs.s), first ? a.qs.h : a.dos.h};
    };
    const Operand mine = operand(warp < 12);
    auto fetch = [&](bool first, int t, int i0) {
      const Operand x = LY::kLoad == 128 ? mine : operand(first);
#pragma unroll
      for (int i = 0; i < kHeld; ++i) {
        const int row = (begin + t) * BN + TB::row(lt, i0 + i);
        const float* p = KEYS ? x.rows + rw.query(row) * x.st_s : x.rows + row * x.st_s;
        if (KEYS && group > 1) p += rw.head(row) * x.st_h;
        raw[i][0] = load4_or_zero(p, row < other_rows), raw[i][1] = load4_or_zero(p + 4, row < other_rows);
      }
    };
    bool careful = false;
    for (int done = 0;; done += n, careful = true) {
      float2 odd = make_float2(0.f, 0.f);
      auto put_mask = [&](int t) {
        const uint32_t at = done + t;
        const int mt_id = tid & 127;
        const int col0 = (begin + t) * BN, w = warp & 3;
        if (t > 0 && !__all_sync(0xffffffffu, ptx::mbar_wait(&ctl->m_free, (at - 1) & 1, abort_flag))) return false;
        const int64_t mask_b = b * a.mask.sb + head0 * a.mask.sh;
        // of the query in row r: whether there is one, and where its mask begins
        auto row_at = [&](int r) { return mask_b + rw.head(r) * a.mask.sh + rw.query(r) * a.mask.sl; };
        if constexpr (MASK == kBoolMask) {
          // 64 keys of a row to bits, by a thread: the aligned words that hold their bytes, shifted into place
          const int r = KEYS ? col0 + mt_id % BN : own0 + mt_id, key = KEYS ? own0 + mt_id / BN * 64 : col0;
          const uintptr_t at_b = reinterpret_cast<uintptr_t>(a.mask.ptr) + row_at(r) + key;
          const int mis = static_cast<int>(at_b & 3), end = r < rows ? min(64, kv_len - key) + mis : 0;
          const uint32_t* words = reinterpret_cast<const uint32_t*>(at_b - mis);
          uint32_t x = 0 < end ? __ldg(words) : 0, two[2] = {0, 0};
#pragma unroll 4
          for (int i = 0; i < 16; ++i) {
            const uint32_t y = 4 * i + 4 < end ? __ldg(words + i + 1) : 0;
            const uint32_t v = mask_bits(x, y, mis) << (4 * (i % 8));
            two[0] |= i < 8 ? v : 0, two[1] |= i < 8 ? 0 : v;
            x = y;
          }
          if constexpr (KEYS) {  // words of 32 keys, one per column
            uint32_t* to = reinterpret_cast<uint32_t*>(smem + LY::kM) + mt_id / BN * 2 * BN + mt_id % BN;
            to[0] = two[0], to[BN] = two[1];
          } else {  // two words a row
            *reinterpret_cast<uint2*>(smem + LY::kM + mt_id * 8) = make_uint2(two[0], two[1]);
          }
          ptx::mbar_arrive(&ctl->m_full);
        } else if constexpr (MASK == kAddMask) {
          const float* any = reinterpret_cast<const float*>(a.mask.ptr);
          auto each_row = [&](int r0, int step, int count, auto f) {
            each_mask_row<2>(a.mask, group, rows, r0, rw.head(r0), row_at(r0), step, count, f);
          };
          if constexpr (KEYS) {  // [column][key], 16 columns a warp
            constexpr int kCols = BN / 4;
            const uint32_t to = base + LY::kM + w * kCols * BM * 4;
            if (a.mask.wide) {
              const int key = own0 + lane * 4, left = min(4, a.Skv - key);
              each_row(col0 + w * kCols, 1, kCols, [&](int e, bool in, int64_t p) {
                in = in && left > 0;
                ptx::cp_async16(to + e * BM * 4 + lane * 16, in ? any + p + key : any, in ? left * 4 : 0);
              });
            } else {
              const int key = own0 + lane, last = kv_len - own0 - lane;  // (keys beyond the length are left as they are: they are hidden)
              each_row(col0 + w * kCols, 1, kCols, [&](int e, bool in, int64_t p) {
                const uint32_t dst = to + (e * BM + lane) * 4;
                const float* from = in ? any + p + key : any;
                copies4(dst, from, in, last > 0, last > 32);
                copies4(dst + 256, from + 64, in, last > 64, last > 96);
              });
            }
          } else {  // [row][64], neighbouring vectors exchanged by row; 32 rows a warp
            constexpr int kOwn = BM / 4;
            if (a.mask.wide) {
              const int ch = lane % 16, r0 = w * kOwn + lane / 16, left = min(4, a.Skv - col0 - ch * 4);
              each_row(own0 + r0, 2, kOwn / 2, [&](int e, bool in, int64_t p) {
                in = in && left > 0;
                ptx::cp_async16(base + LY::kM + (r0 + e) * BN * 4 + ((ch ^ ((r0 + e) & 7)) << 4), in ? any + p + col0 + ch * 4 : any, in ? left * 4 : 0);
              });
            } else {
              each_row(own0 + w * kOwn, 1, kOwn, [&](int e, bool in, int64_t p) {
                const int rr = w * kOwn + e;
                copies4(base + LY::kM + rr * BN * 4 + (((lane / 4) ^ (rr & 7)) << 4) + (lane % 4) * 4, in ? any + p + col0 + lane : any, in,
                        col0 + lane < kv_len, col0 + lane + 32 < kv_len);
              });
            }
          }
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(ptx::smem_u32(&ctl->m_full)) : "memory");
        }
        return true;
      };
      auto bring = [&](bool first, int t) {  // (its first chunks have been asked for); false: a wait has run out
        const uint32_t at = done + t, stage = at % LY::kStages, use = at / LY::kStages;
        // (the first operand's place is free once dK or dQ of its last user has been made, the second's once dP and dV have)
        if (use > 0 && !__all_sync(0xffffffffu, ptx::mbar_wait(first ? &ctl->b1_free[stage] : &ctl->b2_free[stage], (use - 1) & 1, abort_flag)))
          return false;
        if (KEYS && first && lt < BN) {
          const int r = (begin + t) * BN + lt;
          const float2 stats = stats_of(r);
          float* vec = reinterpret_cast<float*>(smem + LY::kVec + (at & 1) * LY::kVecBytes);
          vec[lt] = stats.x, vec[BN + lt] = stats.y;
          vec[2 * BN + lt] = r < rows ? a.delta[stat_at(r)] : 0.f;
        }
#pragma unroll
        for (int i0 = 0; i0 < TB::kChunks; i0 += kHeld) {
          if (i0 > 0) fetch(first, t, i0);
#pragma unroll
          for (int i = 0; i < kHeld; ++i)
            TB::put(base + (first ? LY::kB1 : LY::kB2) + stage * TB::kBytes, lt, i0 + i, reinterpret_cast<const float4(&)[1][2]>(raw[i]), careful, odd);
        }
        ptx::fence_proxy_async_smem();
        ptx::mbar_arrive(first ? &ctl->b1_full[stage] : &ctl->b2_full[stage]);
        return true;
      };
      if constexpr (LY::kLoad == 128) {
        const bool first = warp < 12;
        if (n > 0) fetch(first, 0, 0);
        for (int t = 0; t < n; ++t) {
          if (!bring(first, t)) break;
          if (t + 1 < n) fetch(first, t + 1, 0);
          if (MASK != kNoMask && !first && !put_mask(t)) break;
        }
      } else {
        // (the second operand's place is the first to be free)
        if (n > 0) fetch(false, 0, 0);
        for (int t = 0; t < n; ++t) {
          if (!bring(false, t)) break;
          fetch(true, t, 0);
          if (MASK != kNoMask && warp >= 12 && !put_mask(t)) break;
          if (!bring(true, t)) break;
          if (t + 1 < n) fetch(false, t + 1, 0);
        }
      }
      if (was_odd(odd)) ctl->bad = 1;
      if (last_pass(careful)) break;
    }
    if (SPLIT) ptx::cluster_sync(), ptx::cluster_sync();
  } else {
    // --------------------------------------------------------------------------------------------------- the MMAs --
    ptx::setmaxnreg_dec<LY::kIssueRegs>();
    bool careful = false;
    for (int done = 0, pass = 0;; ++pass, done += n, careful = true) {
      const bool leader = ptx::elect_one();
      auto uwait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag)) != 0; };
      constexpr uint32_t kIdescS1 = ptx::make_idesc_f16(BM, BN, 1, 0, 0), kIdescS2 = ptx::make_idesc_f16(BM, 2 * BN, 1, 0, 0);
      constexpr uint32_t kIdescT1 = ptx::make_idesc_f16(BM, D, 1, 0, 1), kIdescT2 = ptx::make_idesc_f16(BM, 2 * D, 1, 0, 1);
      constexpr uint32_t kHi = ptx::smem_desc_hi_sw128(1024);
      constexpr uint32_t kPA = TA::kPlane >> 4, kPB = TB::kPlane >> 4;
      const uint32_t a2 = ptx::smem_desc_lo(base + LY::kA2, 16), b1 = ptx::smem_desc_lo(base + LY::kB1, 16);
      const uint32_t b2 = ptx::smem_desc_lo(base + LY::kB2, 16);
      constexpr int kLbo = LY::kWide ? TB::kPlane : TB::kBlock;
      const uint32_t b1_mn = ptx::smem_desc_lo(base + LY::kB1, kLbo), b2_mn = ptx::smem_desc_lo(base + LY::kB2, kLbo);
      constexpr Sums kSums = LY::kWide ? kLeadApart : kOneSum, kSumsT = LY::kWide ? kTwoSums : kOneSum;
      // product of a tile: A's planes from TMEM region `region`, B MN-major
      auto issue_t = [&](uint32_t region, uint32_t b_mn) {
#pragma unroll 1  // (all products at once: the addresses do not fit this warp's registers)
        for (int p = 0; p < steps_of(kSumsT); ++p) {
          const Step st = step_of(kSumsT, p);
          const uint32_t d = tmem + LY::kT + (st.second ? D : 0), ap = tmem + region + LY::plane_at(st.a, 0), bp = b_mn + st.b * kPB;
          const uint32_t idesc = st.two ? kIdescT2 : kIdescT1;
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            if (leader) ptx::mma_ts2(d, ap + LY::plane_at(0, ks), bp + ks * (2048 >> 4), kHi, idesc, st.onto || ks > 0 ? 1u : 0u);
        }
      };
      // (Every lane polls every barrier: tcgen05.mma wants the warp together, and lanes that wait for different barriers come apart.)
      // S = K Q^T (Q K^T), tile t; a_full: the own side is there
      auto issue_s = [&](int t) {
        const uint32_t at = done + t, stage = at % LY::kStages, stage_at = stage * (TB::kBytes >> 4);
        if (!uwait(&ctl->b1_full[stage], at / LY::kStages & 1) || !(t == 0 ? uwait(&ctl->a_full, pass & 1) : uwait(&ctl->x_free, (at - 1) & 1))) return false;
        ptx::tc_fence_after();
#pragma unroll 1
        for (int p = 0; p < steps_of(kSums); ++p) {
          const Step st = step_of(kSums, p);
          const uint32_t d = tmem + LY::kX + LY::kScores + (st.second ? BN : 0), ap = tmem + LY::kA1 + st.a * (D / 2), bp = b1 + stage_at + st.b * kPB;
          const uint32_t idesc = st.two ? kIdescS2 : kIdescS1;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            if (leader) ptx::mma_ts2(d, ap + ks * 8, bp + (((ks >> 2) * TB::kBlock + (ks & 3) * 32) >> 4), kHi, idesc, st.onto || ks > 0 ? 1u : 0u);
        }
        if (leader) ptx::mma_commit(&ctl->s_full);
        return true;
      };
      // dP = V dO^T (dO V^T)
      auto issue_dp = [&](int t) {
        const uint32_t at = done + t, stage = at % LY::kStages, b2s = b2 + stage * (TB::kBytes >> 4);
        if (!uwait(&ctl->b2_full[stage], at / LY::kStages & 1) || !(t == 0 ? uwait(&ctl->a_full, pass & 1) : uwait(&ctl->y_free, (at - 1) & 1))) return false;
        ptx::tc_fence_after();
#pragma unroll 1
        for (int p = 0; p < steps_of(kSums); ++p) {
          const Step st = step_of(kSums, p);
          const uint32_t d = tmem + LY::kY + LY::kScores + (st.second ? BN : 0), ap = a2 + st.a * kPA, bp = b2s + st.b * kPB;
          const uint32_t idesc = st.two ? kIdescS2 : kIdescS1;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            if (leader)
              ptx::mma_ss2(d, ap + (((ks >> 2) * TA::kBlock + (ks & 3) * 32) >> 4), kHi, bp + (((ks >> 2) * TB::kBlock + (ks & 3) * 32) >> 4), kHi,
                           idesc, st.onto || ks > 0 ? 1u : 0u);
        }
        if (leader) {
          ptx::mma_commit(&ctl->dp_full);
          ptx::mma_commit(&ctl->b2_free[stage]);
        }
        return true;
      };
      // dV = P^T dO, dK = dS^T Q (dQ = dS K): each once what lay in its place has been read
      auto issue_dv = [&](int t) {
        const uint32_t at = done + t, stage = at % LY::kStages;
        if ((t > 0 && !uwait(&ctl->t2_free, (at - 1) & 1)) || !uwait(&ctl->p_full, at & 1)) return false;
        ptx::tc_fence_after();
        issue_t(LY::kX, b2_mn + stage * (TB::kBytes >> 4));
        if (leader) {
          ptx::mma_commit(&ctl->x_free);
          ptx::mma_commit(&ctl->b2_free[stage]);
          ptx::mma_commit(&ctl->t1_full);
        }
        return true;
      };
      auto issue_dk = [&](int t) {
        const uint32_t at = done + t, stage = at % LY::kStages;
        if (!(KEYS ? uwait(&ctl->t1_free, at & 1) : t == 0 || uwait(&ctl->t2_free, (at - 1) & 1)) || !uwait(&ctl->ds_full, at & 1)) return false;
        ptx::tc_fence_after();
        issue_t(LY::kY, b1_mn + stage * (TB::kBytes >> 4));
        if (leader) {
          ptx::mma_commit(&ctl->y_free);
          ptx::mma_commit(&ctl->b1_free[stage]);
          ptx::mma_commit(&ctl->t2_full);
        }
        return true;
      };
      bool ok = true;
      if (warp == kIssueWarp) {
        // (a second tile of the other side's first operand: S first, so that P is made under dP; else what its place is free for first)
        for (int t = 0; t < n && ok; ++t) ok = LY::kStages == 2 ? issue_s(t) && issue_dp(t) : issue_dp(t) && issue_s(t);
      } else if (warp == kIssueWarp + 1) {
        for (int t = 0; t < n && ok; ++t) ok = (!KEYS || issue_dv(t)) && issue_dk(t);
      }
      if (last_pass(careful)) break;
    }
    if (warp == kIssueWarp) {
      ptx::tc_fence_after();
      ptx::tmem_dealloc(tmem, 512);
    }
    if (SPLIT) ptx::cluster_sync(), ptx::cluster_sync();
  }
}

template <int D, MaskForm MASK, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) bwd_f32_kernel(const BwdArgs a, int key_items, int cluster) {
  using LY = Lay<D, MASK>;
  extern __shared__ __align__(1024) uint8_t smem[];
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + LY::kCtl);
  const uint32_t base = ptx::smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (base & 1023) {  // (the swizzle counts from multiples of 1024)
    if (tid == 0 && a.status) atomicOr(a.status, kStatusBadSmemAlign);
    return;
  }
  const int item = SPLIT ? blockIdx.x / cluster : blockIdx.x, rank = SPLIT ? blockIdx.x % cluster : 0;
  const bool keys = item < key_items;
  if (tid == 0) {
    ptx::mbar_init(&ctl->a_full, kWork);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&ctl->b1_full[i], LY::kLoad), ptx::mbar_init(&ctl->b1_free[i], 1);
      ptx::mbar_init(&ctl->b2_full[i], LY::kLoad), ptx::mbar_init(&ctl->b2_free[i], keys ? 2 : 1);  // (dP, and dV)
    }
    ptx::mbar_init(&ctl->s_full, 1);
    ptx::mbar_init(&ctl->dp_full, 1);
    ptx::mbar_init(&ctl->p_full, kWork);
    ptx::mbar_init(&ctl->ds_full, kWork);
    ptx::mbar_init(&ctl->t1_full, 1);
    ptx::mbar_init(&ctl->t2_full, 1);
    ptx::mbar_init(&ctl->x_free, keys ? 1 : kWork);
    ptx::mbar_init(&ctl->y_free, 1);
    ptx::mbar_init(&ctl->t1_free, 128);
    ptx::mbar_init(&ctl->t2_free, keys ? 128 : kWork);
    ptx::mbar_init(&ctl->m_full, 128);
    ptx::mbar_init(&ctl->m_free, kWork);
    ctl->abort_flag = 0, ctl->bad = 0;
    ptx::fence_barrier_init();
  }
  if (warp == kIssueWarp) {
    ptx::tmem_alloc(&ctl->tmem_base, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  ptx::grid_dep_launch();  // (the next kernel may come up: this grid has its TMEM)
  ptx::grid_dep_wait();    // launched early behind the delta pre-pass
  if (keys)
    walk<D, true, MASK, SPLIT>(a, smem, base, ctl, tmem, item, rank, cluster);
  else
    walk<D, false, MASK, SPLIT>(a, smem, base, ctl, tmem, item - key_items, rank, cluster);
}

// ------------------------------------------------------------------------------------------------------- dQ of dS --
// A CTA owns 128 rows of queries and walks the 64-key tiles that they see: dQ += dS K.
//   warps 0-7    dS, copied into shared memory a tile ahead, into its pieces (thread r of a warpgroup row r, half the columns each), which
//                go to TMEM; then the product of the tile before into the sums (half the columns of dQ each)
//   warps 8-11   K tiles into their pieces
//   warp 12      issues the MMAs
constexpr int kDqThreads = 512;
template <int D>
struct DqLay {
  using TB = Tile<BN, D, 128>;
  static constexpr bool kWide = D == 64;
  static constexpr int kDs = BM * BN * 4;  // bytes of a tile of dS
  static constexpr int kB = 0, kS = 2 * TB::kBytes, kCtl = kS + 2 * kDs, kBytes = kCtl + 128, kLdO = D + 4;
  static constexpr uint32_t kA = 0, kBufA = 96, kT = 2 * kBufA, kBufT = 128;
  static_assert(BM * kLdO * 4 <= kCtl, "sums over the tiles");
};
struct DqCtl {
  uint64_t a_full[2], t_full[2], b_full[2], b_free[2];
  uint32_t tmem_base;
  int abort_flag, bad;
};
static_assert(sizeof(DqCtl) <= 128, "control block");

template <int D, bool SPLIT>
__global__ void __launch_bounds__(kDqThreads, 1) bwd_f32_dq_kernel(const BwdArgs a, int cluster) {
  using LY = DqLay<D>;
  using TB = typename LY::TB;
  extern __shared__ __align__(1024) uint8_t smem[];
  DqCtl* ctl = reinterpret_cast<DqCtl*>(smem + LY::kCtl);
  const uint32_t base = ptx::smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5;
  volatile int* abort_flag = &ctl->abort_flag;
  if (base & 1023) {  // (the swizzle counts from multiples of 1024)
    if (tid == 0 && a.status) atomicOr(a.status, kStatusBadSmemAlign);
    return;
  }
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&ctl->a_full[i], kWork);
      ptx::mbar_init(&ctl->t_full[i], 1);
      ptx::mbar_init(&ctl->b_full[i], 128);
      ptx::mbar_init(&ctl->b_free[i], 1);
    }
    ctl->abort_flag = 0, ctl->bad = 0;
    ptx::fence_barrier_init();
  }
  if (warp == 12) {
    ptx::tmem_alloc(&ctl->tmem_base, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();  // launched early behind the key CTAs, which leave dS

  const int group = a.Hq / a.Hkv, rows = a.Lq * group, heads = a.B * a.Hkv;
  const int item = SPLIT ? blockIdx.x / cluster : blockIdx.x, rank = SPLIT ? blockIdx.x % cluster : 0;
  const int mt = (rows + BM - 1) / BM - 1 - item / heads;  // under a causal mask the last tiles are longest
  const int hk = item % heads % a.Hkv, b = item % heads / a.Hkv, own0 = mt * BM;
  const Group rw(group, rows);
  int kv_len = a.Skv;
  if (a.kv_lens) {
    const int l = a.kv_lens[b];
    kv_len = l < 0 ? 0 : (l < a.Skv ? l : a.Skv);
  }
  const int shift = causal_shift(a.causal, kv_len, a.Lq);
  const int kv_end = a.causal ? max(0, min(kv_len, rw.query(min(own0 + BM, rows) - 1) + shift + 1)) : kv_len;
  const int all_tiles = (kv_end + BN - 1) / BN;
  const int begin = SPLIT ? all_tiles * rank / cluster : 0, n = (SPLIT ? all_tiles * (rank + 1) / cluster : all_tiles) - begin;
  auto uwait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity & 1, abort_flag)) != 0; };
  auto last_pass = [&](bool careful) {  // by all threads at the end of a pass (see walk)
    ptx::named_barrier(1, kDqThreads);
    return !ctl->bad || careful || n == 0 || *abort_flag;
  };

  if (warp < 8) {
    const int wg = warp >> 2, r = tid & 127, j0 = wg * 32;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    // keys that the row sees: what lies behind has not been written
    const int limit = own0 + r < rows ? (a.causal ? min(kv_len, rw.query(own0 + r) + shift + 1) : kv_len) : 0;
    const int pitch = ds_pitch(a), n_rows = ds_rows(a) - own0;
    const float* ds = ds_of(a, b, hk) + static_cast<int64_t>(own0) * pitch;
    auto fetch = [&](int t) {  // two rows of 64 floats a warp at a time, neighbouring vectors exchanged by row
      const int ch = tid % 16;
#pragma unroll
      for (int i = 0; i < BM / 16; ++i) {
        const int row = tid / 16 + i * 16;
        const bool in = row < n_rows;
        ptx::cp_async16(base + LY::kS + (t & 1) * LY::kDs + row * BN * 4 + ((ch ^ (row & 7)) << 4),
                        ds + static_cast<int64_t>(in ? row : 0) * pitch + (begin + t) * BN + ch * 4, in ? 16 : 0);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float2 acc[D / 4];
    bool careful = false;
    for (int done = 0;; done += n, careful = true) {
#pragma unroll
      for (int j = 0; j < D / 4; ++j) acc[j] = make_float2(0.f, 0.f);
      float2 odd = make_float2(0.f, 0.f);
      auto take = [&](uint32_t at) {  // a tile's product into the sums
        if (!uwait(&ctl->t_full[at & 1], at >> 1)) return;
        ptx::tc_fence_after();
        const uint32_t from = tmem + LY::kT + (at & 1) * LY::kBufT + lane_base + wg * (D / 2);
#pragma unroll
        for (int j = 0; j < D / 4; j += 8) {
          uint32_t o[16], o2[16];
          ptx::tmem_ld16(from + 2 * j, o);
          if (LY::kWide) ptx::tmem_ld16(from + D + 2 * j, o2);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e)
            acc[j + e] = ptx::add2(acc[j + e], LY::kWide ? ptx::add2(floats2(o, 2 * e), floats2(o2, 2 * e)) : floats2(o, 2 * e));
        }
        ptx::tc_fence_before();
      };
      if (n > 0) fetch(0);
      for (int t = 0; t < n; ++t) {  // (to its end even if a wait runs out: the others come to the barrier)
        const uint32_t at = done + t;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        ptx::named_barrier(2, kWork);  // the tile is there, and the other place has been read
        if (t + 1 < n) fetch(t + 1);
        const uint32_t from = base + LY::kS + (t & 1) * LY::kDs + r * BN * 4;
        const uint32_t to = tmem + LY::kA + (at & 1) * LY::kBufA + lane_base;
#pragma unroll
        for (int j = 0; j < 32; j += 16) {
          float x[16];
#pragma unroll
          for (int e = 0; e < 16; e += 4) {
            const float4 v = ptx::ld_shared_f4(from + (((j0 + j + e) / 4 ^ (r & 7)) << 4));
            x[e] = v.x, x[e + 1] = v.y, x[e + 2] = v.z, x[e + 3] = v.w;
          }
          const int col0 = (begin + t) * BN + j0 + j;
          if (col0 + 16 > limit) {
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (col0 + e >= limit) x[e] = 0.f;
          }
          uint32_t w[kPieces][8];
          if (rare(careful)) {
#pragma unroll
            for (int e = 0; e < 8; ++e) split2<true>(x[2 * e], x[2 * e + 1], w[0][e], w[1][e], w[2][e], odd);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) split2<false>(x[2 * e], x[2 * e + 1], w[0][e], w[1][e], w[2][e], odd);
          }
#pragma unroll
          for (int i = 0; i < kPieces; ++i) ptx::tmem_st8(to + i * 32 + (j0 + j) / 2, w[i]);
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive(&ctl->a_full[at & 1]);  // (the product of two tiles before, in the same place, has been taken)
        if (t > 0) take(at - 1);
      }
      if (n > 0) take(done + n - 1);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (was_odd(odd)) ctl->bad = 1;
      if (last_pass(careful)) break;
    }
    float* out_s = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int j = 0; j < D / 4; j += 2)
      *reinterpret_cast<float4*>(out_s + r * LY::kLdO + wg * (D / 2) + 2 * j) =
          make_float4(acc[j].x * a.scale, acc[j].y * a.scale, acc[j + 1].x * a.scale, acc[j + 1].y * a.scale);
    auto store = [&](int row, int d, const float4& x) {
      if (own0 + row < rows)
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.dq) + b * a.dqs.b + (hk * group + rw.head(own0 + row)) * a.dqs.h +
                                   rw.query(own0 + row) * a.dqs.s + d) = x;
    };
    const int d = tid % (D / 4) * 4;
    if constexpr (SPLIT) {
      ptx::cluster_sync();
      constexpr int kMost = 8;
      const int share = (BM + cluster - 1) / cluster, first = rank * share, own = min(share, BM - first);
#pragma unroll 1
      for (int e = tid / (D / 4); e < own; e += kWork / (D / 4)) {
        const uint32_t at = ptx::smem_u32(out_s + (first + e) * LY::kLdO + d);
        float4 x[kMost], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kMost; ++i)
          if (i < cluster) x[i] = ptx::ld_cluster_f4(ptx::map_rank(at, i));
#pragma unroll
        for (int i = 0; i < kMost; ++i)
          if (i < cluster) sum.x += x[i].x, sum.y += x[i].y, sum.z += x[i].z, sum.w += x[i].w;
        store(first + e, d, sum);
      }
      ptx::cluster_sync();  // no CTA leaves while another still reads its share
    } else {
      ptx::named_barrier(2, kWork);
#pragma unroll 4
      for (int e = tid / (D / 4); e < BM; e += kWork / (D / 4)) store(e, d, *reinterpret_cast<const float4*>(out_s + e * LY::kLdO + d));
    }
    if (tid == 0 && *abort_flag && a.status) atomicOr(a.status, kStatusWaitExpired);
  } else if (warp < 12) {
    const int lt = tid & 127;
    const float* k = reinterpret_cast<const float*>(a.k) + b * a.ks.b + hk * a.ks.h + TB::col(lt);
    constexpr int kHeld = TB::kChunks;
    float4 raw[kHeld][2];
    auto fetch = [&](int t, int i) {
      const int row = (begin + t) * BN + TB::row(lt, i);
      const float* p = k + row * a.ks.s;
      raw[i][0] = load4_or_zero(p, row < kv_len), raw[i][1] = load4_or_zero(p + 4, row < kv_len);
    };
    bool careful = false;
    for (int done = 0;; done += n, careful = true) {
      float2 odd = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kHeld; ++i)
        if (n > 0) fetch(0, i);
      for (int t = 0; t < n; ++t) {
        const uint32_t at = done + t, stage = at & 1, use = at >> 1;
        if (use > 0 && !uwait(&ctl->b_free[stage], use - 1)) break;
#pragma unroll
        for (int i = 0; i < TB::kChunks; i += 2)
          TB::put(base + LY::kB + stage * TB::kBytes, lt, i, reinterpret_cast<const float4(&)[2][2]>(raw[i]), careful, odd);
#pragma unroll
        for (int i = 0; i < kHeld; ++i)
          if (t + 1 < n) fetch(t + 1, i);
        ptx::fence_proxy_async_smem();
        ptx::mbar_arrive(&ctl->b_full[stage]);
      }
      if (was_odd(odd)) ctl->bad = 1;
      if (last_pass(careful)) break;
    }
    if (SPLIT) ptx::cluster_sync(), ptx::cluster_sync();
  } else {
    bool careful = false;
    for (int done = 0;; done += n, careful = true) {
      const bool leader = ptx::elect_one();
      constexpr uint32_t kIdesc1 = ptx::make_idesc_f16(BM, D, 1, 0, 1), kIdesc2 = ptx::make_idesc_f16(BM, 2 * D, 1, 0, 1);
      constexpr uint32_t kHi = ptx::smem_desc_hi_sw128(1024), kPB = TB::kPlane >> 4;
      const uint32_t b_mn = ptx::smem_desc_lo(base + LY::kB, LY::kWide ? TB::kPlane : TB::kBlock);
      for (int t = 0; warp == 12 && t < n; ++t) {
        const uint32_t at = done + t, two = at & 1;
        if (!uwait(&ctl->b_full[two], at >> 1) || !uwait(&ctl->a_full[two], at >> 1)) break;
        ptx::tc_fence_after();
        constexpr Sums kSumsT = LY::kWide ? kTwoSums : kOneSum;
#pragma unroll 1
        for (int p = 0; p < steps_of(kSumsT); ++p) {
          const Step st = step_of(kSumsT, p);
          const uint32_t d = tmem + LY::kT + two * LY::kBufT + (st.second ? D : 0), ap = tmem + LY::kA + two * LY::kBufA + st.a * 32;
          const uint32_t bp = b_mn + two * (TB::kBytes >> 4) + st.b * kPB, idesc = st.two ? kIdesc2 : kIdesc1;
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            if (leader) ptx::mma_ts2(d, ap + ks * 8, bp + ks * (2048 >> 4), kHi, idesc, st.onto || ks > 0 ? 1u : 0u);
        }
        if (leader) {
          ptx::mma_commit(&ctl->b_free[two]);
          ptx::mma_commit(&ctl->t_full[two]);
        }
      }
      if (last_pass(careful)) break;
    }
    if (warp == 12) {
      ptx::tc_fence_after();
      ptx::tmem_dealloc(tmem, 512);
    }
    if (SPLIT) ptx::cluster_sync(), ptx::cluster_sync();
  }
}

template <int D, MaskForm MASK>
cudaError_t launch_t(const BwdArgs& a, int cluster, int device, cudaStream_t stream) {
  auto kern = cluster > 1 ? bwd_f32_kernel<D, MASK, true> : bwd_f32_kernel<D, MASK, false>;
  const long long heads = static_cast<long long>(a.B) * a.Hkv;
  const long long key_items = a.dk || a.dv ? heads * ((a.Skv + BM - 1) / BM) : 0;
  const long long query_items = a.dq && !a.ds ? heads * ((static_cast<long long>(a.Lq) * (a.Hq / a.Hkv) + BM - 1) / BM) : 0;
  const long long ctas = (key_items + query_items) * cluster;
  if (ctas > 0x7fffffffll) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  return launch_early(kern, dim3(static_cast<unsigned>(ctas)), dim3(kThreads), Lay<D, MASK>::kBytes, stream, cluster, a,
                      static_cast<int>(key_items), cluster);
}

// CTAs per cluster, that share a walk: what is expected to take the least time, with one CTA to an SM, items whose walk takes `step_us` a
// tile and whose rest `item_us`.  `walk` and `mean`: the longest and the average walk in tiles.  Measured, us, undivided -> chosen: D = 64,
// causal 3 x 1000 58 -> 32 (3), 2 x 16/2 heads x 700 causal 314 -> 85 (6), 2 x 4 x 128 14.6 (2: 17.1); D = 128, 8/1 heads x 33 on 1000 104 -> 25 (8).
struct Items {
  double count, walk, mean, step_us;
};
struct Plan {
  int cluster;
  double us;
};
Plan plan_of(const Items& x, const Items& y, double item_us, double merge_us, int device) {
  Plan best{1, 1e30};
  for (int c = 1; c <= 8; ++c) {
    const int room = cluster_room(device, c);
    if (room <= 0) continue;
    const double longest = item_us + std::max(x.count > 0 ? std::ceil(x.walk / c) * x.step_us : 0.0, y.count > 0 ? std::ceil(y.walk / c) * y.step_us : 0.0);
    const double all = c * (x.count * (item_us + x.mean / c * x.step_us) + y.count * (item_us + y.mean / c * y.step_us)) / room;
    // (CTAs of one length come in whole rounds)
    const double us = std::max(longest, all + ((x.count + y.count) * c > room ? 0.35 * longest : 0.0)) + (c > 1 ? merge_us : 0.0);
    if (us < best.us) best = Plan{c, us};
  }
  return best;
}

// dQ by CTAs of its own, in one launch with those of dK and dV, or of their dS in another: what is expected to take less.  The constants are fitted to
// 148 calls timed both ways (35 shapes, plain, causal, with boolean and additive masks); the choice is the faster way but for four, by 2, 3, 3 and 20 % (D = 64,
// 3 x 1000: 40 stored, 48 as clusters for which there is no room at once).
// us, recomputed and stored: D = 64, 4 x 8 heads x 500 63.0 and 58.2, causal 45.4 and 56.0, additive mask 83 and 77, 16 x 16 x 128 causal 55.6 and 49.1,
// 3 x 1000 causal 31.6 and 40.2, boolean mask 50.9 and 44.1, 2 x 16/2 x 700 204 and 151 with it; D = 128, 4 x 8 x 500 123 and 109, causal 90 and 97, additive
// mask 169 and 142, 3 x 1000 causal 52.7 and 57.8, 4 x 8 x 200 43 and 47, additive 59 and 53, 8 x 8 x 512 252 and 221.
struct Plans {
  Plan recomputed, stored, dq;
  bool take_ds;
};
Plans plans_of(int D, const BwdArgs& a, int device) {
  const double heads = static_cast<double>(a.B) * a.Hkv, rows = static_cast<double>(a.Lq) * (a.Hq / a.Hkv);
  const double key_walk = std::ceil(rows / BN), query_walk = std::ceil(static_cast<double>(a.Skv) / BN);
  const double seen = a.causal == TT_ATTN_CAUSAL_TOP_LEFT ? 0.5 : 1.0;  // of all tiles
  const double mask = a.mask.ptr ? (D == 64 ? 0.8 : 2.6) : 0.0;          // us a tile, of both walks
  const Items keys{a.dk || a.dv ? heads * std::ceil(static_cast<double>(a.Skv) / BM) : 0.0, key_walk, seen * key_walk, (D == 64 ? 3.25 : 6.9) + mask};
  Items queries{a.dq ? heads * std::ceil(rows / BM) : 0.0, query_walk, seen * query_walk, (D == 64 ? 1.87 : 4.6) + mask};
  const double item = D == 64 ? 9.54 : 14.8, merge = D == 64 ? 4.0 : 3.0;
  const Items none{0.0, 0.0, 0.0, 0.0};
  Plans p{plan_of(keys, queries, item, merge, device), plan_of(keys, none, item, merge, device), {1, 0.0}, false};
  // The pass that reads dS, where the two launches take less than the one.
  queries.step_us = D == 64 ? 1.61 : 2.35;
  p.dq = plan_of(queries, none, D == 64 ? 5.2 : 7.6, 3.0, device);
  p.take_ds = p.stored.us + p.dq.us < p.recomputed.us;
  return p;
}

template <int D>
cudaError_t launch_d(const BwdArgs& a, int cluster, int device, cudaStream_t stream) {
  if (!a.mask.ptr) return launch_t<D, kNoMask>(a, cluster, device, stream);
  return a.mask.kind == TT_ATTN_MASK_BOOL ? launch_t<D, kBoolMask>(a, cluster, device, stream)
                                          : launch_t<D, kAddMask>(a, cluster, device, stream);
}

template <int D>
cudaError_t launch_dq(const BwdArgs& a, int cluster, int device, cudaStream_t stream) {
  auto kern = cluster > 1 ? bwd_f32_dq_kernel<D, true> : bwd_f32_dq_kernel<D, false>;
  const long long ctas = (static_cast<long long>(a.Lq) * (a.Hq / a.Hkv) + BM - 1) / BM * a.Hkv * a.B * cluster;
  if (ctas > 0x7fffffffll) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  return launch_early(kern, dim3(static_cast<unsigned>(ctas)), dim3(kDqThreads), DqLay<D>::kBytes, stream, cluster, a, cluster);
}

}  // namespace

constexpr double kPairBytes = BN * BN * sizeof(float);
double bwd_ds_bytes_of(int B, int Hq, int Lq, int Skv) {
  return static_cast<double>(B) * Hq * ((Lq + BN - 1) / BN) * ((Skv + BN - 1) / BN) * kPairBytes;
}
// Where there is room for dS, dQ is one product more instead of three, by a kernel of its own: 16 KB of scratch for 64 queries and 64
// keys, written and read once.  Up to 192 MB of it, and from as many pairs of tiles on as storing can pay for (whether it does is the plan's, which knows
// the device, causal form and mask).  us, recomputed and stored: D = 64, 256 pairs (2 x 8 x 256) 21.2 and 26.5 causal, additive mask 25.4 and 29.2, 512
// (16 x 8 x 128) 31.2 and 27.5, 36.3 and 31.7; D = 128, 256 pairs 33.4 and 36.0, 41.4 and 40.2, 512 52.3 and 46.8, 62.6 and 52.0.
size_t bwd_ds_bytes(int B, int Hq, int Hkv, int Lq, int Skv, int D) {
  if (B <= 0 || Hq <= 0 || Lq <= 0 || Skv <= 0) return 0;
  const double bytes = bwd_ds_bytes_of(B, Hq, Lq, Skv);
  return bytes <= 192e6 && bytes >= (D == 64 ? 500 : 250) * kPairBytes ? static_cast<size_t>(bytes) : 0;
}

bool bwd_f32_takes_ds(int D, const BwdArgs& a, int device) { return plans_of(D, a, device).take_ds; }

cudaError_t launch_bwd_f32(int D, const BwdArgs& args, bool take_ds, int device, cudaStream_t stream) {
  BwdArgs a = args;
  const Plans plans = plans_of(D, a, device);
  if (!take_ds && !plans.take_ds) a.ds = nullptr;
  const int cluster = a.ds ? plans.stored.cluster : plans.recomputed.cluster;
  cudaError_t e = launch_bwd_delta(TT_ATTN_F32, D, a, stream);
  if (e == cudaSuccess) e = D == 64 ? launch_d<64>(a, cluster, device, stream) : launch_d<128>(a, cluster, device, stream);
  if (e != cudaSuccess || !a.ds) return e;
  return D == 64 ? launch_dq<64>(a, plans.dq.cluster, device, stream) : launch_dq<128>(a, plans.dq.cluster, device, stream);
}

}  // namespace ttattn
