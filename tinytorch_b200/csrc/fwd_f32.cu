// Prefill forward for Float32 tensors on the tensor cores: fp32 products as sums of bf16 ones (f32_pieces.cuh).
//
// A CTA owns 128 rows of one (batch, kv head) and walks its 64-key tiles.  The rows are the queries of all heads of the group, query by
// query (row = query * group + head), so that short prompts of grouped-query models fill the tiles.  Roles:
//   warps 0-3    softmax: thread r owns row r (TMEM lane r).  Per key tile S from TMEM, mask, running maximum and sum, P as three bf16
//                planes into TMEM, and the factor that the row's older sums shrink by
//   warps 4-7    O: each tile's P V is read from TMEM and added to the rows' sums in registers
//   warps 8-15   K and V tiles into their pieces: a warpgroup each (D = 64), or both together K first (D = 128, see below)
//   warps 16, 17 issue the MMAs of S and of P V: S of the next tile as soon as the softmax has read this one's, P V of a tile under
//                the softmax of the next.  (One warp for both spends 850 of 3100 clocks per tile in waits for what is there already.)
//   warps 18, 19 masks
// An MMA of 64 columns takes 52 (A from TMEM) or 66 clocks (from shared memory) where 32 would do and 128 columns take 64: the first two planes
// of K (and of V, D = 64) are read as one operand of 128.  S and O come as two sums then (f32_pieces.cuh).
// A probability that is 0 takes part in P V, as in the composition: what is not finite in V spoils the rows that share a tile with it (all 128 that walk
// as far, also those whose causal limit lies before it), and no others.
//
// Bound by the chain of a tile: softmax 2000 clocks and 300 until S is seen (D = 64: a tile 2400, the MMAs under them), for D = 128,
// where only one K tile fits, K into pieces, then S 1800.  Against the same in fp32 FMAs on CUDA cores (64 x 64 tiles, whose FMA pipes were
// 58 % busy), us: D = 64, 4 x 8 heads x 500 72 -> 18.4 (additive mask 74 -> 27, 6 x 333 padding 53 -> 19), causal 16 x 2048 294 -> 54.5,
// 11 x 32/8 heads x 22 14.7 -> 9.1, one query on one key 7.2 -> 6.4, but 2 x 8/4 heads x 99 on 131 with an additive mask 10.4 -> 11.0; D = 128,
// 4 x 8 x 500 117 -> 32 (additive 126 -> 38), causal 4 x 4096 506 -> 107.
// Tried: P over the S that it is made of, two such buffers, S up to two tiles ahead: 2700 clocks a tile.  One place for P: 3150.
// Additive rows by bulk copies of 256 bytes: 29.7 -> 32.3, D = 128 43 -> 53.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cluster_host.cuh"
#include "f32_pieces.cuh"

namespace ttattn {
namespace {

using namespace pieces;
enum MaskForm { kNoMask, kBoolMask, kAddRow, kAddMask };  // kAddRow: additive and the same for all rows of a CTA
constexpr int BM = 128, BN = 64;
constexpr int kThreads = 640, kIssueWarp = 16;

struct Ctl {
  uint64_t q_full, k_full[2], k_free[2], v_full[2], v_free[2], p_full[2], s_full, s_free, o_full, o_free, m_full[2], m_free[2];
  uint32_t tmem_base;
  int abort_flag, bad;
};

template <int D, MaskForm MASK>
struct Lay {
  using TQ = Tile<BM, D, 256>;
  static constexpr int kLoad = D == 64 ? 128 : 256;  // threads that bring a tile
  using TK = Tile<BN, D, kLoad>;
  static constexpr int kStages = D == 64 ? 2 : 1;  // of K, and of V
  static constexpr bool kWideV = D == 64;
  // a boolean mask: two words of bits per row; an additive one: 64 floats, of one row or of each
  static constexpr int kMaskBytes = MASK == kNoMask ? 0 : (MASK == kBoolMask ? BM * 8 : (MASK == kAddRow ? BN * 4 : BM * BN * 4));
  static constexpr int kMaskStages = D == 64 || MASK != kAddMask ? 2 : 1;
  static constexpr int kQ = 0, kK = TQ::kBytes, kV = kK + kStages * TK::kBytes, kM = kV + kStages * TK::kBytes;
  static constexpr int kAlpha = kM + kMaskStages * kMaskBytes;  // [4][128]: the oldest that may still be read is of two tiles before
  static constexpr int kCtl = kAlpha + 4 * BM * 4;
  static constexpr int kBytes = kCtl + 256;
  static constexpr int kLdO = D + 4;  // floats a row of O on its way out, over the planes of Q
  // TMEM: S (two sums of 64 columns); O (one or two sums); two buffers for P, three planes of 32
  static constexpr uint32_t kO = 2 * BN, kP = kO + 128, kBufP = 96;
  static_assert(kP + 2 * kBufP <= 512, "TMEM");
  static constexpr int kSoftmaxRegs = D == 64 ? 128 : 120, kSumRegs = D == 64 ? 112 : 160, kLoadRegs = D == 64 ? 88 : 72, kIssueRegs = D == 64 ? 64 : 56;
  static_assert(kSoftmaxRegs + kSumRegs + 2 * kLoadRegs + kIssueRegs <= 5 * 96, "registers of the launch");
  static_assert(BM * kLdO * 4 + BM * 32 <= TQ::kBytes, "O and the weights over Q");
};
static_assert(sizeof(Ctl) <= 256, "control block");
static_assert(Lay<128, kAddMask>::kBytes <= 227 * 1024 && Lay<128, kAddRow>::kBytes <= 227 * 1024, "shared memory");

template <int D, MaskForm MASK, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) fwd_f32_kernel(const FwdArgs a, int cluster) {
  using LY = Lay<D, MASK>;
  using TQ = typename LY::TQ;
  using TK = typename LY::TK;
  constexpr int kStages = LY::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + LY::kCtl);
  const uint32_t base = ptx::smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort_flag = &ctl->abort_flag;

  if (base & 1023) {  // (the swizzle counts from multiples of 1024)
    if (tid == 0 && a.status) atomicOr(a.status, kStatusBadSmemAlign);
    return;
  }
  if (tid == 0) {
    ptx::mbar_init(&ctl->q_full, 256);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&ctl->k_full[i], LY::kLoad);
      ptx::mbar_init(&ctl->v_full[i], LY::kLoad);
      ptx::mbar_init(&ctl->k_free[i], 1);
      ptx::mbar_init(&ctl->v_free[i], 1);
      ptx::mbar_init(&ctl->p_full[i], BM);
    }
    ptx::mbar_init(&ctl->s_full, 1);
    ptx::mbar_init(&ctl->s_free, BM);
    ptx::mbar_init(&ctl->o_full, 1);
    ptx::mbar_init(&ctl->o_free, BM);
#pragma unroll
    for (int i = 0; i < 2; ++i) ptx::mbar_init(&ctl->m_full[i], 64), ptx::mbar_init(&ctl->m_free[i], BM);
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
  const uint32_t tmem = ctl->tmem_base, tmem_o = tmem + LY::kO;
  ptx::grid_dep_launch();  // (the next kernel may come up: this grid has its TMEM)
  ptx::grid_dep_wait();    // launched early: everything below reads or writes global memory

  // ------------------------------------------------------------------------------------------------ what to do --
  const int group = a.Hq / a.Hkv, rows = a.Lq * group, heads = a.B * a.Hkv;
  const Group gr(group, rows);
  const int item = SPLIT ? blockIdx.x / cluster : blockIdx.x, rank = SPLIT ? blockIdx.x % cluster : 0;
  const int n_mt = (rows + BM - 1) / BM, mt = n_mt - 1 - item / heads;  // under a causal mask the last tiles are longest
  const int hk = item % heads % a.Hkv, b = item % heads / a.Hkv, row0 = mt * BM;
  int kv_len = a.Skv;
  if (a.kv_lens) {
    const int l = a.kv_lens[b];
    kv_len = l < 0 ? 0 : (l < a.Skv ? l : a.Skv);
  }
  const int shift = causal_shift(a.causal, kv_len, a.Lq);
  const int first_q = gr.query(row0), last_q = gr.query(min(row0 + BM, rows) - 1);
  const int kv_end = a.causal ? max(0, min(kv_len, last_q + shift + 1)) : kv_len;
  const int all_edge = a.causal ? min(kv_len, first_q + shift + 1) : kv_len;  // keys before it are seen by all rows
  const int all_tiles = (kv_end + BN - 1) / BN;
  const int t0 = SPLIT ? all_tiles * rank / cluster : 0, n = (SPLIT ? all_tiles * (rank + 1) / cluster : all_tiles) - t0;
  // row r of this CTA's: query and head of the group (rows beyond the last: query Lq, nothing is read or written for them)
  auto query_of = [&](int r) { return gr.query(row0 + r); };
  auto head_of = [&](int r) { return hk * group + gr.head(row0 + r); };

  // One pass, or two: where values that are not finite have been met (in V, or in scores that count), the second splits so that infinities
  // stay what they are.  `done`: tiles before this pass; tile t of a pass has number done + t, from which buffers and barriers' phases follow.
  // (A barrier that may complete again before all have seen it complete exists twice.)
  auto last_pass = [&](bool careful) {  // by all threads at the end of a pass
    ptx::named_barrier(1, kThreads);
    return !ctl->bad || careful || n == 0 || *abort_flag;
  };
  auto uwait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity & 1, abort_flag)) != 0; };
  // Q into its pieces, by warps 0-7
  auto stage_q = [&](bool careful) {
    float2 odd = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int i0 = 0; i0 < TQ::kChunks && n > 0; i0 += 4) {
      float4 x[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = TQ::row(tid, i0 + i), i_q = query_of(r);
        const float* p = reinterpret_cast<const float*>(a.q) + b * a.qs.b + head_of(r) * a.qs.h + static_cast<int64_t>(i_q) * a.qs.s + TQ::col(tid);
        x[i][0] = load4_or_zero(p, i_q < a.Lq), x[i][1] = load4_or_zero(p + 4, i_q < a.Lq);
      }
#pragma unroll
      for (int i = 0; i < 4; i += 2) TQ::put(base + LY::kQ, tid, i0 + i, reinterpret_cast<const float4(&)[2][2]>(x[i]), careful, odd);
    }
    ptx::fence_proxy_async_smem();
    ptx::mbar_arrive(&ctl->q_full);
  };
  // O, where warps 0-7 find it: [row][kLdO] over the planes of Q; maxima and sums (or their inverses) over the alphas, [2][128]
  float* out_s = reinterpret_cast<float*>(smem);
  float* stat = reinterpret_cast<float*>(smem + LY::kAlpha);
  float* lse = a.lse ? a.lse + static_cast<int64_t>(b) * a.Hq * a.Lq : nullptr;
  auto store = [&](int r, int d, const float4& x) {
    const int i_q = query_of(r);
    if (i_q < a.Lq)
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.o) + b * a.os.b + head_of(r) * a.os.h + static_cast<int64_t>(i_q) * a.os.s + d) = x;
  };
  // Warps 0-7, once O and the rows' numbers are in shared memory.
  auto write_out = [&]() {
    const int d = tid % (D / 4) * 4;
    constexpr int kStep = 256 / (D / 4);  // rows at a time
    if constexpr (SPLIT) {
      // the shares of the cluster's CTAs, added in rank order; every CTA writes a share of the rows
      constexpr int kMost = 8;
      ptx::cluster_sync();
      const int share = (BM + cluster - 1) / cluster, first = rank * share, own = min(share, BM - first);
      float* weight = out_s + BM * LY::kLdO;  // [row][CTA]
      if (tid < own) {
        const int r = first + tid;
        float m[kMost], l[kMost], mx = -INFINITY, ls = 0.f;
#pragma unroll
        for (int p = 0; p < kMost; ++p)
          if (p < cluster) {
            m[p] = ptx::ld_cluster_f1(ptx::map_rank(ptx::smem_u32(stat + r), p));
            l[p] = ptx::ld_cluster_f1(ptx::map_rank(ptx::smem_u32(stat + BM + r), p));
            mx = fmaxf(mx, m[p]);
          }
        const float ref = mx == -INFINITY ? 0.f : mx;
#pragma unroll
        for (int p = 0; p < kMost; ++p)
          if (p < cluster) ls += l[p] * exp2f(m[p] - ref);
        const float inv = ls > 0.f ? 1.f / ls : 0.f;
#pragma unroll
        for (int p = 0; p < kMost; ++p)
          if (p < cluster) weight[tid * kMost + p] = exp2f(m[p] - ref) * inv;
        if (lse && query_of(r) < a.Lq)
          lse[static_cast<int64_t>(head_of(r)) * a.Lq + query_of(r)] = ls > 0.f ? (mx + log2f(ls)) * kLn2 : -INFINITY;
      }
      ptx::named_barrier(2, 256);
#pragma unroll 1
      for (int r = tid / (D / 4); r < own; r += kStep) {
        float4 x[kMost], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int p = 0; p < kMost; ++p)
          if (p < cluster) x[p] = ptx::ld_cluster_f4(ptx::map_rank(ptx::smem_u32(out_s + (first + r) * LY::kLdO + d), p));
#pragma unroll
        for (int p = 0; p < kMost; ++p)
          if (p < cluster) {
            const float w = weight[r * kMost + p];
            sum.x = fmaf(x[p].x, w, sum.x), sum.y = fmaf(x[p].y, w, sum.y), sum.z = fmaf(x[p].z, w, sum.z), sum.w = fmaf(x[p].w, w, sum.w);
          }
        store(first + r, d, sum);
      }
      ptx::cluster_sync();  // no CTA leaves while another still reads its share
    } else {
      ptx::named_barrier(2, 256);
#pragma unroll 4
      for (int r = tid / (D / 4); r < BM; r += kStep) {
        const float4 x = *reinterpret_cast<const float4*>(out_s + r * LY::kLdO + d);
        const float inv = stat[BM + r];
        store(r, d, make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv));
      }
    }
    if (tid == 0 && *abort_flag && a.status) atomicOr(a.status, kStatusWaitExpired);
  };
  // Nothing follows where the roles' ways meet: a warp that has given registers back must not come to code that is compiled for more.

  if (warp < 4) {
    // ------------------------------------------------------------------------------------------------ softmax --
    ptx::setmaxnreg_inc<LY::kSoftmaxRegs>();
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const int limit = a.causal ? min(kv_len, query_of(tid) + shift + 1) : kv_len;  // keys that the row sees
    float c = fabsf(a.scale) * kLog2e;
    if (c < 1e-45f) c = 1e-45f;  // (never zero: a hidden score's -inf times it stays one)
    constexpr bool SCALED = MASK == kAddRow || MASK == kAddMask;  // scores are multiplied by c before the maximum is taken
    float m_row, l_row;
    bool careful = false;
    for (int done = 0;; done += n, careful = true) {
      stage_q(careful);
      m_row = -INFINITY, l_row = 0.f;
      for (int t = 0; t < n; ++t) {
        const uint32_t at = done + t, two = at & 1, p_at = tmem + LY::kP + two * LY::kBufP + lane_base;
        const int col0 = (t0 + t) * BN;
        if (!uwait(&ctl->s_full, at)) break;
        ptx::tc_fence_after();
        float s[BN];
#pragma unroll
        for (int j = 0; j < BN; j += 32) {
          uint32_t x[32], y[32];
          ptx::tmem_ld32(tmem + lane_base + j, x);
          ptx::tmem_ld32(tmem + lane_base + BN + j, y);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float2 z = ptx::add2(make_float2(__uint_as_float(x[e]), __uint_as_float(x[e + 1])),
                                       make_float2(__uint_as_float(y[e]), __uint_as_float(y[e + 1])));
            s[j + e] = z.x, s[j + e + 1] = z.y;
          }
        }
        ptx::tc_fence_before();
        ptx::mbar_arrive(&ctl->s_free);
        if constexpr (MASK != kNoMask) {
          const uint32_t stage = at % LY::kMaskStages, mask_at = base + LY::kM + stage * LY::kMaskBytes;
          if (!uwait(&ctl->m_full[stage], at / LY::kMaskStages)) break;
          if constexpr (MASK == kBoolMask) {
            uint32_t seen[2];
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(seen[0]), "=r"(seen[1]) : "r"(mask_at + tid * 8) : "memory");
#pragma unroll
            for (int j = 0; j < BN; ++j)
              if (!(seen[j / 32] >> (j % 32) & 1)) s[j] = -INFINITY;
          } else {
#pragma unroll
            for (int j = 0; j < BN; j += 4) {
              const float4 m4 = ptx::ld_shared_f4(mask_at + (MASK == kAddRow ? j * 4 : tid * BN * 4 + (((j / 4) ^ (tid & 7)) << 4)));
              if constexpr (D == 64) {  // (29.8 -> 28.6, 2048 queries 56.8 -> 54.0; D = 128, with fewer registers, 43.6 -> 44.1 and 82.2 -> 81.1)
                const float2 c2 = make_float2(c, c), log2e = make_float2(kLog2e, kLog2e);
                const float2 lo = ptx::fma2(make_float2(m4.x, m4.y), log2e, ptx::mul2(make_float2(s[j], s[j + 1]), c2));
                const float2 hi = ptx::fma2(make_float2(m4.z, m4.w), log2e, ptx::mul2(make_float2(s[j + 2], s[j + 3]), c2));
                s[j] = lo.x, s[j + 1] = lo.y, s[j + 2] = hi.x, s[j + 3] = hi.y;
              } else {
                const float mk[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) s[j + e] = fmaf(mk[e], kLog2e, s[j + e] * c);
              }
            }
          }
          ptx::mbar_arrive(&ctl->m_free[stage]);
        }
        if (col0 + BN > all_edge) {
#pragma unroll
          for (int j = 0; j < BN; ++j)
            if (col0 + j >= limit) s[j] = -INFINITY;
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int j = 0; j < BN; j += 8)
#pragma unroll
          for (int e = 0; e < 4; ++e) mx[e] = ptx::max3(mx[e], s[j + e], s[j + 4 + e]);
        float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        if (!SCALED) top *= c;
        const float m_new = fmaxf(m_row, top);
        // a row that has seen no participating key yet keeps m = -inf; its exponentials are taken against 0 and are all 0
        const float m_use = m_new == -INFINITY ? 0.f : m_new;
        const float alpha = exp2f(m_row - m_use);
        m_row = m_new;
        reinterpret_cast<float*>(smem + LY::kAlpha)[(at & 3) * BM + tid] = alpha;
        float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        const float2 c2 = make_float2(c, c), neg2 = make_float2(-m_use, -m_use);
        auto probabilities = [&](auto keep_signs, const float* sp, int j) {  // of 16 scores, those of columns j ..
          uint32_t ph[8], pm[8], pl[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float2 sc = make_float2(sp[2 * e], sp[2 * e + 1]);
            const float2 y = SCALED ? ptx::add2(sc, neg2) : ptx::fma2(sc, c2, neg2);
            const float2 p = make_float2(ptx::ex2(y.x), ptx::ex2(y.y));
            sum[e & 1] = ptx::add2(sum[e & 1], p);
            split2<decltype(keep_signs)::value>(p.x, p.y, ph[e], pm[e], pl[e]);
          }
          ptx::tmem_st8(p_at + j / 2, ph);
          ptx::tmem_st8(p_at + 32 + j / 2, pm);
          ptx::tmem_st8(p_at + 64 + j / 2, pl);
        };
        if (t >= 2) {  // P of two tiles before has been read
          if (!uwait(&ctl->v_free[two], (at - 2) >> 1)) break;
          ptx::tc_fence_after();
        }
        if (rare(careful)) {
          // Its code stands once, and s moves up: four times it costs the other pass registers (additive mask, 4 x 8 heads x 500: 28.7 us,
          // boolean 23.5; once 27.8 and 22.8; D = 128, 4 x 4096 causal 110.7 and 107.3).  D = 64 without a mask has it four times: 18.3; once 18.7.
#pragma unroll(MASK == kNoMask && D == 64 ? 4 : 1)
          for (int j = 0; j < BN; j += 16) {
            probabilities(std::true_type{}, s, j);
#pragma unroll
            for (int e = 0; e < BN - 16; ++e) s[e] = s[e + 16];
          }
        } else {
#pragma unroll
          for (int j = 0; j < BN; j += 16) probabilities(std::false_type{}, s + j, j);
        }
        sum[0] = ptx::add2(sum[0], sum[1]);
        l_row = fmaf(l_row, alpha, sum[0].x + sum[0].y);
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        ptx::mbar_arrive(&ctl->p_full[two]);
      }
      if (l_row != l_row) ctl->bad = 1;  // (what is hidden may be anything)
      if (last_pass(careful)) break;
    }
    stat[tid] = m_row, stat[BM + tid] = SPLIT ? l_row : (l_row > 0.f ? 1.f / l_row : 0.f);
    if (!SPLIT && lse && query_of(tid) < a.Lq)
      lse[static_cast<int64_t>(head_of(tid)) * a.Lq + query_of(tid)] = l_row > 0.f ? (m_row + log2f(l_row)) * kLn2 : -INFINITY;
    write_out();
  } else if (warp < 8) {
    // ------------------------------------------------------------------------------------------------------ O --
    ptx::setmaxnreg_inc<LY::kSumRegs>();
    const uint32_t from = tmem_o + (static_cast<uint32_t>((warp - 4) * 32) << 16);
    float2 acc[D / 2];
    bool careful = false;
    for (int done = 0;; done += n, careful = true) {
      stage_q(careful);
#pragma unroll
      for (int j = 0; j < D / 2; ++j) acc[j] = make_float2(0.f, 0.f);
      for (int t = 0; t < n; ++t) {
        const uint32_t at = done + t;
        if (!uwait(&ctl->o_full, at)) break;
        ptx::tc_fence_after();
        const float alpha = reinterpret_cast<const float*>(smem + LY::kAlpha)[(at & 3) * BM + tid - 128];
        const float2 alpha2 = make_float2(alpha, alpha);
#pragma unroll
        for (int j = 0; j < D; j += 16) {
          uint32_t x[16], y[16];
          ptx::tmem_ld16(from + j, x);
          if (LY::kWideV) ptx::tmem_ld16(from + D + j, y);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float2 z = make_float2(__uint_as_float(x[2 * e]), __uint_as_float(x[2 * e + 1]));
            acc[j / 2 + e] = ptx::fma2(acc[j / 2 + e], alpha2,
                                       LY::kWideV ? ptx::add2(z, make_float2(__uint_as_float(y[2 * e]), __uint_as_float(y[2 * e + 1]))) : z);
          }
        }
        ptx::tc_fence_before();
        ptx::mbar_arrive(&ctl->o_free);
      }
      if (last_pass(careful)) break;
    }
#pragma unroll
    for (int j = 0; j < D / 2; j += 2)
      *reinterpret_cast<float4*>(out_s + (tid - 128) * LY::kLdO + 2 * j) = make_float4(acc[j].x, acc[j].y, acc[j + 1].x, acc[j + 1].y);
    write_out();
  } else if (warp < kIssueWarp) {
    // --------------------------------------------------------------------------------------------- K or V, by tile --
    ptx::setmaxnreg_dec<LY::kLoadRegs>();
    // A thread's chunks of a tile are in flight together, asked for as those of the tile before leave the registers, and are
    // converted two at a time.  (Each asked for as the one before leaves: D = 128 34.5 -> 38 us, 4 x 8 heads x 500; K's next tile as it is in
    // shared memory: 42.6.)
    // D = 128: K's tiles have one place, and wait for it: a tile's time is K into its place, 2500 clocks by one warpgroup, and S,
    // 1800.  Both warpgroups bring K, then V.
    constexpr bool kBoth = D == 128;
    const bool keys = !kBoth && warp < 12;
    const int ht = tid & (LY::kLoad - 1);
    const float* k = reinterpret_cast<const float*>(a.k) + b * a.ks.b + hk * a.ks.h + TK::col(ht);
    const float* v = reinterpret_cast<const float*>(a.v) + b * a.vs.b + hk * a.vs.h + TK::col(ht);
    static_assert(TK::kChunks == 4, "chunks of a thread");
    float4 raw[4][2];
    auto fetch = [&](bool of_k, int t) {  // rows at or beyond the length are zero
      const float* src = of_k ? k : v;
      const int64_t stride = of_k ? a.ks.s : a.vs.s;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = (t0 + t) * BN + TK::row(ht, i);
        const float* p = src + static_cast<int64_t>(r) * stride;
        raw[i][0] = load4_or_zero(p, r < kv_len), raw[i][1] = load4_or_zero(p + 4, r < kv_len);
      }
    };
    bool careful = false;
    for (int done = 0;; done += n, careful = true) {
      float2 odd = make_float2(0.f, 0.f);
      auto put = [&](bool of_k, int t) {  // false: a wait has run out
        const uint32_t at = done + t, stage = at % kStages, last = at - kStages;
        if (t >= kStages) {  // the stage's last user has been read
          if (!uwait(of_k ? &ctl->k_free[last & 1] : &ctl->v_free[last & 1], last >> 1)) return false;
        }
        const uint32_t dst = base + (of_k ? LY::kK : LY::kV) + stage * TK::kBytes;
        float2 seen = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; i += 2) TK::put(dst, ht, i, reinterpret_cast<const float4(&)[2][2]>(raw[i]), careful, seen);
        if (!of_k) odd = ptx::add2(odd, seen);
        ptx::fence_proxy_async_smem();
        ptx::mbar_arrive(of_k ? &ctl->k_full[stage] : &ctl->v_full[stage]);
        return true;
      };
      if (n > 0) fetch(kBoth || keys, 0);
      for (int t = 0; t < n; ++t) {
        if (!put(kBoth || keys, t)) break;
        if (kBoth) {
          fetch(false, t);
          if (!put(false, t)) break;
        }
        if (t + 1 < n) fetch(kBoth || keys, t + 1);
      }
      if (was_odd(odd)) ctl->bad = 1;
      if (last_pass(careful)) break;
    }
    if (SPLIT) ptx::cluster_sync(), ptx::cluster_sync();
  } else {
    // ------------------------------------------------------------------------------------------------- the MMAs --
    ptx::setmaxnreg_dec<LY::kIssueRegs>();
    bool careful = false;
    for (int done = 0, pass = 0;; ++pass, done += n, careful = true) {
      const bool leader = ptx::elect_one();
      // (a negative scale is folded into the sign of Q, so that the softmax works with a positive multiplier)
      const uint32_t idesc_s1 = ptx::make_idesc_f16(BM, BN, 1, 0, 0) | (a.scale < 0.f ? 1u << 13 : 0u);
      const uint32_t idesc_s2 = ptx::make_idesc_f16(BM, 2 * BN, 1, 0, 0) | (a.scale < 0.f ? 1u << 13 : 0u);
      constexpr uint32_t kIdescO1 = ptx::make_idesc_f16(BM, D, 1, 0, 1), kIdescO2 = ptx::make_idesc_f16(BM, 2 * D, 1, 0, 1);
      constexpr uint32_t kHi = ptx::smem_desc_hi_sw128(1024);
      constexpr uint32_t kPQ = TQ::kPlane >> 4, kPK = TK::kPlane >> 4;
      const uint32_t qlo = ptx::smem_desc_lo(base + LY::kQ, 16), klo = ptx::smem_desc_lo(base + LY::kK, 16);
      const uint32_t vlo = ptx::smem_desc_lo(base + LY::kV, LY::kWideV ? TK::kPlane : TK::kBlock);
      constexpr Sums kSumsS = D == 64 ? kLeadApart : kTwoSums, kSumsO = LY::kWideV ? kLeadApart : kOneSum;
      auto issue_qk = [&](uint32_t at) {
        const uint32_t d = tmem, k0 = klo + at % kStages * (TK::kBytes >> 4);
#pragma unroll 1
        for (int p = 0; p < steps_of(kSumsS); ++p) {
          const Step st = step_of(kSumsS, p);
          const uint32_t qo = qlo + st.a * kPQ, ko = k0 + st.b * kPK, to = d + (st.second ? BN : 0), idesc = st.two ? idesc_s2 : idesc_s1;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            if (leader)
              ptx::mma_ss2(to, qo + (((ks >> 2) * TQ::kBlock + (ks & 3) * 32) >> 4), kHi, ko + (((ks >> 2) * TK::kBlock + (ks & 3) * 32) >> 4), kHi,
                           idesc, st.onto || ks > 0 ? 1u : 0u);
        }
        if (leader) {
          ptx::mma_commit(&ctl->k_free[at & 1]);
          ptx::mma_commit(&ctl->s_full);
        }
      };
      auto issue_pv = [&](uint32_t at) {
        const uint32_t p0 = tmem + LY::kP + (at & 1) * LY::kBufP, v0 = vlo + at % kStages * (TK::kBytes >> 4);
#pragma unroll 1
        for (int p = 0; p < steps_of(kSumsO); ++p) {
          const Step st = step_of(kSumsO, p);
          const uint32_t po = p0 + st.a * 32, vo = v0 + st.b * kPK, to = tmem_o + (st.second ? D : 0), idesc = st.two ? kIdescO2 : kIdescO1;
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            if (leader) ptx::mma_ts2(to, po + ks * 8, vo + ks * (2048 >> 4), kHi, idesc, st.onto || ks > 0 ? 1u : 0u);
        }
        if (leader) {
          ptx::mma_commit(&ctl->v_free[at & 1]);
          ptx::mma_commit(&ctl->o_full);
        }
      };
      if (warp == kIssueWarp) {
        for (int t = 0; t < n; ++t) {
          const uint32_t at = done + t;
          if (!uwait(&ctl->k_full[at % kStages], at / kStages)) break;
          if (!(t == 0 ? uwait(&ctl->q_full, pass) : uwait(&ctl->s_free, at - 1))) break;
          ptx::tc_fence_after();
          issue_qk(at);
        }
      } else if (warp == kIssueWarp + 1) {
        for (int t = 0; t < n; ++t) {
          const uint32_t at = done + t;
          if (!uwait(&ctl->v_full[at % kStages], at / kStages) || (t > 0 && !uwait(&ctl->o_free, at - 1))) break;
          if (!uwait(&ctl->p_full[at & 1], at >> 1)) break;
          ptx::tc_fence_after();
          issue_pv(at);
        }
      } else if (MASK != kNoMask) {
        // ------------------------------------------------------------------------------------------------ masks --
        const int mt_id = tid & 63, w = warp - kIssueWarp - 2;  // 64 rows a warp
        const bool same = a.mask.sl == 0 && (a.mask.sh == 0 || group == 1);  // for all rows of this CTA
        const int r0 = w * 64 + (MASK == kAddMask && a.mask.wide ? lane / 16 : (MASK == kBoolMask ? lane : 0));
        const int first_iq = query_of(r0), first_g = gr.head(row0 + r0);
        for (int t = 0; t < n; ++t) {
          const uint32_t at = done + t;
          const int col0 = (t0 + t) * BN;
          const uint32_t stage = at % LY::kMaskStages, use = at / LY::kMaskStages, mask_at = base + LY::kM + stage * LY::kMaskBytes;
          if (use > 0 && !uwait(&ctl->m_free[stage], use - 1)) break;
          const int64_t mask_b = b * a.mask.sb + hk * group * a.mask.sh + col0;
          auto each_row = [&](int step, int count, auto f) {  // from r0 on
            each_mask_row<8>(a.mask, group, rows, row0 + r0, first_g, mask_b + first_g * a.mask.sh + first_iq * a.mask.sl, step, count,
                             [&](int e, bool in, int64_t p) { f(r0 + e, in, p); });
          };
          if constexpr (MASK == kBoolMask) {
            // a row's 64 bytes to bits: the aligned words that hold them, shifted into place
            auto bits = [&](int r, bool in, int64_t p) {
              const uintptr_t from = reinterpret_cast<uintptr_t>(a.mask.ptr) + p;
              const int mis = static_cast<int>(from & 3), end = min(BN, kv_len - col0) + mis;
              const uint32_t* words = reinterpret_cast<const uint32_t*>(from - mis);
              uint32_t x[BN / 4 + 1];
#pragma unroll
              for (int i = 0; i <= BN / 4; ++i) {
                x[i] = 0;
                if (in && 4 * i < end) x[i] = __ldg(words + i);
              }
              uint32_t two[2] = {0, 0};
#pragma unroll
              for (int i = 0; i < BN / 4; ++i) two[i / 8] |= mask_bits(x[i], x[i + 1], mis) << (4 * (i % 8));
              if (same)
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %1, %2};" ::"r"(mask_at + mt_id * 16), "r"(two[0]), "r"(two[1]) : "memory");
              else
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(mask_at + r * 8), "r"(two[0]), "r"(two[1]) : "memory");
            };
            if (same)
              bits(0, true, mask_b);
            else
              each_row(32, 2, bits);
            ptx::mbar_arrive(&ctl->m_full[stage]);
          } else {
            const float* any = reinterpret_cast<const float*>(a.mask.ptr);
            auto copy4 = [&](uint32_t to, const float* p, bool in) {
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(in ? p : any), "r"(in ? 4 : 0) : "memory");
            };
            if constexpr (MASK == kAddRow) {
              copy4(mask_at + mt_id * 4, any + mask_b + mt_id, col0 + mt_id < kv_len);
            } else if (a.mask.wide) {  // two rows of 64 floats at a time
              const int ch = lane % 16, left = min(4, a.Skv - col0 - ch * 4);
              each_row(2, 32, [&](int r, bool in, int64_t p) {
                in = in && left > 0;
                ptx::cp_async16(mask_at + r * BN * 4 + ((ch ^ (r & 7)) << 4), in ? any + p + ch * 4 : any, in ? left * 4 : 0);
              });
            } else {
              // (keys beyond the length are left as they are: they are hidden)
              const bool in0 = col0 + lane < kv_len, in1 = col0 + lane + 32 < kv_len;
              each_row(1, 64, [&](int r, bool in, int64_t p) {
                const uint32_t to = mask_at + r * BN * 4 + (((lane / 4) ^ (r & 7)) << 4) + (lane % 4) * 4;
                copies4(to, in ? any + p + lane : any, in, in0, in1);
              });
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(ptx::smem_u32(&ctl->m_full[stage])) : "memory");
          }
        }
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

template <int D, MaskForm MASK>
cudaError_t launch_t(const FwdArgs& a, int cluster, int device, cudaStream_t stream) {
  auto kern = cluster > 1 ? fwd_f32_kernel<D, MASK, true> : fwd_f32_kernel<D, MASK, false>;
  const long long tiles = (static_cast<long long>(a.Lq) * (a.Hq / a.Hkv) + BM - 1) / BM, ctas = tiles * a.Hkv * a.B * cluster;
  if (ctas > 0x7fffffffll) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  return launch_early(kern, dim3(static_cast<unsigned>(ctas)), dim3(kThreads), Lay<D, MASK>::kBytes, stream, cluster, a, cluster);
}

// CTAs per cluster, that share a walk: what is expected to take the least time, with one CTA to an SM; constants from a sweep of 23
// shapes with 1 .. 8.  Measured, us, undivided -> chosen: D = 64, 2 heads x 512 on 4000 keys 86 -> 21 (8), causal 3 x 1000 26.5 -> 14.7
// (5; 6, for which there is no room at once: 20.9), 2 x 8/2 heads x 130 on 1500 37 -> 15.5 (6); D = 128, 8/1 heads x 33 on 1000 66 -> 18 (8),
// causal 4 heads x 4096 222 -> 115 (2; 4: 151).
int split_of(const FwdArgs& a, int D, int device) {
  const double step = D == 64 ? 1.4 : 3.6, item = D == 64 ? 5.0 : 6.0, merge = 2.4;
  const long long rows = static_cast<long long>(a.Lq) * (a.Hq / a.Hkv), ctas = (rows + BM - 1) / BM * a.Hkv * a.B;
  const bool triangle = a.causal == TT_ATTN_CAUSAL_TOP_LEFT;
  const int tiles = (a.Skv + BN - 1) / BN, longest = triangle ? std::min(tiles, (a.Lq + BN - 1) / BN) : tiles;
  int best = 1;
  double best_us = 1e30;
  for (int c = 1; c <= 8; ++c) {
    const int room = cluster_room(device, c), walk = (longest + c - 1) / c;
    if (room <= 0) continue;
    // (walks of one length come in whole rounds, those of a triangle fill them up, but for what a CTA takes besides)
    const double rounds = static_cast<double>(ctas) * c / room;
    const double all = std::ceil(rounds) * item + (triangle ? rounds * 0.5 * (walk + 1) : std::ceil(rounds) * walk) * step;
    const double us = std::max(item + walk * step, all) + (c > 1 ? merge : 0.0);
    if (us < best_us) best = c, best_us = us;
  }
  return best;
}

template <int D>
cudaError_t launch_d(const FwdArgs& a, int cluster, int device, cudaStream_t stream) {
  if (!a.mask.ptr) return launch_t<D, kNoMask>(a, cluster, device, stream);
  if (a.mask.kind == TT_ATTN_MASK_BOOL) return launch_t<D, kBoolMask>(a, cluster, device, stream);
  if (a.mask.sl == 0 && (a.mask.sh == 0 || a.Hq == a.Hkv)) return launch_t<D, kAddRow>(a, cluster, device, stream);
  return launch_t<D, kAddMask>(a, cluster, device, stream);
}

}  // namespace

cudaError_t launch_fwd_f32(int D, const FwdArgs& a, int device, cudaStream_t stream) {
  const int cluster = split_of(a, D, device);
  return D == 64 ? launch_d<64>(a, cluster, device, stream) : launch_d<128>(a, cluster, device, stream);
}

}  // namespace ttattn
