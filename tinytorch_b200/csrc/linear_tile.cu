// y[M,N] = x[M,K] w[N,K]^T + bias[N] and its gradient products for outputs between those of linear_tc.cu and linear_split.cu: too
// few tiles of 256 x 256 to fill the machine evenly, too many to divide the contraction.  They are bound by the way of the operands
// into the SMs that have a tile (119-135 bytes a ns each, measured with up to 160 columns) and by a last round of tiles that is not full, so the tile is made
// to measure: 128 rows by 64..256 columns in steps of 32 for single CTAs, and 256 x 192 for pairs of them (clusters of two, tcgen05
// cta_group::2, each CTA with 128 rows of the tile and of x and HALF of its rows of w).  Persistent, one CTA per SM.
//   warp 0     producer (both CTAs): cp.async.bulk.tensor loads (128-byte swizzle) of 64 contraction elements of its rows of x and
//              w into a ring of up to 8 stages; both CTAs' loads complete on the LEADER's barrier of the stage
//   warp 1     issuer (leader only): one elected lane issues the MMAs into one of two TMEM accumulators per
//              CTA, used in turn, so that the epilogue of a tile runs under the main loop of the next; its commits
//              reach the barriers of both CTAs
//   warps 4-7, epilogue (both CTAs): two warpgroups take blocks of 64 columns (a single CTA: 32) alternately, thread r of each owns
//   warps 8-11 output row r of the CTA's half (TMEM lane r); a block is read with tcgen05.ld, gets the bias (fp32), is rounded
//              to the tensor dtype and leaves through one of the warpgroup's two swizzled staging tiles and a TMA store (rows and
//              columns beyond M, N are clipped by the tensor map; the K tail reads as zero)
// Measured against the better of the other two kernels, us: 349 x 2096 -> 9704 27.4 -> 17.6, 3000 x 1024 -> 1024 12.9 -> 7.7, 1455 x
// 512 -> 3616 10.8 -> 8.0, 786 x 6536 -> 3304 50.5 -> 41.2, dW of 128 x 4096 -> 1024 7.2 -> 5.0.  Two blocks of the contraction per stage, a look at
// the next stage's barrier ahead of the MMAs of this one, or CTAs that start at different blocks of the contraction: slower.
// X_MN / W_MN: the operand is stored with the contraction as its slow dimension (x as [K, M], w as [K, N]) and is read
// as an MN-major MMA operand.
// Every mbarrier wait is bounded; after an expired one the CTA still meets the barrier at the end.
#include <type_traits>

#include "common.cuh"
#include "linear_order.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"

namespace ttattn {
namespace {

constexpr int BK = 64;           // contraction elements per stage: one 128-byte swizzled row
constexpr int HM = 128;          // rows of x in one CTA
constexpr int kMaxBN = 256;      // columns of a tile, at most
constexpr int kMaxStage = 8, kPairStages = 5;
constexpr int kThreads = 384;
constexpr int kEpi = 128;        // threads of an epilogue warpgroup
constexpr int kABytes = HM * BK * 2;
constexpr int kMnBlock = 64 * BK * 2;  // 64 columns of an MN-major operand
// Columns that an epilogue warpgroup stores at a time: a staging tile of 128 rows of 128 or 64 bytes.
template <bool PAIR>
constexpr int kOutCols = PAIR ? 64 : 32;
template <bool PAIR>
constexpr int kOutBytes = HM * kOutCols<PAIR> * 2;

struct __align__(8) SmemCtl {
  uint64_t full[kMaxStage], empty[kMaxStage];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

// a stage of one CTA: 64 contraction elements of 128 rows of x and of a tile's rows of w, or half of a pair's
template <bool PAIR>
__host__ __device__ constexpr int stage_bytes(int bn) {
  return kABytes + (PAIR ? bn / 2 : bn) * BK * 2;
}
template <bool PAIR>
constexpr int kFixedBytes = 4 * kOutBytes<PAIR> + kMaxBN * 4 + static_cast<int>(sizeof(SmemCtl));
template <bool PAIR>
constexpr int smem_bytes(int bn, int stages) {
  return stages * stage_bytes<PAIR>(bn) + kFixedBytes<PAIR>;
}
constexpr int kSmemMost = 232448;  // what a CTA may request
static_assert(smem_bytes<true>(192, kPairStages) <= kSmemMost, "exceeds the shared memory a CTA may request");

struct LinArgs {
  const void* bias;  // [N] in the tensor dtype, or null
  int M, N, K;
  int bn, stages;    // columns of a tile; ring depth
  int group_m;       // row-tiles per L2 group (see rows_per_group)
  uint32_t tmem_cols;
  int32_t* status;
};

// PAIR_BN: a pair's columns, or 0: a single CTA, whose tile width comes as an argument.
template <bool BF16, bool X_MN, bool W_MN, int PAIR_BN>
__global__ void __launch_bounds__(kThreads, 1)
    linear_tile_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                     const __grid_constant__ CUtensorMap tmY, const LinArgs a) {
  using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
  constexpr bool PAIR = PAIR_BN != 0;
  static_assert(!(PAIR && W_MN), "the 96 columns of w that a CTA of a pair loads are not whole blocks of 64");
  constexpr int BM = PAIR ? 2 * HM : HM, CW = kOutCols<PAIR>, OB = kOutBytes<PAIR>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int bn = PAIR ? PAIR_BN : a.bn, stages = PAIR ? kPairStages : a.stages, sbytes = stage_bytes<PAIR>(bn);
  const uint32_t acc_cols = PAIR ? 256 : a.tmem_cols / 2;  // from one accumulator to the other
  uint8_t* sOut = smem + stages * sbytes;
  float* sBias = reinterpret_cast<float*>(sOut + 4 * OB);
  SmemCtl* ctl = reinterpret_cast<SmemCtl*>(sBias + kMaxBN);
  volatile int* abort_flag = &ctl->abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = PAIR ? static_cast<int>(ptx::cluster_rank()) : 0;
  const int tiles_m = (a.M + BM - 1) / BM, tiles_n = (a.N + bn - 1) / bn;
  const int n_tiles = tiles_m * tiles_n;
  const int n_kb = (a.K + BK - 1) / BK;
  const int first = blockIdx.x / (PAIR ? 2 : 1), step = gridDim.x / (PAIR ? 2 : 1);  // the tiles of this pair or CTA

  if (warp == 0 && lane == 0) {
    for (int s = 0; s < stages; ++s) {
      ptx::mbar_init(&ctl->full[s], 1);
      ptx::mbar_init(&ctl->empty[s], 1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&ctl->acc_full[i], 1);
      ptx::mbar_init(&ctl->acc_empty[i], PAIR ? 16 : 8);  // the epilogue warps (of both CTAs)
    }
    ctl->abort_flag = (ptx::smem_u32(smem) & 1023u) != 0;  // the swizzled tiles need a 1024-byte boundary
    ptx::fence_barrier_init();
    ptx::tma_prefetch_desc(&tmX);
    ptx::tma_prefetch_desc(&tmW);
    ptx::tma_prefetch_desc(&tmY);
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      ptx::tmem_alloc_pair(&ctl->tmem_base, a.tmem_cols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(&ctl->tmem_base, a.tmem_cols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR) ptx::cluster_sync();  // the barriers of both CTAs are initialised
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  ptx::grid_dep_wait();    // everything below reads or writes global memory
  // The next kernel may come up: this grid has its TMEM.  (After the wait, so that column_sums_kernel, which reads only x,
  // may run beside this one: once all CTAs here have come this far, everything before is complete.)
  ptx::grid_dep_launch();
  const bool usable = *abort_flag == 0;

  if (warp == 0) {
    // -------------------------------------------------------------- producer --
    if (lane == 0 && usable) {
      int s = 0;
      uint32_t ph = 1;
      uint8_t* sa = smem;
      bool ok = true;
      const uint32_t full0 = ptx::smem_u32(&ctl->full[0]), bar0 = PAIR ? ptx::map_rank(full0, 0) : full0;  // (the leader's)
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
        if constexpr (PAIR)
          ptx::tma_load_4d_pair(dst, map, bar, c0, c1, 0, 0);
        else
          ptx::tma_load_4d(dst, map, bar, c0, c1, 0, 0);
      };
      const int wn = PAIR ? bn / 2 : bn;
      for (int t = first; t < n_tiles && ok; t += step) {
        int mt, nt;
        tile_of(t, a.group_m, tiles_m, tiles_n, &mt, &nt);
        const int m0 = mt * BM + rank * HM, n0 = nt * bn + rank * wn;
        for (int kb = 0; kb < n_kb; ++kb) {
          if (!(ok = ptx::mbar_wait(&ctl->empty[s], ph, abort_flag))) break;
          const uint32_t bar = bar0 + s * 8;
          if (rank == 0) ptx::mbar_arrive_expect_tx(&ctl->full[s], PAIR ? 2 * sbytes : sbytes);  // both CTAs' loads
          if constexpr (X_MN) {  // blocks of [64 contraction rows][64 columns]
            load(sa, &tmX, bar, m0, kb * BK);
            load(sa + kMnBlock, &tmX, bar, m0 + 64, kb * BK);
          } else {
            load(sa, &tmX, bar, kb * BK, m0);  // rows beyond M read as zero
          }
          if constexpr (W_MN) {
            for (int c = 0; c < wn; c += 64) load(sa + kABytes + c * (BK * 2), &tmW, bar, n0 + c, kb * BK);
          } else {
            load(sa + kABytes, &tmW, bar, kb * BK, n0);
          }
          sa += sbytes;
          if (++s == stages) s = 0, ph ^= 1, sa = smem;
        }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ---------------------------------------------------------------- issuer --
    // the whole warp runs the loop (waits made uniform by a vote), one elected lane issues: addresses and
    // descriptors stay warp-uniform
    const bool leader = ptx::elect_one();
    constexpr uint32_t kHi = ptx::smem_desc_hi_sw128(1024);
    const uint32_t idesc = ptx::make_idesc_f16(BM, bn, BF16 ? 1 : 0, X_MN ? 1 : 0, W_MN ? 1 : 0);
    const uint32_t alo = ptx::smem_desc_lo(ptx::smem_u32(smem), X_MN ? kMnBlock : 16);
    const uint32_t blo = ptx::smem_desc_lo(ptx::smem_u32(smem + kABytes), W_MN ? kMnBlock : 16);
    // one k-step: 16 contraction rows of 128 bytes (MN-major), or 32 bytes of the 128-byte swizzled row
    constexpr uint32_t kAStep = X_MN ? 128 : 2, kBStep = W_MN ? 128 : 2;
    auto commit = [&](uint64_t* bar) {
      if constexpr (PAIR)
        ptx::mma_commit_pair(bar);
      else
        ptx::mma_commit(bar);
    };
    int s = 0;
    uint32_t ph = 0;
    bool ok = usable;
    int i = 0;
    for (int t = first; t < n_tiles && ok; t += step, ++i) {
      const int buf = i & 1;
      // the epilogues of both CTAs have read what this accumulator held before
      if (!(ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->acc_empty[buf], ((i >> 1) & 1) ^ 1, abort_flag)) != 0)) break;
      ptx::tc_fence_after();
      const uint32_t d = tmem + buf * acc_cols;
      for (int kb = 0; kb < n_kb; ++kb) {
        if (!(ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->full[s], ph, abort_flag)) != 0)) break;
        ptx::tc_fence_after();
        const uint32_t so = static_cast<uint32_t>(s * sbytes) >> 4;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          if (leader) {
            const uint32_t acc = (kb > 0 || k > 0) ? 1u : 0u;
            if constexpr (PAIR)
              ptx::mma_ss2_pair(d, alo + so + k * kAStep, kHi, blo + so + k * kBStep, kHi, idesc, acc);
            else
              ptx::mma_ss2(d, alo + so + k * kAStep, kHi, blo + so + k * kBStep, kHi, idesc, acc);
          }
        if (leader) commit(&ctl->empty[s]);
        if (++s == stages) s = 0, ph ^= 1;
      }
      if (leader && ok) commit(&ctl->acc_full[buf]);
    }
  } else if (warp >= 4) {
    // -------------------------------------------------------------- epilogue --
    const int wg = (warp - 4) >> 2, r = tid & (kEpi - 1);  // output row within the CTA's half = TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t empty0 = ptx::smem_u32(&ctl->acc_empty[0]), acc_empty0 = PAIR ? ptx::map_rank(empty0, 0) : empty0;  // the leader's
    float* bias = sBias + wg * (kMaxBN / 2);  // of this warpgroup's blocks
    const int n_blocks = bn / CW;             // two at least: one for each warpgroup
    bool ok = usable;
    int i = 0;
    uint32_t stored = 0;  // blocks so far: they alternate between the two staging tiles
    for (int t = first; t < n_tiles; t += step, ++i) {
      int mt, nt;
      tile_of(t, a.group_m, tiles_m, tiles_n, &mt, &nt);
      const int n0 = nt * bn, m0 = mt * BM + rank * HM, buf = i & 1;
      {  // (threads that see an expired wait still meet the barriers)
        const int n = n0 + (wg + r / CW * 2) * CW + r % CW;  // blocks wg, wg + 2, ...
        bias[r] = (a.bias && n < a.N) ? to_f32<T>(reinterpret_cast<const T*>(a.bias)[n]) : 0.f;
      }
      if (ok) ok = ptx::mbar_wait(&ctl->acc_full[buf], (i >> 1) & 1, abort_flag);
      ptx::tc_fence_after();
#pragma unroll 1
      for (int c = wg; c < n_blocks; c += 2, ++stored) {
        uint8_t* stage = sOut + (wg * 2 + (stored & 1)) * OB;
        const float* bc = bias + (c >> 1) * CW;
        uint32_t v[CW];
#pragma unroll
        for (int e = 0; e < CW; e += 32) ptx::tmem_ld32p(tmem + buf * acc_cols + lane_addr + c * CW + e, v + e);
        // at most one earlier store (the other staging tile) may still be reading shared memory
        if (r == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        ptx::tmem_wait_ld();
        if (c + 2 >= n_blocks) {
          // this warp's share of the accumulator is in registers / already stored
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if constexpr (PAIR)
              ptx::mbar_arrive_cluster(acc_empty0 + buf * 8);
            else
              ptx::mbar_arrive(&ctl->acc_empty[buf]);
          }
        }
        ptx::named_barrier(1 + wg, kEpi);
#pragma unroll
        for (int ch = 0; ch < CW / 8; ++ch) {
          const int e = ch * 8;
          const float4 b0 = *reinterpret_cast<const float4*>(bc + e);
          const float4 b1 = *reinterpret_cast<const float4*>(bc + e + 4);
          uint4 w;
          w.x = pack2<BF16>(__uint_as_float(v[e + 0]) + b0.x, __uint_as_float(v[e + 1]) + b0.y);
          w.y = pack2<BF16>(__uint_as_float(v[e + 2]) + b0.z, __uint_as_float(v[e + 3]) + b0.w);
          w.z = pack2<BF16>(__uint_as_float(v[e + 4]) + b1.x, __uint_as_float(v[e + 5]) + b1.y);
          w.w = pack2<BF16>(__uint_as_float(v[e + 6]) + b1.z, __uint_as_float(v[e + 7]) + b1.w);
          const int at = PAIR ? ch ^ (r & 7) : ch ^ ((r >> 1) & 3);  // the 128- or 64-byte swizzle
          *reinterpret_cast<uint4*>(stage + r * (CW * 2) + (at << 4)) = w;
        }
        ptx::fence_proxy_async_smem();
        // (also: every thread has read the bias before the next tile's is written)
        ptx::named_barrier(1 + wg, kEpi);
        if (r == 0) {
          if (ok && n0 + c * CW < a.N && m0 < a.M) ptx::tma_store_4d(&tmY, stage, n0 + c * CW, m0, 0, 0);
          // also where nothing was stored (a block beyond M or N): the wait above counts groups, one per block
          ptx::bulk_commit();
        }
      }
    }
    if (r == 0) ptx::bulk_wait_all();
  }

  __syncwarp();
  ptx::tc_fence_before();
  if (PAIR)
    ptx::cluster_sync();  // neither CTA leaves while the other may still signal its barriers
  else
    __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    if constexpr (PAIR)
      ptx::tmem_dealloc_pair(tmem, a.tmem_cols);
    else
      ptx::tmem_dealloc(tmem, a.tmem_cols);
  }
  if (tid == 0 && ctl->abort_flag && a.status) atomicOr(a.status, kStatusWaitExpired);
}

template <bool BF16, bool X_MN, bool W_MN, int PAIR_BN>
cudaError_t launch_t(const LinearCall& c, int tile_bn) {
  constexpr bool PAIR = PAIR_BN != 0;
  constexpr int BM = PAIR ? 2 * HM : HM;
  const int bn = PAIR ? PAIR_BN : tile_bn;
  const int fit = (kSmemMost - kFixedBytes<PAIR>) / stage_bytes<PAIR>(bn), stages = PAIR ? kPairStages : (fit < kMaxStage ? fit : kMaxStage);
  auto kern = linear_tile_kernel<BF16, X_MN, W_MN, PAIR_BN>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost);
  if (e != cudaSuccess) return e;
  CUtensorMap tx, tw, ty;
  // 128-byte swizzle; boxes of 64 contiguous elements (the contraction, or for an MN-major operand its other dimension)
  if (!make_map_2d(&tx, c.dtype, c.x, X_MN ? c.M : c.K, X_MN ? c.K : c.M, c.ldx, X_MN ? BK : HM) ||
      !make_map_2d(&tw, c.dtype, c.w, W_MN ? c.N : c.K, W_MN ? c.K : c.N, c.ldw, W_MN ? BK : (PAIR ? bn / 2 : bn)) ||
      !make_map_2d(&ty, c.dtype, c.y, c.N, c.M, c.ldy, HM, kOutCols<PAIR>))
    return cudaErrorInvalidValue;
  uint32_t cols = 64;  // two accumulators
  while (static_cast<int>(cols) < 2 * bn) cols *= 2;
  const long long tiles = static_cast<long long>((c.M + BM - 1) / BM) * ((c.N + bn - 1) / bn);
  const int slots = sm_count(c.device) / (PAIR ? 2 : 1), ctas = static_cast<int>(tiles < slots ? tiles : slots) * (PAIR ? 2 : 1);
  return launch_early(kern, dim3(ctas), dim3(kThreads), smem_bytes<PAIR>(bn, stages), c.stream, PAIR ? 2 : 1,
                      tx, tw, ty, LinArgs{c.bias, c.M, c.N, c.K, bn, stages, rows_per_group(c, BM), cols, c.status});
}

template <bool BF16>
cudaError_t launch_bf(const LinearCall& c, bool pair, int bn) {
  if (pair) return c.x_t ? launch_t<BF16, true, false, 192>(c, bn) : launch_t<BF16, false, false, 192>(c, bn);
  if (c.x_t) return c.w_t ? launch_t<BF16, true, true, 0>(c, bn) : launch_t<BF16, true, false, 0>(c, bn);
  return c.w_t ? launch_t<BF16, false, true, 0>(c, bn) : launch_t<BF16, false, false, 0>(c, bn);
}

}  // namespace

// What a tile shape (256 x 256 pairs among them) is expected to take, us: a model fitted to a sweep of 218 problems, half of them gradients (1 x 2392 x 7512 to
// 16000 x 2048 x 512), with 8 shapes each; 7 % rms.  2.1 us (a pair 1.6 more), then whole rounds of tiles, each 0.52 us and
// per 64 of the contraction the slower of the MMAs and the operands' way into shared memory (1.14 rows of 128 bytes per ns,
// see row_lines), and the last epilogue; or the output's way to memory at 4.2 TB/s.
double linear_tile_us(const LinearCall& c, bool pair, int bn) {
  const int bm = pair ? 2 * HM : HM, slots = sm_count(c.device) / (pair ? 2 : 1);
  const long long tiles = static_cast<long long>((c.M + bm - 1) / bm) * ((c.N + bn - 1) / bn);
  const double rows = HM * row_lines(c.ldx) + (pair ? bn / 2 : bn) * row_lines(c.ldw);
  double kb = bn * 1.288e-3;
  if (rows * 0.881e-3 > kb) kb = rows * 0.881e-3;
  if (kb < 0.21) kb = 0.21;
  const double epi = bn * 5e-3, one = static_cast<double>((c.K + BK - 1) / BK) * kb + 0.52;
  const double body = static_cast<double>((tiles + slots - 1) / slots) * (one > epi ? one : epi), out = 2.0 * c.M * c.N / 4.2e6;
  return 2.1 + (pair ? 1.6 : 0.0) + (body > out ? body + 0.1 * out : out + 0.1 * body) + epi;
}

bool linear_tile_fits(const LinearCall& c, bool pair, int bn) {
  return pair ? bn == 192 && !c.w_t : bn >= 64 && bn <= kMaxBN && bn % (c.w_t ? 64 : 32) == 0;
}

cudaError_t launch_linear_tile(const LinearCall& c, bool pair, int bn) {
  if (!linear_tile_fits(c, pair, bn)) return cudaErrorInvalidValue;
  return c.dtype == TT_ATTN_BF16 ? launch_bf<true>(c, pair, bn) : launch_bf<false>(c, pair, bn);
}

}  // namespace ttattn
