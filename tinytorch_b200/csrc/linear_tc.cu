// y[M,N] = x[M,K] w[N,K]^T + bias[N] for fp16 / bf16 on sm_100a tensor cores: the
// projections either side of attention (reference: function::linear =
// op::matmul(input, weight, false, true, bias), src/Function/FuncNNLayer.h:14-19, which
// calls a library gemm and, for the bias, pre-fills C, src/Operation/OpLinalgCuda.cuh:141-215),
// and its two gradient products.
//
// Persistent CTA PAIRS (clusters of two, tcgen05 cta_group::2), one CTA per SM, output tiles of 256 x 256: each CTA of
// a pair holds 128 rows of the tile and of x, and HALF of the tile's rows of w; an MMA of M = 256, N = 256, K = 16
// reads 8 KB from each CTA's shared memory in 128 clocks and the fills bring in another 8 KB, i.e. 128 bytes per clock
// of tensor time where two independent 128 x 256 tiles need 192 (shared memory moves 128).
//   warp 0     producer (both CTAs): cp.async.bulk.tensor loads (128-byte swizzle) of its 128 x 64 slices of x and w
//              into a 5-stage ring; both CTAs' loads complete on the LEADER's barrier of the stage
//   warp 1     issuer (leader only): one elected lane issues the MMAs into one of two 256-column TMEM accumulators per
//              CTA, used in turn, so that the epilogue of a tile runs under the main loop of the next; its commits
//              reach the barriers of both CTAs
//   warps 4-7, epilogue (both CTAs): two warpgroups take the 64-column blocks alternately, thread r of each owns output
//   warps 8-11 row r of the CTA's half (TMEM lane r); a block is read with tcgen05.ld, gets the bias (fp32), is rounded
//              to the tensor dtype and leaves through one of the warpgroup's two swizzled staging tiles and a TMA store (rows and
//              columns beyond M, N are clipped by the tensor map; the K tail reads as zero)
// Tiles are ordered in groups of row-tiles so that CTAs running at the same time share slices of x and w in L2.
// X_MN / W_MN: the operand is stored with the contraction as its slow dimension (x as [K, M], w as [K, N]) and is read
// as an MN-major MMA operand, so that the gradients dX = dY W and dW = dY^T X need no transposed copies.
// Every mbarrier wait is bounded; after an expired one the CTA still meets the cluster barrier at the end.
#include <type_traits>

#include "common.cuh"
#include "linear_order.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"

namespace ttattn {
namespace {

constexpr int BM = 256, BN = 256, BK = 64;  // tile of a pair
constexpr int HM = BM / 2, HN = BN / 2;     // what one CTA loads of it
constexpr int NSTAGE = 5;
constexpr int kThreads = 384;
constexpr int kEpi = 128;  // threads of an epilogue warpgroup
constexpr int kABytes = HM * BK * 2, kBBytes = HN * BK * 2;
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kOutBytes = HM * 128;  // staging: 128 rows x 64 columns of 16 bits

struct __align__(8) SmemCtl {
  uint64_t full[NSTAGE], empty[NSTAGE];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

constexpr int kSmemBytes = NSTAGE * kStageBytes + 4 * kOutBytes + BN * 4 + static_cast<int>(sizeof(SmemCtl));
static_assert(kSmemBytes <= 232448, "exceeds the shared memory a CTA may request");

struct LinArgs {
  const void* bias;  // [N] in the tensor dtype, or null
  int M, N, K;
  int group_m;       // row-tiles per L2 group (see rows_per_group)
  int32_t* status;
};

template <bool BF16, bool X_MN, bool W_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    linear_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                     const __grid_constant__ CUtensorMap tmY, const LinArgs a) {
  using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sOut = smem + NSTAGE * kStageBytes;
  float* sBias = reinterpret_cast<float*>(sOut + 4 * kOutBytes);
  SmemCtl* ctl = reinterpret_cast<SmemCtl*>(sBias + BN);
  volatile int* abort_flag = &ctl->abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = ptx::cluster_rank();
  const int tiles_m = (a.M + BM - 1) / BM, tiles_n = (a.N + BN - 1) / BN;
  const int n_tiles = tiles_m * tiles_n;
  const int n_kb = (a.K + BK - 1) / BK;
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;  // the pair's tiles

  if (warp == 0 && lane == 0) {
#pragma unroll
    for (int s = 0; s < NSTAGE; ++s) {
      ptx::mbar_init(&ctl->full[s], 1);
      ptx::mbar_init(&ctl->empty[s], 1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&ctl->acc_full[i], 1);
      ptx::mbar_init(&ctl->acc_empty[i], 16);  // the epilogue warps of both CTAs
    }
    ctl->abort_flag = (ptx::smem_u32(smem) & 1023u) != 0;  // the swizzled tiles need a 1024-byte boundary
    ptx::fence_barrier_init();
    ptx::tma_prefetch_desc(&tmX);
    ptx::tma_prefetch_desc(&tmW);
    ptx::tma_prefetch_desc(&tmY);
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(&ctl->tmem_base, 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();  // the barriers of both CTAs are initialised
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
      bool ok = true;
      uint32_t full0 = ptx::map_rank(ptx::smem_u32(&ctl->full[0]), 0);  // the leader's
      for (int t = first; t < n_tiles && ok; t += step) {
        int mt, nt;
        tile_of(t, a.group_m, tiles_m, tiles_n, &mt, &nt);
        const int m0 = mt * BM + static_cast<int>(rank) * HM, n0 = nt * BN + static_cast<int>(rank) * HN;
        for (int kb = 0; kb < n_kb; ++kb) {
          if (!(ok = ptx::mbar_wait(&ctl->empty[s], ph, abort_flag))) break;
          uint8_t* sa = smem + s * kStageBytes;
          uint8_t* sb = sa + kABytes;
          const uint32_t bar = full0 + s * 8;
          if (rank == 0) ptx::mbar_arrive_expect_tx(&ctl->full[s], 2 * kStageBytes);  // both CTAs' loads
          if constexpr (X_MN) {  // blocks of [64 contraction rows][64 columns]
            ptx::tma_load_4d_pair(sa, &tmX, bar, m0, kb * BK, 0, 0);
            ptx::tma_load_4d_pair(sa + kABytes / 2, &tmX, bar, m0 + 64, kb * BK, 0, 0);
          } else {
            ptx::tma_load_4d_pair(sa, &tmX, bar, kb * BK, m0, 0, 0);  // rows beyond M read as zero
          }
          if constexpr (W_MN) {
            ptx::tma_load_4d_pair(sb, &tmW, bar, n0, kb * BK, 0, 0);
            ptx::tma_load_4d_pair(sb + kBBytes / 2, &tmW, bar, n0 + 64, kb * BK, 0, 0);
          } else {
            ptx::tma_load_4d_pair(sb, &tmW, bar, kb * BK, n0, 0, 0);
          }
          if (++s == NSTAGE) s = 0, ph ^= 1;
        }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ---------------------------------------------------------------- issuer --
    // the whole warp runs the loop (waits made uniform by a vote), one elected lane issues: addresses and
    // descriptors stay warp-uniform
    const bool leader = ptx::elect_one();
    constexpr uint32_t kHi = ptx::smem_desc_hi_sw128(1024);
    const uint32_t idesc = ptx::make_idesc_f16(BM, BN, BF16 ? 1 : 0, X_MN ? 1 : 0, W_MN ? 1 : 0);
    const uint32_t alo = ptx::smem_desc_lo(ptx::smem_u32(smem), X_MN ? kABytes / 2 : 16);
    const uint32_t blo = ptx::smem_desc_lo(ptx::smem_u32(smem + kABytes), W_MN ? kBBytes / 2 : 16);
    // one k-step: 16 contraction rows of 128 bytes (MN-major), or 32 bytes of the 128-byte swizzled row
    constexpr uint32_t kAStep = X_MN ? 128 : 2, kBStep = W_MN ? 128 : 2;
    int s = 0;
    uint32_t ph = 0;
    bool ok = usable;
    int i = 0;
    for (int t = first; t < n_tiles && ok; t += step, ++i) {
      const int buf = i & 1;
      // the epilogues of both CTAs have read what this accumulator held before
      if (!(ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->acc_empty[buf], ((i >> 1) & 1) ^ 1, abort_flag)) != 0)) break;
      ptx::tc_fence_after();
      const uint32_t d = tmem + buf * BN;
      for (int kb = 0; kb < n_kb; ++kb) {
        if (!(ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->full[s], ph, abort_flag)) != 0)) break;
        ptx::tc_fence_after();
        const uint32_t so = s * (kStageBytes >> 4);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          if (leader)
            ptx::mma_ss2_pair(d, alo + so + k * kAStep, kHi, blo + so + k * kBStep, kHi, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        if (leader) ptx::mma_commit_pair(&ctl->empty[s]);
        if (++s == NSTAGE) s = 0, ph ^= 1;
      }
      if (leader && ok) ptx::mma_commit_pair(&ctl->acc_full[buf]);
    }
  } else if (warp >= 4) {
    // -------------------------------------------------------------- epilogue --
    const int wg = (warp - 4) >> 2, r = tid & (kEpi - 1);  // output row within the CTA's half = TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t acc_empty0 = ptx::map_rank(ptx::smem_u32(&ctl->acc_empty[0]), 0);  // the leader's
    float* bias = sBias + wg * (BN / 2);  // of this warpgroup's two blocks
    bool ok = usable;
    int i = 0;
    for (int t = first; t < n_tiles; t += step, ++i) {
      int mt, nt;
      tile_of(t, a.group_m, tiles_m, tiles_n, &mt, &nt);
      const int n0 = nt * BN, m0 = mt * BM + static_cast<int>(rank) * HM, buf = i & 1;
      {  // (threads that see an expired wait still meet the barriers)
        const int n = n0 + wg * 64 + (r >> 6) * 128 + (r & 63);  // blocks wg and wg + 2
        bias[r] = (a.bias && n < a.N) ? to_f32<T>(reinterpret_cast<const T*>(a.bias)[n]) : 0.f;
      }
      if (ok) ok = ptx::mbar_wait(&ctl->acc_full[buf], (i >> 1) & 1, abort_flag);
      ptx::tc_fence_after();
#pragma unroll 1
      for (int cc = 0; cc < 2; ++cc) {
        const int c = wg + 2 * cc;
        uint8_t* stage = sOut + (wg * 2 + cc) * kOutBytes;
        uint32_t v[64];
        ptx::tmem_ld32p(tmem + buf * BN + lane_addr + c * 64, v);
        ptx::tmem_ld32p(tmem + buf * BN + lane_addr + c * 64 + 32, v + 32);
        // at most one earlier store (the other staging tile) may still be reading shared memory
        if (r == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        ptx::tmem_wait_ld();
        if (cc == 1) {
          // this warp's share of the accumulator is in registers / already stored
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(acc_empty0 + buf * 8);
        }
        ptx::named_barrier(1 + wg, kEpi);
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) {
          const int e = ch * 8;
          const float4 b0 = *reinterpret_cast<const float4*>(bias + cc * 64 + e);
          const float4 b1 = *reinterpret_cast<const float4*>(bias + cc * 64 + e + 4);
          uint4 w;
          w.x = pack2<BF16>(__uint_as_float(v[e + 0]) + b0.x, __uint_as_float(v[e + 1]) + b0.y);
          w.y = pack2<BF16>(__uint_as_float(v[e + 2]) + b0.z, __uint_as_float(v[e + 3]) + b0.w);
          w.z = pack2<BF16>(__uint_as_float(v[e + 4]) + b1.x, __uint_as_float(v[e + 5]) + b1.y);
          w.w = pack2<BF16>(__uint_as_float(v[e + 6]) + b1.z, __uint_as_float(v[e + 7]) + b1.w);
          *reinterpret_cast<uint4*>(stage + r * 128 + ((ch ^ (r & 7)) << 4)) = w;
        }
        ptx::fence_proxy_async_smem();
        // (also: every thread has read the bias before the next tile's is written)
        ptx::named_barrier(1 + wg, kEpi);
        if (r == 0) {
          if (ok && n0 + c * 64 < a.N && m0 < a.M) ptx::tma_store_4d(&tmY, stage, n0 + c * 64, m0, 0, 0);
          // also where nothing was stored (a block beyond M or N): the wait above counts groups, one per block
          ptx::bulk_commit();
        }
      }
    }
    if (r == 0) ptx::bulk_wait_all();
  }

  __syncwarp();
  ptx::tc_fence_before();
  ptx::cluster_sync();  // neither CTA leaves while the other may still signal its barriers
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem, 512);
  }
  if (tid == 0 && ctl->abort_flag && a.status) atomicOr(a.status, kStatusWaitExpired);
}

template <bool BF16, bool X_MN, bool W_MN>
cudaError_t launch_t(const LinearCall& c, int ctas) {
  auto kern = linear_tc_kernel<BF16, X_MN, W_MN>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  if (e != cudaSuccess) return e;
  CUtensorMap tx, tw, ty;
  // 128-byte swizzle; boxes of 64 contiguous elements (the contraction, or for an MN-major operand its other dimension)
  if (!make_map_2d(&tx, c.dtype, c.x, X_MN ? c.M : c.K, X_MN ? c.K : c.M, c.ldx, X_MN ? BK : HM) ||
      !make_map_2d(&tw, c.dtype, c.w, W_MN ? c.N : c.K, W_MN ? c.K : c.N, c.ldw, W_MN ? BK : HN) ||
      !make_map_2d(&ty, c.dtype, c.y, c.N, c.M, c.ldy, HM))
    return cudaErrorInvalidValue;
  return launch_early(kern, dim3(ctas), dim3(kThreads), kSmemBytes, c.stream, 1,
                      tx, tw, ty, LinArgs{c.bias, c.M, c.N, c.K, rows_per_group(c, BM), c.status});
}

template <bool BF16>
cudaError_t launch_bf(const LinearCall& c, int ctas) {
  if (c.x_t) return c.w_t ? launch_t<BF16, true, true>(c, ctas) : launch_t<BF16, true, false>(c, ctas);
  return c.w_t ? launch_t<BF16, false, true>(c, ctas) : launch_t<BF16, false, false>(c, ctas);
}

}  // namespace

namespace {
struct Plan {
  enum { kSplit, kTiles, kPairs } kernel;
  bool pair;  // kTiles: the shape
  int bn;
};

// Which kernel and which tiles.  Pairs of 256 x 256 read the fewest bytes for a product and keep the tensor pipe busy: large
// problems (two rounds of tiles) get them, and small ones a contraction divided over clusters where that is expected to be faster
// (linear_split.cu; always up to 128 rows).  Between the two lie problems for which a shape of linear_tile.cu puts a tile on nearly
// every SM; it is taken where it is expected to save 6 % and 0.25 us (10 % where x is MN-major), about the error of the models.  Of 251 problems with more
// than 128 rows that the models were not fitted to the mean is 0.94 of the time before (1.04 of the best shape's), the worst 1.03.
Plan plan_of(const LinearCall& c, SplitPlan* split) {
  const long long tiles = static_cast<long long>((c.M + BM - 1) / BM) * ((c.N + BN - 1) / BN);
  if (tiles >= sm_count(c.device) / 2 * 2) return Plan{Plan::kPairs, false, 0};
  *split = plan_linear_split(c);
  if (c.M <= HM) return Plan{Plan::kSplit, false, 0};
  Plan best{Plan::kPairs, false, 0};
  double us = linear_tile_us(c, true, BN);
  auto take = [&](const Plan& p, double t) {
    if (t < us) best = p, us = t;
  };
  take(Plan{Plan::kSplit, false, 0}, linear_split_us(c, *split));
  us = us * (c.x_t ? 0.9 : 0.94) - 0.25;
  if (!c.w_t) take(Plan{Plan::kTiles, true, 192}, linear_tile_us(c, true, 192));
  // (an MN-major w comes in blocks of 64 columns)
  for (int bn = 64; bn <= 256; bn += c.w_t ? 64 : 32) take(Plan{Plan::kTiles, false, bn}, linear_tile_us(c, false, bn));
  return best;
}
}  // namespace

int linear_shape(const LinearCall& c) {
  SplitPlan split;
  const Plan p = plan_of(c, &split);
  return p.kernel == Plan::kSplit ? 0 : (p.kernel == Plan::kPairs ? -BN : (p.pair ? -p.bn : p.bn));
}

cudaError_t launch_linear_tc(const LinearCall& c, bool* persistent) {
  if (persistent) *persistent = false;
  if (c.dtype != TT_ATTN_BF16 && c.dtype != TT_ATTN_F16) return cudaErrorInvalidValue;
  SplitPlan split;
  const Plan p = plan_of(c, &split);
  if (p.kernel == Plan::kSplit) return launch_linear_split(c, split);
  if (persistent) *persistent = true;
  if (p.kernel == Plan::kTiles) return launch_linear_tile(c, p.pair, p.bn);
  const long long tiles = static_cast<long long>((c.M + BM - 1) / BM) * ((c.N + BN - 1) / BN);
  const int pairs = sm_count(c.device) / 2;
  const int ctas = 2 * static_cast<int>(tiles < pairs ? tiles : pairs);
  return c.dtype == TT_ATTN_BF16 ? launch_bf<true>(c, ctas) : launch_bf<false>(c, ctas);
}

}  // namespace ttattn
