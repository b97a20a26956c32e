// y[M,N] = x[M,K] w[N,K]^T + bias[N] for shapes whose output has too few tiles to occupy the machine: token steps
// (a few rows against a large weight, where reading w once is all there is to do) and small problems in general.
// linear_tc.cu gives such a problem one CTA per 128 x 256 tile, 16 CTAs for 8 x 4096, and those draw 0.7 TB/s.
//
//  * The operands change places: 128 rows of w are the M dimension of the MMA (TMEM lanes), the rows of x (padded to a
//    multiple of 16, up to 256) its N dimension.  A token step then spends a 128 x 16 MMA on a tile of w instead of
//    128 x 256 with 120 rows of zeros, and the output has N / 128 tiles.
//  * The contraction is divided among the CTAs of a thread-block cluster (up to 8), so that N / 128 x 8 CTAs stream
//    w at the same time.  Each leaves its fp32 partial tile in its own shared memory; after a cluster barrier every
//    CTA sums a share of the rows over the cluster through distributed shared memory, in rank order (the result does
//    not depend on timing), adds the bias and rounds once.  No scratch memory, no second kernel, no atomics.
//  * Up to three CTAs share an SM (72 KB of shared memory each), so that the start of one and the end of another
//    overlap with the stream of a third.
//  * Launched early behind the kernel before it (programmatic dependent launch): barriers, TMEM and descriptors are
//    set up, and the first tiles of w are asked for in L2, while that kernel still runs.
//
// X_MN / W_MN: the operand is stored with the contraction as its slow dimension (the gradients dX = dY W and dW = dY^T X)
// and is read as an MN-major MMA operand instead of being transposed in memory.
//
// Warps 0-3: epilogue (thread r = TMEM lane r = output column); warp 4: TMA producer; warp 5: MMA issuer.
// Every mbarrier wait is bounded; after an expired one the CTA still meets the cluster barriers.
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"
#include "tma_host.cuh"

namespace ttattn {
namespace {

constexpr int BW = 128;  // rows of w (output columns) per tile
constexpr int BK = 64;   // contraction elements per stage: one 128-byte swizzled row
constexpr int kThreads = 192;
constexpr int kWBytes = BW * BK * 2;
constexpr int kMaxStage = 8;
constexpr int kMaxCluster = 8;
constexpr int kPrefetch = 8;  // stages of w asked for in L2 ahead of the kernel before this one

struct __align__(8) SmemCtl {
  uint64_t full[kMaxStage], empty[kMaxStage];
  uint64_t acc_full;
  uint32_t tmem_base;
  int abort_flag;
};

struct SplitArgs {
  const void* bias;  // [N] in the tensor dtype, or null
  void* y;
  int64_t ldy;
  int M, N, K;
  int mt;      // rows of x per tile: the N dimension of the MMA, a multiple of 16 (X_MN: of 64)
  int tiles_m, tiles_n;
  int stages, cluster;
  uint32_t tmem_cols;
  int32_t* status;
};

// Sum over the cluster of row m of the partial tiles (columns 4 * lane ..), bias, rounding: rows first, first + step, ...
// of the tile.  kRows rows are in flight at once, so that 8 distributed-shared-memory loads are, whatever the cluster.
template <typename T, int CS>
__device__ __forceinline__ void reduce_rows(const SplitArgs& a, uint32_t part, int first, int step, int rows, int m0, int n,
                                            const float4& bias) {
  constexpr int kRows = 8 / CS;
  uint32_t peer[CS];
#pragma unroll
  for (int r = 0; r < CS; ++r) peer[r] = CS > 1 ? ptx::map_rank(part, r) : part;
  for (int m = first; m < rows; m += kRows * step) {
    float4 p[kRows][CS];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      // (rows beyond the tile's last: any row that exists, the result is dropped)
      const uint32_t off = static_cast<uint32_t>(m + i * step < rows ? m + i * step : m) * (BW * 4);
#pragma unroll
      for (int r = 0; r < CS; ++r) p[i][r] = ptx::ld_cluster_f4(peer[r] + off);
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      float4 acc = p[i][0];
#pragma unroll
      for (int r = 1; r < CS; ++r) acc.x += p[i][r].x, acc.y += p[i][r].y, acc.z += p[i][r].z, acc.w += p[i][r].w;
      const T out[4] = {from_f32<T>(acc.x + bias.x), from_f32<T>(acc.y + bias.y), from_f32<T>(acc.z + bias.z),
                        from_f32<T>(acc.w + bias.w)};
      if (m + i * step < rows)
        *reinterpret_cast<uint2*>(reinterpret_cast<T*>(a.y) + static_cast<int64_t>(m0 + m + i * step) * a.ldy + n) =
            *reinterpret_cast<const uint2*>(out);
    }
  }
}

template <bool BF16, bool X_MN, bool W_MN>
__global__ void __launch_bounds__(kThreads)
    linear_split_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SplitArgs a) {
  using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int stage_bytes = kWBytes + a.mt * 128;
  SmemCtl* ctl = reinterpret_cast<SmemCtl*>(smem + a.stages * stage_bytes);
  float* part = reinterpret_cast<float*>(smem);  // [mt][128] partial tile, over the stages once they are consumed
  volatile int* abort_flag = &ctl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = a.cluster > 1 ? ptx::cluster_rank() : 0;
  const int tile = blockIdx.x / a.cluster;
  // Neighbouring CTAs share the larger operand, which then comes from HBM once (M = 13787, N = 264, K = 9848 with the rows of x
  // fastest: every column tile read x again, 171 us; 141 with the columns fastest).
  const bool columns = a.M > a.N;
  const int tm = columns ? tile / a.tiles_n : tile % a.tiles_m, tn = columns ? tile % a.tiles_n : tile / a.tiles_m;
  const int m0 = tm * a.mt, n0 = tn * BW;
  // this CTA's share of the contraction
  const int n_kb = (a.K + BK - 1) / BK, per = (n_kb + a.cluster - 1) / a.cluster;
  const int kb0 = static_cast<int>(rank) * per;
  const int kb1 = kb0 + per < n_kb ? kb0 + per : n_kb;  // (<= kb0 where nothing is left)

  if (tid == 128) {
    for (int s = 0; s < a.stages; ++s) {
      ptx::mbar_init(&ctl->full[s], 1);
      ptx::mbar_init(&ctl->empty[s], 1);
    }
    ptx::mbar_init(&ctl->acc_full, 1);
    ctl->abort_flag = (ptx::smem_u32(smem) & 1023u) != 0;  // the swizzled tiles need a 1024-byte boundary
    ptx::fence_barrier_init();
    ptx::tma_prefetch_desc(&tmW);
    ptx::tma_prefetch_desc(&tmX);
  }
  if (warp == 5) {
    ptx::tmem_alloc(&ctl->tmem_base, a.tmem_cols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  // The next kernel may come up only now that this CTA has its TMEM columns: one that took them first would wait for
  // this grid, and this CTA for its columns.  (Among CTAs that are resident together columns never run out: a kernel
  // with 512 of them leaves no shared memory for this one, and this one's own share per SM is at most 256.)
  ptx::grid_dep_launch();

  bool ok = *abort_flag == 0;
  if (warp == 4) {
    // -------------------------------------------------------------- producer --
    if (lane == 0 && ok) {
      const int pre = kb0 + kPrefetch < kb1 ? kb0 + kPrefetch : kb1;
      for (int kb = kb0; kb < pre; ++kb) {
        if constexpr (W_MN) {
          ptx::tma_prefetch_4d(&tmW, n0, kb * BK, 0, 0);
          ptx::tma_prefetch_4d(&tmW, n0 + 64, kb * BK, 0, 0);
        } else {
          ptx::tma_prefetch_4d(&tmW, kb * BK, n0, 0, 0);
        }
      }
      ptx::grid_dep_wait();
      int s = 0;
      uint32_t ph = 1;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!ptx::mbar_wait(&ctl->empty[s], ph, abort_flag)) break;
        uint8_t* st = smem + s * stage_bytes;
        ptx::mbar_arrive_expect_tx(&ctl->full[s], stage_bytes);
        if constexpr (W_MN) {  // two blocks of 64 output columns, [64 contraction rows][64 columns] each
          ptx::tma_load_4d(st, &tmW, &ctl->full[s], n0, kb * BK, 0, 0);
          ptx::tma_load_4d(st + kWBytes / 2, &tmW, &ctl->full[s], n0 + 64, kb * BK, 0, 0);
        } else {
          ptx::tma_load_4d(st, &tmW, &ctl->full[s], kb * BK, n0, 0, 0);
        }
        if constexpr (X_MN) {
          for (int c = 0; c < a.mt; c += 64)
            ptx::tma_load_4d(st + kWBytes + c * 128, &tmX, &ctl->full[s], m0 + c, kb * BK, 0, 0);
        } else {
          ptx::tma_load_4d(st + kWBytes, &tmX, &ctl->full[s], kb * BK, m0, 0, 0);  // rows beyond M read as zero
        }
        if (++s == a.stages) s = 0, ph ^= 1;
      }
    }
  } else if (warp == 5) {
    // ---------------------------------------------------------------- issuer --
    if (ok) {
      const bool leader = ptx::elect_one();
      constexpr uint32_t kHi = ptx::smem_desc_hi_sw128(1024);
      const uint32_t idesc = ptx::make_idesc_f16(BW, a.mt, BF16 ? 1 : 0, W_MN ? 1 : 0, X_MN ? 1 : 0);
      const uint32_t wlo = ptx::smem_desc_lo(ptx::smem_u32(smem), W_MN ? kWBytes / 2 : 16);
      const uint32_t xlo = ptx::smem_desc_lo(ptx::smem_u32(smem + kWBytes), X_MN ? 64 * 128 : 16);
      // one k-step: 16 contraction rows of 128 bytes (MN-major), or 32 bytes of the 128-byte swizzled row
      constexpr uint32_t kXStep = X_MN ? 128 : 2, kWStep = W_MN ? 128 : 2;
      int s = 0;
      uint32_t ph = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!(ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->full[s], ph, abort_flag)) != 0)) break;
        ptx::tc_fence_after();
        const uint32_t so = static_cast<uint32_t>(s * stage_bytes) >> 4;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          if (leader)
            ptx::mma_ss2(tmem, wlo + so + k * kWStep, kHi, xlo + so + k * kXStep, kHi, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        if (leader) ptx::mma_commit(&ctl->empty[s]);
        if (++s == a.stages) s = 0, ph ^= 1;
      }
      if (leader && ok) ptx::mma_commit(&ctl->acc_full);
    }
  } else {
    // ---------------------------------------------- partial tile -> shared memory --
    const uint32_t lane_addr = static_cast<uint32_t>(warp * 32) << 16;
    if (kb1 > kb0) {
      if (ok) ok = ptx::mbar_wait(&ctl->acc_full, 0, abort_flag);
      ptx::tc_fence_after();
    }
    // (every MMA of this CTA is complete, so the stages are free; adjacent threads write adjacent words)
    for (int c = 0; c < a.mt; c += 16) {
      uint32_t v[16];
      if (kb1 > kb0) {
        ptx::tmem_ld16(tmem + lane_addr + c, v);
        ptx::tmem_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0u;
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) part[(c + i) * BW + tid] = __uint_as_float(v[i]);
    }
    ptx::tc_fence_before();
  }
  __syncwarp();
  if (a.cluster > 1)
    ptx::cluster_sync();
  else
    __syncthreads();

  // ------------------------------------- sum over the cluster, bias, rounding: rows rank, rank + cluster, ... --
  if (*abort_flag == 0) {
    ptx::grid_dep_wait();  // the bias is read and y written here
    const int rows = a.M - m0 < a.mt ? a.M - m0 : a.mt;
    const int n = n0 + lane * 4;
    if (n < a.N) {  // (N is a multiple of 8)
      float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
      if (a.bias) {
        const T* bp = reinterpret_cast<const T*>(a.bias) + n;
        bias = make_float4(to_f32<T>(bp[0]), to_f32<T>(bp[1]), to_f32<T>(bp[2]), to_f32<T>(bp[3]));
      }
      const uint32_t pl = ptx::smem_u32(part + lane * 4);
      const int step = kThreads / 32 * a.cluster, first = static_cast<int>(rank) + warp * a.cluster;
      if (a.cluster == 8)
        reduce_rows<T, 8>(a, pl, first, step, rows, m0, n, bias);
      else if (a.cluster == 4)
        reduce_rows<T, 4>(a, pl, first, step, rows, m0, n, bias);
      else if (a.cluster == 2)
        reduce_rows<T, 2>(a, pl, first, step, rows, m0, n, bias);
      else
        reduce_rows<T, 1>(a, pl, first, step, rows, m0, n, bias);
    }
  }
  __syncwarp();
  if (a.cluster > 1)
    ptx::cluster_sync();  // no CTA leaves while another still reads its shared memory
  else
    __syncthreads();
  if (warp == 5) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, a.tmem_cols);
  }
  if (tid == 0 && ctl->abort_flag && a.status) atomicOr(a.status, kStatusWaitExpired);
}

// How the problem is divided: the cheapest of the candidates by a model fitted to a sweep of 20 problems from 1 x 1024 x
// 1024 to 2000 x 1024 x 1024 and 64 x 4096 x 28672 (B200; within 1.5 us of the measured time for the plans near the
// best, and the plan it picks within 8 % of the best of the sweep):
//   2.8 us     launch, set-up, first tile, cluster barriers, last store
//   + the slower of  weight and x from HBM (6.0 TB/s, or less where the stages in flight do not cover 1.7 us)  and
//     an SM's share of the tiles through its L2 port (135 B/ns)
//   + 10 ns per row of x: the partial tile through shared memory;  + 12.5 ns more where the cluster sums it
//   + 2.5 us and the partial tile again for every further wave of CTAs (half where CTAs that share an SM overlap)
// Candidates: 16..256 rows of x per tile, clusters of 1, 2, 4, 8 with at least two stages of work per CTA, up to three
// CTAs per SM, which share its 224 KB.
// CTAs of such clusters that can be resident at once, at `per_sm` to an SM: a cluster lives inside one GPC, and GPCs
// differ in size, so clusters of 8 leave up to a fifth of the SMs unused.  Asked once per device, size and share.
int cluster_slots(int device, int cluster, int per_sm);

SplitPlan plan_split(int M, int N, int K, bool x_t, int device) {
  const int sms = sm_count(device);
  SplitPlan best{};
  best.us = 1e30;
  const int n_kb = (K + BK - 1) / BK, tiles_n = (N + BW - 1) / BW;
  const double bytes = 2.0 * K * (static_cast<double>(N) + M);
  int last_mt = 0;
  const int unit = x_t ? 64 : 16;
  for (int tm = (M + 255) / 256; tm <= (M + unit - 1) / unit; tm += tm < 16 ? 1 : tm / 8) {
    const int mt = ((M + tm - 1) / tm + unit - 1) / unit * unit;
    if (mt == last_mt) continue;
    last_mt = mt;
    SplitPlan p;
    p.mt = mt;
    p.tiles_m = (M + mt - 1) / mt;
    const long long tiles = static_cast<long long>(p.tiles_m) * tiles_n;
    if (tiles > 1 << 24) break;
    p.tiles = static_cast<int>(tiles);
    const int stage = kWBytes + mt * 128;
    for (p.cluster = 1; p.cluster <= kMaxCluster; p.cluster *= 2) {
      if (p.cluster > 1 && n_kb < 2 * p.cluster) break;
      const long long ctas = tiles * p.cluster;
      int per_sm = static_cast<int>((ctas + sms - 1) / sms < 3 ? (ctas + sms - 1) / sms : 3);
      // at least three stages, and room for the partial tile over them
      while (per_sm > 1 && (224 * 1024 / per_sm - 2048) / stage < (mt > 64 ? 4 : 3)) --per_sm;
      const int fit = (224 * 1024 / per_sm - 2048) / stage;
      p.stages = fit < kMaxStage ? fit : kMaxStage;
      const long long slots = cluster_slots(device, p.cluster, per_sm), waves = (ctas + slots - 1) / slots;
      const double sm_us = static_cast<double>(waves) * per_sm * ((n_kb + p.cluster - 1) / p.cluster) * stage / 135e3;
      const double in_flight = static_cast<double>(ctas < slots ? ctas : slots) * p.stages * kWBytes / 1.7;
      p.hbm_rate = in_flight < 6.0e6 ? in_flight : 6.0e6;
      p.per_sm = per_sm, p.waves = static_cast<int>(waves);
      const double hbm_us = bytes / p.hbm_rate;
      p.us = 2.8 + (sm_us > hbm_us ? sm_us : hbm_us) + 0.010 * mt + (p.cluster > 1 ? 0.0125 * mt : 0.0) +
             static_cast<double>(waves - 1) * (2.5 + 0.010 * mt) * (per_sm == 1 ? 1.0 : 0.5);
      p.smem = p.stages * stage + static_cast<int>(sizeof(SmemCtl));
      if (p.us < best.us) best = p;
    }
  }
  return best;
}

template <bool BF16, bool X_MN, bool W_MN>
cudaError_t launch_t(const LinearCall& c, const SplitPlan& p) {
  auto kern = linear_split_kernel<BF16, X_MN, W_MN>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return e;
  CUtensorMap tw, tx;
  if (!make_map_2d(&tw, c.dtype, c.w, W_MN ? c.N : c.K, W_MN ? c.K : c.N, c.ldw, W_MN ? BK : BW) ||
      !make_map_2d(&tx, c.dtype, c.x, X_MN ? c.M : c.K, X_MN ? c.K : c.M, c.ldx, X_MN ? BK : p.mt))
    return cudaErrorInvalidValue;
  uint32_t cols = 32;
  while (static_cast<int>(cols) < p.mt) cols *= 2;
  const SplitArgs a{c.bias, c.y, c.ldy, c.M, c.N, c.K, p.mt, p.tiles_m, p.tiles / p.tiles_m, p.stages, p.cluster, cols, c.status};
  return launch_early(kern, dim3(static_cast<unsigned>(p.tiles) * p.cluster), dim3(kThreads), p.smem, c.stream, p.cluster,
                      tw, tx, a);
}

template <bool BF16>
cudaError_t launch_bf(const LinearCall& c, const SplitPlan& p) {
  if (c.x_t) return c.w_t ? launch_t<BF16, true, true>(c, p) : launch_t<BF16, true, false>(c, p);
  return c.w_t ? launch_t<BF16, false, true>(c, p) : launch_t<BF16, false, false>(c, p);
}

int cluster_slots(int device, int cluster, int per_sm) {
  static std::atomic<int> known[64][3][3];
  const int full = per_sm * sm_count(device);
  if (cluster == 1 || device < 0 || device >= 64) return full;
  std::atomic<int>& k = known[device][cluster == 2 ? 0 : (cluster == 4 ? 1 : 2)][per_sm - 1];
  int n = k.load(std::memory_order_relaxed);
  if (n == 0) {
    auto kern = linear_split_kernel<true, false, false>;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(full / cluster * cluster);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = 224 * 1024 / per_sm - 2048;
    cfg.attrs = attr, cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters <= 0) {
      cudaGetLastError();
      clusters = full / cluster;
    }
    n = clusters * cluster < full ? clusters * cluster : full;
    k.store(n, std::memory_order_relaxed);
  }
  return n;
}

}  // namespace

// What the plan is expected to take, for the choice between the kernels: as above, fitted to 170 problems (6 % rms) that the plans
// themselves do not depend on: operands whose rows do not lie on cache lines, and the output's way to memory.
double linear_split_us(const LinearCall& c, const SplitPlan& p) {
  const int n_kb = (c.K + BK - 1) / BK;
  const double lines = BW * row_lines(c.ldw) + p.mt * row_lines(c.ldx), bytes = 2.0 * c.K * (static_cast<double>(c.N) + c.M);
  const double sm_us = static_cast<double>(p.waves) * p.per_sm * ((n_kb + p.cluster - 1) / p.cluster) * lines * 128 / 137e3;
  const double hbm_us = bytes / p.hbm_rate;
  const double body = 3.1 + (sm_us > hbm_us ? sm_us : hbm_us) + 0.0097 * p.mt + (p.cluster > 1 ? 0.016 * p.mt : 0.0) +
                      (p.waves - 1) * (3.7 + 0.0097 * p.mt) * (p.per_sm == 1 ? 1.0 : 0.5);
  const double out = 2.0 * c.M * c.N / 1.44e6 * (c.N % 16 ? 1.18 : 1.0);
  return body > out ? body + 0.1 * out : out + 0.1 * body;
}

SplitPlan plan_linear_split(const LinearCall& c) { return plan_split(c.M, c.N, c.K, c.x_t, c.device); }

cudaError_t launch_linear_split(const LinearCall& c, const SplitPlan& p) {
  return c.dtype == TT_ATTN_BF16 ? launch_bf<true>(c, p) : launch_bf<false>(c, p);
}

}  // namespace ttattn
