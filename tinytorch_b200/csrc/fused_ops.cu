// Fused add + RMS norm and SiLU-gated multiply: the two hand-fused transformer-block
// operators of the reference (src/Operation/OpFusedCuda.cuh:16-142), as HBM-bound
// streaming kernels.
//
// fusedAddRmsNorm: the reference's kernel makes two passes over a row and re-reads
// the residual it has just written.  Here a row (or a few short rows) lives in the
// registers of a thread group between the sum of squares and the scaling, so every
// byte crosses HBM once: read input, read residual, write residual, write input.
// All 16-byte loads of a thread are issued before the first use.
//
// siluMul: one pass, 16-byte streaming loads and stores, several vectors in flight
// per thread; long rows are tiled (row, chunk) so that indexing needs no division.
//
// columnSums: the bias gradient of a projection, sum over the rows of dY.
#include "common.cuh"
#include "ptx.cuh"

namespace ttattn {
namespace {

constexpr int kThreads = 256;
constexpr int64_t kKeepBytes = 64 << 20;  // half of L2: larger tensors are streamed past it

template <typename T>
struct Pack {
  static constexpr int N = 16 / sizeof(T);
  static __device__ __forceinline__ void unpack(const uint4& w, float (&f)[N]) {
    const T* t = reinterpret_cast<const T*>(&w);
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = to_f32<T>(t[i]);
  }
  static __device__ __forceinline__ uint4 pack(const float (&f)[N]) {
    uint4 w;
    T* t = reinterpret_cast<T*>(&w);
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = from_f32<T>(f[i]);
    return w;
  }
};

__device__ __forceinline__ uint4 ld_cs(const void* p) {
  uint4 r;
  asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}
// KEEP: the tensors fit L2, where the next operator finds them
template <bool KEEP>
__device__ __forceinline__ uint4 ld_vec(const void* p) {
  if constexpr (KEEP) return *reinterpret_cast<const uint4*>(p);
  else return ld_cs(p);
}
__device__ __forceinline__ void st_cs(void* p, const uint4& v) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
template <bool KEEP>
__device__ __forceinline__ void st_vec(void* p, const uint4& v) {
  if constexpr (KEEP) *reinterpret_cast<uint4*>(p) = v;
  else st_cs(p, v);
}

// A group of `tpr` threads (a power of two, 32..256) owns one row; a CTA holds
// kThreads / tpr rows.  Each thread keeps VPT 16-byte vectors of the row.
// FEW: so few rows that the kernel is a chain of latencies: the weight is fetched with the row instead of after the sum
// (with many rows it comes from L1, and its registers would cost resident warps).
template <typename T, int VPT, bool FEW, bool KEEP>
__global__ void __launch_bounds__(kThreads) add_rms_norm_kernel(T* __restrict__ input, T* __restrict__ residual,
                                                                const T* __restrict__ weight, int64_t rows, int dim,
                                                                int tpr, float eps) {
  constexpr int N = Pack<T>::N;
  __shared__ float s_part[kThreads / 32];
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rows_per_cta = kThreads / tpr;
  const int t_in_row = tid % tpr;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * rows_per_cta + tid / tpr;
  const bool row_ok = row < rows;
  const int vecs = dim / N;
  T* in_row = input + row * dim;
  T* res_row = residual + row * dim;

  uint4 a[VPT], b[VPT], wv[FEW ? VPT : 1];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int idx = t_in_row + v * tpr;
    const bool ok = row_ok && idx < vecs;
    a[v] = ok ? ld_vec<KEEP>(in_row + idx * N) : make_uint4(0, 0, 0, 0);
    b[v] = ok ? ld_vec<KEEP>(res_row + idx * N) : make_uint4(0, 0, 0, 0);
    if (FEW) wv[v] = ok ? __ldg(reinterpret_cast<const uint4*>(weight + idx * N)) : make_uint4(0, 0, 0, 0);
  }
  float sum_sq = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int idx = t_in_row + v * tpr;
    float fa[N], fb[N];
    Pack<T>::unpack(a[v], fa);
    Pack<T>::unpack(b[v], fb);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      fa[i] += fb[i];
      sum_sq = fmaf(fa[i], fa[i], sum_sq);  // of the unrounded sum, as the reference does
    }
    b[v] = Pack<T>::pack(fa);  // residual, rounded to T; the scaling below uses this rounded value
    if (row_ok && idx < vecs) st_vec<KEEP>(res_row + idx * N, b[v]);
  }
  // sum over the thread group: warp shuffles, then the group's warps through shared memory
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, o);
  if (tpr > 32) {
    if (lane == 0) s_part[warp] = sum_sq;
    __syncthreads();
    const int w0 = (tid / tpr) * (tpr / 32);
    sum_sq = 0.f;
    for (int w = 0; w < tpr / 32; ++w) sum_sq += s_part[w0 + w];
  }
  const float inv_rms = rsqrtf(sum_sq / static_cast<float>(dim) + eps);
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int idx = t_in_row + v * tpr;
    if (!(row_ok && idx < vecs)) continue;
    float fr[N], fw[N];
    Pack<T>::unpack(b[v], fr);
    Pack<T>::unpack(FEW ? wv[FEW ? v : 0] : __ldg(reinterpret_cast<const uint4*>(weight + idx * N)), fw);
#pragma unroll
    for (int i = 0; i < N; ++i) fr[i] = fr[i] * inv_rms * fw[i];
    st_vec<KEEP>(in_row + idx * N, Pack<T>::pack(fr));
  }
}

// Any dim and alignment: one CTA per row, two passes (the second re-reads the
// residual through the cache).
template <typename T>
__global__ void __launch_bounds__(kThreads) add_rms_norm_generic_kernel(T* input, T* residual, const T* weight, int64_t dim,
                                                                        float eps) {
  __shared__ float s_part[kThreads / 32];
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T* in_row = input + static_cast<int64_t>(blockIdx.x) * dim;
  T* res_row = residual + static_cast<int64_t>(blockIdx.x) * dim;
  float sum_sq = 0.f;
  for (int64_t i = tid; i < dim; i += kThreads) {
    const float r = to_f32<T>(in_row[i]) + to_f32<T>(res_row[i]);
    res_row[i] = from_f32<T>(r);
    sum_sq = fmaf(r, r, sum_sq);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, o);
  if (lane == 0) s_part[warp] = sum_sq;
  __syncthreads();
  sum_sq = 0.f;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) sum_sq += s_part[w];
  const float inv_rms = rsqrtf(sum_sq / static_cast<float>(dim) + eps);
  for (int64_t i = tid; i < dim; i += kThreads)
    in_row[i] = from_f32<T>(to_f32<T>(res_row[i]) * inv_rms * to_f32<T>(weight[i]));
}

constexpr int kSiluUnroll = 4;

// silu(g) * u with the fast exponential and reciprocal (the reference's kernel uses __expf as well)
__device__ __forceinline__ float silu_mul1(float g, float u) { return __fdividef(g, 1.f + __expf(-g)) * u; }

template <typename T>
__device__ __forceinline__ uint4 silu_vec(const uint4& g, const uint4& u) {
  constexpr int N = Pack<T>::N;
  float fg[N], fu[N];
  Pack<T>::unpack(g, fg);
  Pack<T>::unpack(u, fu);
#pragma unroll
  for (int i = 0; i < N; ++i) fg[i] = silu_mul1(fg[i], fu[i]);
  return Pack<T>::pack(fg);
}

// x [rows, 2d] -> out [rows, d], long rows: CTA (row, chunk) handles kThreads * kSiluUnroll
// vectors of one row, so that no index needs a division.  vecs_per_row = d / N.
template <typename T, bool KEEP>
__global__ void __launch_bounds__(kThreads) silu_mul_rows_kernel(T* __restrict__ out, const T* __restrict__ x,
                                                                 int vecs_per_row) {
  constexpr int N = Pack<T>::N;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int64_t row = blockIdx.x;
  const int v0 = blockIdx.y * (kThreads * kSiluUnroll) + threadIdx.x;
  const T* gp = x + row * 2 * vecs_per_row * N;
  const T* up = gp + static_cast<int64_t>(vecs_per_row) * N;
  T* op = out + row * vecs_per_row * N;
  uint4 g[kSiluUnroll], u[kSiluUnroll];
#pragma unroll
  for (int k = 0; k < kSiluUnroll; ++k) {
    const int v = v0 + k * kThreads;
    if (v < vecs_per_row) g[k] = ld_vec<KEEP>(gp + v * N), u[k] = ld_vec<KEEP>(up + v * N);
  }
#pragma unroll
  for (int k = 0; k < kSiluUnroll; ++k) {
    const int v = v0 + k * kThreads;
    if (v < vecs_per_row) st_vec<KEEP>(op + v * N, silu_vec<T>(g[k], u[k]));
  }
}

// Short rows: a flat index over all vectors (32-bit arithmetic; the launcher checks the range).
template <typename T>
__global__ void __launch_bounds__(kThreads) silu_mul_kernel(T* __restrict__ out, const T* __restrict__ x, uint32_t total_vecs,
                                                            uint32_t vecs_per_row) {
  constexpr int N = Pack<T>::N;
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const uint32_t idx = blockIdx.x * kThreads + threadIdx.x;
  if (idx >= total_vecs) return;
  const uint32_t row = idx / vecs_per_row, col = idx - row * vecs_per_row;
  const T* gp = x + (static_cast<int64_t>(row) * 2 * vecs_per_row + col) * N;
  st_vec<true>(out + static_cast<int64_t>(idx) * N, silu_vec<T>(ld_vec<true>(gp), ld_vec<true>(gp + static_cast<int64_t>(vecs_per_row) * N)));
}

template <typename T>
__global__ void __launch_bounds__(kThreads) silu_mul_generic_kernel(T* out, const T* x, int64_t n, int64_t d) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  if (i >= n) return;
  const int64_t row = i / d, col = i - row * d;
  const float g = to_f32<T>(x[row * 2 * d + col]), u = to_f32<T>(x[row * 2 * d + d + col]);
  out[i] = from_f32<T>(silu_mul1(g, u));
}

// out[c] = sum over the rows of x[rows, n] (row stride ld) in fp32, rounded once.  A CTA is one warp: 16 lanes across (128
// columns, 256 bytes of a row), two rows at a time, 16 loads per lane in flight; the CTAs of a cluster share the rows of
// a block of columns and are summed in rank order through distributed shared memory: no scratch memory, no second
// kernel, and the same result every time.  `beside`: the kernel before in the stream is the gradient product that reads
// the same x; it leaves 1.8 KB of shared memory and most of HBM's bandwidth unused, and 1.5 KB, 1 of them the system's, are all that a CTA
// here asks for, so it runs beside it instead of behind it (32 us of a pass over 4096 x 12288, and 185 us as a copy to
// fp32 and a library reduction).
constexpr int kSumCols = 128;

template <typename T>
__global__ void __launch_bounds__(32) column_sums_kernel(const T* __restrict__ x, T* __restrict__ out, int64_t rows, int64_t n,
                                                         int64_t ld, int cluster, bool beside) {
  constexpr int N = Pack<T>::N;
  static_assert(N == 8, "16-bit types");
  ptx::grid_dep_launch();
  if (!beside) ptx::grid_dep_wait();
  __shared__ __align__(16) float s_sum[kSumCols];
  const int rank = blockIdx.x % cluster, lane = threadIdx.x;
  const int64_t col = static_cast<int64_t>(blockIdx.x / cluster) * kSumCols + (lane % 16) * N;
  const int64_t per = (rows + cluster - 1) / cluster, r0 = rank * per, r1 = r0 + per < rows ? r0 + per : rows;
  float acc[N] = {};
  if (col < n) {
    constexpr int U = 16;
    for (int64_t r = r0 + lane / 16; r < r1; r += 2 * U) {
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = r + 2 * u < r1 ? __ldcg(reinterpret_cast<const uint4*>(x + (r + 2 * u) * ld + col)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float f[N];
        Pack<T>::unpack(v[u], f);
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] += f[i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
  if (lane < 16) {
#pragma unroll
    for (int i = 0; i < N; ++i) s_sum[lane * N + i] = acc[i];
  }
  if (cluster > 1)
    ptx::cluster_sync();
  else
    __syncwarp();
  if (rank == 0) {
    const int64_t c0 = static_cast<int64_t>(blockIdx.x / cluster) * kSumCols + lane * 4;
    if (c0 < n) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int r = 0; r < cluster; ++r) {
        const float4 p = ptx::ld_cluster_f4(ptx::map_rank(ptx::smem_u32(s_sum + lane * 4), r));
        t.x += p.x, t.y += p.y, t.z += p.z, t.w += p.w;
      }
      out[c0] = from_f32<T>(t.x), out[c0 + 1] = from_f32<T>(t.y), out[c0 + 2] = from_f32<T>(t.z), out[c0 + 3] = from_f32<T>(t.w);
    }
  }
  if (cluster > 1) ptx::cluster_sync();  // no CTA leaves while rank 0 still reads its sums
  // what comes after this grid waits for its end only: it does not end before the grid beside it
  if (beside && blockIdx.x == 0) ptx::grid_dep_wait();
}

template <typename T>
cudaError_t sums_t(const void* x, void* out, int64_t rows, int64_t n, int64_t ld, bool beside, cudaStream_t stream) {
  // the rows of a column block are divided while a CTA keeps at least 64 of them
  int cluster = 1;
  while (cluster < 8 && rows >= cluster * 2 * 64) cluster *= 2;
  auto kern = column_sums_kernel<T>;
  // (the SM's shared memory stays divided as the kernel beside needs it)
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return e;
  return launch_early(kern, dim3(static_cast<unsigned>((n + kSumCols - 1) / kSumCols) * cluster), dim3(32), 0, stream, cluster,
                      static_cast<const T*>(x), static_cast<T*>(out), rows, n, ld, cluster, beside);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <typename T>
cudaError_t rms_t(void* input, void* residual, const void* weight, int64_t rows, int64_t dim, float eps,
                  cudaStream_t stream) {
  constexpr int N = Pack<T>::N;
  T* in = static_cast<T*>(input);
  T* res = static_cast<T*>(residual);
  const T* w = static_cast<const T*>(weight);
  const int64_t vecs = dim / N;
  const bool vec_ok = dim % N == 0 && vecs <= kThreads * 8 && aligned16(in) && aligned16(res) && aligned16(w);
  if (!vec_ok) {
    return launch_early(add_rms_norm_generic_kernel<T>, dim3(static_cast<unsigned>(rows)), dim3(kThreads), 0, stream, 1, in, res,
                        w, dim, eps);
  }
  // threads per row: the fewest (>= 32) that keep a thread at <= 8 vectors ... but prefer
  // <= 4 so that enough loads are in flight without starving occupancy; with fewer rows than SMs as many as there are
  // vectors, up to a whole CTA per row
  const bool few = rows < kSms;
  int tpr = 32;
  while (tpr < kThreads && vecs > static_cast<int64_t>(tpr) * (few ? 1 : 4)) tpr <<= 1;
  const int vpt = static_cast<int>((vecs + tpr - 1) / tpr);
  const int rows_per_cta = kThreads / tpr;
  const unsigned grid = static_cast<unsigned>((rows + rows_per_cta - 1) / rows_per_cta);
  const int d = static_cast<int>(dim);
  const bool keep = 2 * rows * dim * static_cast<int64_t>(sizeof(T)) <= kKeepBytes;
#define TT_RMS(V) \
  (few ? add_rms_norm_kernel<T, V, true, true> : keep ? add_rms_norm_kernel<T, V, false, true> : add_rms_norm_kernel<T, V, false, false>)
  auto kern = vpt <= 1 ? TT_RMS(1) : vpt <= 2 ? TT_RMS(2) : vpt <= 4 ? TT_RMS(4) : TT_RMS(8);
#undef TT_RMS
  return launch_early(kern, dim3(grid), dim3(kThreads), 0, stream, 1, in, res, w, rows, d, tpr, eps);
}

template <typename T>
cudaError_t silu_t(void* out, const void* x, int64_t rows, int64_t d, cudaStream_t stream) {
  constexpr int N = Pack<T>::N;
  T* o = static_cast<T*>(out);
  const T* xi = static_cast<const T*>(x);
  const int64_t vpr = d / N, total = rows * vpr;
  const bool vec_ok = d % N == 0 && aligned16(o) && aligned16(xi);
  constexpr int kChunk = kThreads * kSiluUnroll;
  // (a handful of rows: one vector per thread, four times the CTAs)
  const bool few = rows * ((vpr + kChunk - 1) / kChunk) < kSms;
  if (vec_ok && !few && vpr >= kThreads && (vpr + kChunk - 1) / kChunk <= 65535 && rows <= 0x7fffffff) {
    dim3 grid(static_cast<unsigned>(rows), static_cast<unsigned>((vpr + kChunk - 1) / kChunk));
    const bool keep = 3 * rows * d * static_cast<int64_t>(sizeof(T)) <= kKeepBytes;
    return launch_early(keep ? silu_mul_rows_kernel<T, true> : silu_mul_rows_kernel<T, false>, grid, dim3(kThreads), 0, stream, 1, o,
                        xi, static_cast<int>(vpr));
  }
  if (vec_ok && total < 0x7fffff00ll)
    return launch_early(silu_mul_kernel<T>, dim3(static_cast<unsigned>((total + kThreads - 1) / kThreads)), dim3(kThreads), 0,
                        stream, 1, o, xi, static_cast<uint32_t>(total), static_cast<uint32_t>(vpr));
  const int64_t n = rows * d;
  return launch_early(silu_mul_generic_kernel<T>, dim3(static_cast<unsigned>((n + kThreads - 1) / kThreads)), dim3(kThreads), 0,
                      stream, 1, o, xi, n, d);
}

}  // namespace

cudaError_t launch_fused_add_rms_norm(int dtype, void* input, void* residual, const void* weight, int64_t rows,
                                      int64_t dim, float eps, cudaStream_t stream) {
  if (dtype == TT_ATTN_F32) return rms_t<float>(input, residual, weight, rows, dim, eps, stream);
  if (dtype == TT_ATTN_F16) return rms_t<__half>(input, residual, weight, rows, dim, eps, stream);
  return rms_t<__nv_bfloat16>(input, residual, weight, rows, dim, eps, stream);
}

cudaError_t launch_column_sums(int dtype, const void* x, void* out, int64_t rows, int64_t n, int64_t ldx, bool beside,
                               cudaStream_t stream) {
  return dtype == TT_ATTN_F16 ? sums_t<__half>(x, out, rows, n, ldx, beside, stream)
                              : sums_t<__nv_bfloat16>(x, out, rows, n, ldx, beside, stream);
}

cudaError_t launch_silu_mul(int dtype, void* out, const void* x, int64_t rows, int64_t d, cudaStream_t stream) {
  if (dtype == TT_ATTN_F32) return silu_t<float>(out, x, rows, d, stream);
  if (dtype == TT_ATTN_F16) return silu_t<__half>(out, x, rows, d, stream);
  return silu_t<__nv_bfloat16>(out, x, rows, d, stream);
}

}  // namespace ttattn
