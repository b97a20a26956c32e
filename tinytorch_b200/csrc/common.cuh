// Shared host/device declarations of the attention library's internal launchers.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/tt_attn.h"
#include "ptx.cuh"

namespace ttattn {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// SMs of the part this library is written for: plans that the workspace query makes too, without a device at hand, divide by
// it (the planners of the projections and of the prefill forward ask the device).
constexpr int kSms = 148;

// Status bits a kernel may OR into the caller's status word.
constexpr int kStatusWaitExpired = 1;
constexpr int kStatusBadSmemAlign = 2;   // dynamic shared memory did not start on a 1024-byte boundary
constexpr int kStatusCacheFull = 4;      // decode-append: no free row in the cache of some sequence
constexpr int kStatusRopeRange = 8;      // decode-append: position beyond the rotary tables

// two values, rounded to the 16-bit type, in one register
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (BF16) {
    __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
  } else {
    __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
  }
}

struct Str3 {
  int64_t b, h, s;
};

inline Str3 dense_or(const tt_attn_strides& st, int64_t H, int64_t S, int64_t D) {
  if (st.b == 0 && st.h == 0 && st.s == 0) return Str3{H * S * D, S * D, D};
  return Str3{st.b, st.h, st.s};
}

// Optional mask, broadcast against [B, Hq, Lq, Skv]; the key dimension is contiguous.
struct MaskArgs {
  const void* ptr;  // null: no mask
  int kind;         // tt_attn_mask_kind
  int64_t sb, sh, sl;
  bool wide;        // every row starts on a 16-byte boundary
};

// Arguments common to the prefill kernels.
struct FwdArgs {
  const void* q;
  const void* k;
  const void* v;
  void* o;
  float* lse;
  Str3 qs, ks, vs, os;
  int B, Hq, Hkv, Lq, Skv;
  int causal;  // tt_attn_causal
  float scale;
  const int32_t* kv_lens;
  int32_t* status;
  MaskArgs mask;
  int* sched;  // tensor-core path: work counter in scratch memory
  int32_t* mask_lens;        // tensor-core path: scratch of 2 B integers for masked_lens, or null: a padding mask is read in full
  const int32_t* mask_pure;  // with masked_lens: whether the mask is all true up to the length
};

struct BwdArgs {
  const void* q;
  const void* k;
  const void* v;
  const void* o;
  const void* d_o;
  const float* lse;
  float* delta;     // workspace [B, Hq, Lq]
  float* dq_accum;  // workspace [B, Hq, Lq, D] fp32 (tensor-core path), zeroed by the delta pre-pass
  int zero_dq_accum;  // set by the tensor-core launcher: the delta kernel also clears dq_accum
  int tail_heads;     // tensor-core kernel: (batch, kv head) pairs at the end of the item order whose key tiles are
                      // ordered longest walk first across heads (set by its launcher)
  int* sched;         // tensor-core kernel: work counter in scratch memory, zeroed by the delta pre-pass
  int parts;          // tensor-core kernel: work items per key tile (see bwd_parts); > 1: each leaves its dK / dV in ...
  float* dkv_part;    // ... workspace [dK, dV][parts][B * Hkv][Skv][D] fp32
  float2* row_stats;  // fp32 kernels with an additive mask: workspace [B, Hq, Lq] for what a row's probabilities are made with (see exponent_base), or null
  float* ds;          // fp32 kernels: dS on its way from the dK / dV pass to the dQ pass, or null (see bwd_ds_bytes)
  void* dq;
  void* dk;
  void* dv;
  Str3 qs, ks, vs, os, dos, dqs, dks, dvs;
  int B, Hq, Hkv, Lq, Skv;
  int causal;  // tt_attn_causal
  float scale;
  const int32_t* kv_lens;
  int32_t* status;
  MaskArgs mask;
  int32_t* mask_lens;        // as in FwdArgs
  const int32_t* mask_pure;  // as in FwdArgs
};

struct DecodeArgs {
  const void* q;
  const void* k;
  const void* v;
  void* o;
  float* lse;
  float* partial;  // workspace [B, Hq, nsplit, D + 2] when nsplit > 1
  Str3 qs, ks, vs, os;
  int B, Hq, Hkv, capacity;
  int nsplit, chunk;
  float scale;
  const int32_t* kv_lens;
  // append variant only: the step's new key / value row per (b, kv head), rotary tables, outputs
  const void* k_new;
  const void* v_new;
  int64_t kn_b, kn_h, vn_b, vn_h;  // element strides of k_new / v_new
  const float* rope_cos;           // [rope_positions, D/2] or null: no rotation
  const float* rope_sin;
  int rope_positions;
  int rope_interleaved;            // pairs (2i, 2i+1) instead of (i, i + D/2)
  int32_t* new_lens;               // optional [B]: kv_lens[b] + 1
  int32_t* status;
  int* sched;                      // tensor-core path: work counter in scratch memory, zeroed ahead of the scan (see chained)
  void* q_rot;                     // append on the tensor-core path: scratch [B, Hq, D] for the rotated q
  int32_t* lens_scratch;           // ... and [B] for the lengths after the append
  int chained;                     // tensor-core path: the kernel before this one in the stream has zeroed the
                                   // work counter
  const int32_t* lens_hint;        // tensor-core path: lengths that may be read while the kernel before this one
                                   // still runs, good enough to ask for cache rows in L2 (or null)
};

// Each returns a cudaError_t from the launch (no synchronisation).
cudaError_t launch_fwd_tc(int dtype, int D, const FwdArgs& a, int device, cudaStream_t stream);
cudaError_t launch_fwd_f32(int D, const FwdArgs& a, int device, cudaStream_t stream);
// (take_ds: dQ of a.ds, if it is there, as planned or in any case)
cudaError_t launch_bwd_f32(int D, const BwdArgs& a, bool take_ds, int device, cudaStream_t stream);
// rowsum(dO o O) into a.delta only (first step of every backward)
cudaError_t launch_bwd_delta(int dtype, int D, const BwdArgs& a, cudaStream_t stream);
// Work items per key tile of the tensor-core backward, and the workspace they need beside dq_accum (0 for one item)
int bwd_parts(int B, int Hq, int Hkv, int Lq, int Skv, int D, bool causal);
size_t bwd_part_bytes(int B, int Hq, int Hkv, int Lq, int Skv, int D);
size_t bwd_part_bytes_of(int parts, int B, int Hkv, int Skv, int D);
// dS of the fp32 backward (0: dQ recomputes it; a caller without room for it gets that too)
size_t bwd_ds_bytes(int B, int Hq, int Hkv, int Lq, int Skv, int D);
double bwd_ds_bytes_of(int B, int Hq, int Lq, int Skv);  // ... of any size
bool bwd_f32_takes_ds(int D, const BwdArgs& a, int device);  // whether the call makes dQ of it, given room
// fp16 / bf16 backward on the tensor cores; needs a.delta, a.dq_accum and what a.parts asks for
cudaError_t launch_bwd_tc(int dtype, int D, const BwdArgs& a, int device, cudaStream_t stream);
cudaError_t launch_decode(int dtype, int D, const DecodeArgs& a, cudaStream_t stream);
// grouped-query decode on the tensor cores (decode_tc.cu): 16-bit tensors, 2..16 query heads per kv head
bool decode_tc_applies(int dtype, int D, const DecodeArgs& a);
cudaError_t launch_decode_tc(int dtype, int D, const DecodeArgs& a, cudaStream_t stream);
// rotary embedding of q and the new key, append of the new key / value row, then the same scan
cudaError_t launch_decode_append(int dtype, int D, const DecodeArgs& a, cudaStream_t stream);

cudaError_t launch_decode_static(int dtype, int D, DecodeArgs a, size_t need, int device, cudaStream_t stream,
                                 bool* too_large);

// The reference's two fused transformer-block operators (fused_ops.cu).
cudaError_t launch_fused_add_rms_norm(int dtype, void* input, void* residual, const void* weight, int64_t rows,
                                      int64_t dim, float eps, cudaStream_t stream);
cudaError_t launch_silu_mul(int dtype, void* out, const void* x, int64_t rows, int64_t d, cudaStream_t stream);

// y = x w^T + bias on the tensor cores; ld* are row strides in elements, x_t / w_t as in tt_linear_params
struct LinearCall {
  int dtype;
  const void* x;
  const void* w;
  const void* bias;
  void* y;
  int M, N, K;
  int64_t ldx, ldw, ldy;
  bool x_t, w_t;
  int32_t* status;
  int device;
  cudaStream_t stream;
};
// Cache lines that 128 bytes of a row cost: rows of `ld` 16-bit elements that are not a multiple of a line long touch two, and five
// sectors instead of four where they are not a multiple of a sector (from the fits in linear_tile.cu and linear_split.cu).
inline double row_lines(int64_t ld) { return ld % 16 ? 1.74 : (ld % 64 ? 1.17 : 1.0); }
// *persistent: a kernel was taken beside which launch_column_sums may run
cudaError_t launch_linear_tc(const LinearCall& c, bool* persistent = nullptr);
// What it takes: 0, the contraction divided; single CTAs: the columns of a tile; pairs: minus the columns of a tile.
int linear_shape(const LinearCall& c);
// ... with tiles made to measure (linear_tile.cu): single CTAs with 128 x `bn`, or pairs with 256 x 192
double linear_tile_us(const LinearCall& c, bool pair, int bn);  // what it, or pairs with 256 x 256, are expected to take
bool linear_tile_fits(const LinearCall& c, bool pair, int bn);  // whether there is such a tile for operands stored like these
cudaError_t launch_linear_tile(const LinearCall& c, bool pair, int bn);
// ... for outputs with too few tiles to occupy the machine: contraction split over clusters (linear_split.cu)
struct SplitPlan {
  int mt, tiles_m, tiles, cluster, stages, smem;
  int per_sm, waves;
  double hbm_rate;  // bytes per us
  double us;        // what it is expected to take, among plans
};
SplitPlan plan_linear_split(const LinearCall& c);
double linear_split_us(const LinearCall& c, const SplitPlan& p);  // ... beside the other kernels
cudaError_t launch_linear_split(const LinearCall& c, const SplitPlan& p);
// out[n] = sum over the rows of x[rows, n] (fused_ops.cu); n and ldx are multiples of 8
// `beside`: the kernel launched just before is linear_tc_kernel or linear_tile_kernel, whose CTAs let this one in once all before
// them is complete (grid_dep_launch behind grid_dep_wait) and leave the 1.5 KB of shared memory that a CTA here takes
cudaError_t launch_column_sums(int dtype, const void* x, void* out, int64_t rows, int64_t n, int64_t ldx, bool beside,
                               cudaStream_t stream);

// one CTA waiting `limit_ns` on an mbarrier nobody arrives on (selftest.cu)
cudaError_t launch_wait_expiry(int32_t* status, uint64_t limit_ns, unsigned long long* waited_ns, cudaStream_t stream);

// Split planning for decode, shared by the launcher and the workspace query.
void decode_plan(int B, int Hkv, int capacity, int* nsplit, int* chunk);
// ... for the tensor-core path (several query heads per kv head): longer chunks, see decode.cu
void decode_plan_for(int dtype, int D, int B, int Hq, int Hkv, int capacity, int* nsplit, int* chunk);
size_t decode_scratch_bytes(int dtype, int D, int B, int Hq, int Hkv, int nsplit);  // what a plan's partial results take
// ... in `room` bytes of scratch: longer chunks, up to those of a large batch, where the partial results would not fit
size_t decode_plan_within(int dtype, int D, int B, int Hq, int Hkv, int capacity, size_t room, int* nsplit, int* chunk);

// Launches a kernel that calls ptx::grid_dep_wait() before it touches global memory: it may come up, and set itself up,
// while the kernel before it in the stream ends (or, if that one allows it, still runs).  `cluster`: CTAs per cluster.
template <typename... P, typename... A>
cudaError_t launch_early(void (*kern)(P...), dim3 grid, dim3 block, int smem, cudaStream_t stream, int cluster, A... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster, attr[1].val.clusterDim.y = 1, attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr, cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// Zeroes a work counter ahead of the kernel that draws from it: 1 us between two kernels that are launched early, where a
// memset, which waits for the one and is waited for by the other, takes 3.3.
static __global__ void zero_word_kernel(int* word) {
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  if (threadIdx.x == 0) *word = 0;
}
inline cudaError_t launch_zero_word(int* word, cudaStream_t stream) {
  return launch_early(zero_word_kernel, dim3(1), dim3(32), 0, stream, 1, word);
}

// Scratch integers of the tensor-core prefill kernels: the work counter and, for a padding mask, a length and a flag per
// sequence.  (The counter alone: 256 bytes, as every scratch block is rounded up to.)
constexpr size_t scratch_words(int B) { return 1 + 2 * static_cast<size_t>(B); }

// A boolean mask that is the same for all heads and rows is most often padding: true up to a length.  Its sequences are
// then worth no more than that many keys, and within them the mask need not be looked at.  (Not under the bottom-right
// alignment, which is taken from the number of cache rows.)
inline bool is_padding_mask(const MaskArgs& m, int causal) {
  return m.ptr && m.kind == TT_ATTN_MASK_BOOL && m.sh == 0 && m.sl == 0 && causal != TT_ATTN_CAUSAL_BOTTOM_RIGHT;
}
// By all threads of a CTA: lens[b] = 1 + the last key that takes part, pure[b] = whether all before it do.
__device__ __forceinline__ void masked_lens(const MaskArgs& m, const int32_t* kv_lens, int Skv, int b, int32_t* lens,
                                            int32_t* pure) {
  __shared__ int s_last, s_count;
  if (threadIdx.x == 0) s_last = 0, s_count = 0;
  __syncthreads();
  int len = Skv;
  if (kv_lens) {
    const int l = kv_lens[b];
    len = l < 0 ? 0 : (l < Skv ? l : Skv);
  }
  const uint8_t* p = reinterpret_cast<const uint8_t*>(m.ptr) + b * m.sb;
  const int lead = static_cast<int>(reinterpret_cast<uintptr_t>(p) & 15), n = (lead + len + 15) / 16;
  int last = 0, count = 0;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {  // the aligned vectors that hold the row
    const uint4 v = reinterpret_cast<const uint4*>(p - lead)[j];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int key = j * 16 + i - lead;
      if (key >= 0 && key < len && ((w[i / 4] >> (i % 4 * 8)) & 0xffu)) last = key + 1, ++count;
    }
  }
  last = __reduce_max_sync(0xffffffffu, last);
  count = __reduce_add_sync(0xffffffffu, count);
  if (threadIdx.x % 32 == 0 && count > 0) atomicMax(&s_last, last), atomicAdd(&s_count, count);
  __syncthreads();
  if (threadIdx.x == 0) lens[b] = s_last, pure[b] = s_count == s_last;
  __syncthreads();
}

template <typename T>
__device__ __forceinline__ float to_f32(T x);
template <>
__device__ __forceinline__ float to_f32<float>(float x) {
  return x;
}
template <>
__device__ __forceinline__ float to_f32<__half>(__half x) {
  return __half2float(x);
}
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) {
  return __bfloat162float(x);
}
template <typename T>
__device__ __forceinline__ T from_f32(float x);
template <>
__device__ __forceinline__ float from_f32<float>(float x) {
  return x;
}
template <>
__device__ __forceinline__ __half from_f32<__half>(float x) {
  return __float2half_rn(x);
}
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) {
  return __float2bfloat16_rn(x);
}


// Query i sees key j under a causal mask iff j <= i + causal_shift(...).
__host__ __device__ __forceinline__ int causal_shift(int causal, int kv_len, int Lq) {
  return causal == TT_ATTN_CAUSAL_BOTTOM_RIGHT ? kv_len - Lq : 0;
}

}  // namespace ttattn
