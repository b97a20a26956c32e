// extern "C" entry points of libtt_attn.so: argument validation, workspace
// handling through the caller's allocator hook, device guard, kernel dispatch.
// See include/tt_attn.h for the contract of each function.
#include <cstddef>
#include <cstdio>
#include <cstring>

#include "../../include/tt_fused.h"
#include "common.cuh"
#include "tma_host.cuh"

namespace ttattn {
namespace {

thread_local char g_cuda_error[256] = "";

int launch_failed(cudaError_t e) {
  std::snprintf(g_cuda_error, sizeof(g_cuda_error), "%s: %s", cudaGetErrorName(e), cudaGetErrorString(e));
  return TT_ATTN_ERR_LAUNCH;
}

// Equivalent of the reference's CudaDeviceGuard (src/Utils/CUDAUtils.h:100-113).
struct DeviceGuard {
  int prev = -1;
  bool ok = false;
  explicit DeviceGuard(int device) {
    if (cudaGetDevice(&prev) != cudaSuccess) return;
    ok = (prev == device) || cudaSetDevice(device) == cudaSuccess;
    if (prev == device) prev = -1;
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

inline size_t elem_size(int dtype) { return dtype == TT_ATTN_F32 ? 4 : 2; }
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline bool strides_ok(const Str3& s, size_t es) {
  return s.b >= 0 && s.h >= 0 && s.s > 0 && (s.b * es) % 16 == 0 && (s.h * es) % 16 == 0 && (s.s * es) % 16 == 0;
}
inline size_t round256(size_t n) { return (n + 255) & ~size_t(255); }

// Scratch memory for one call: the caller's buffer, or a block from the hook
// that is handed back when this object goes out of scope (after the launches
// have been enqueued; reuse is stream-ordered).
struct Workspace {
  void* ptr = nullptr;
  const tt_attn_alloc_hook* hook = nullptr;
  int device = 0;
  bool owned = false;
  int acquire(size_t need, void* user, size_t user_bytes, const tt_attn_alloc_hook* h, int dev) {
    if (need == 0) return TT_ATTN_OK;
    if (user) {
      if (user_bytes < need) return TT_ATTN_ERR_WORKSPACE;
      if (!aligned16(user)) return TT_ATTN_ERR_ALIGN;
      ptr = user;
      return TT_ATTN_OK;
    }
    if (!h || !h->alloc || !h->free) return TT_ATTN_ERR_WORKSPACE;
    ptr = h->alloc(h->ctx, need, dev);
    if (!ptr) return TT_ATTN_ERR_WORKSPACE;
    hook = h, device = dev, owned = true;
    return TT_ATTN_OK;
  }
  ~Workspace() {
    if (owned) hook->free(hook->ctx, ptr, device);
  }
};

int check_common(int dtype, int B, int Hq, int Hkv, int Lq, int Skv, int D) {
  if (dtype != TT_ATTN_F32 && dtype != TT_ATTN_F16 && dtype != TT_ATTN_BF16) return TT_ATTN_ERR_DTYPE;
  if (B <= 0 || Hq <= 0 || Hkv <= 0 || Lq <= 0 || Skv <= 0 || Hq % Hkv != 0) return TT_ATTN_ERR_SHAPE;
  if (D != 64 && D != 128) return TT_ATTN_ERR_HEAD_DIM;
  if (B > 65535 || Hq > 65535) return TT_ATTN_ERR_TOO_LARGE;  // grid.y / grid.z
  return TT_ATTN_OK;
}

}  // namespace
}  // namespace ttattn

using namespace ttattn;

// What tt_linear is asked for, checked; sums_only: just the sums of x (w and y, and what describes them, are not looked at).
static int linear_call(const tt_linear_params* p, LinearCall* c, bool* sums_only) {
  if (!p) return TT_ATTN_ERR_NULL;
  const bool ext = p->struct_size == sizeof(tt_linear_params);
  if (!ext && p->struct_size != offsetof(tt_linear_params, x_t)) return TT_ATTN_ERR_STRUCT;
  if (p->dtype != TT_ATTN_F16 && p->dtype != TT_ATTN_BF16) return TT_ATTN_ERR_DTYPE;
  if (p->M < 0 || p->N <= 0 || p->K <= 0 || p->M > 0x7fffffff || p->N > 0x7fffffff || p->K > 0x7fffffff)
    return TT_ATTN_ERR_SHAPE;
  const bool x_t = ext && p->x_t != 0, w_t = ext && p->w_t != 0;
  const void* x_sum = ext ? p->x_sum : nullptr;
  const int64_t x_cols = x_t ? p->M : p->K, w_cols = w_t ? p->N : p->K;  // the contiguous dimensions
  const int64_t ldx = p->ldx ? p->ldx : x_cols, ldw = p->ldw ? p->ldw : w_cols, ldy = p->ldy ? p->ldy : p->N;
  *c = LinearCall{p->dtype, p->x, p->w, p->bias, p->y, static_cast<int>(p->M), static_cast<int>(p->N), static_cast<int>(p->K),
                  ldx, ldw, ldy, x_t, w_t, p->status, p->device, static_cast<cudaStream_t>(p->stream)};
  *sums_only = x_sum && !p->w && !p->y;
  if (p->M == 0) return TT_ATTN_OK;
  if (!p->x || (!*sums_only && (!p->w || !p->y))) return TT_ATTN_ERR_NULL;
  if (x_sum && !x_t) return TT_ATTN_ERR_SHAPE;
  if (ldx < x_cols || ldw < w_cols || ldy < p->N) return TT_ATTN_ERR_SHAPE;
  auto odd = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 2 != 0; };
  if (x_cols % 8 || ldx % 8 || !aligned16(p->x) || odd(x_sum)) return TT_ATTN_ERR_ALIGN;
  if (!*sums_only && (w_cols % 8 || p->N % 8 || ldw % 8 || ldy % 8 || !aligned16(p->w) || !aligned16(p->y) || odd(p->bias)))
    return TT_ATTN_ERR_ALIGN;
  return TT_ATTN_OK;
}

extern "C" {

int tt_attn_version(void) { return TT_ATTN_ABI_VERSION; }

const char* tt_attn_last_cuda_error(void) { return g_cuda_error; }

const char* tt_attn_strerror(int status) {
  switch (status) {
    case TT_ATTN_OK: return "ok";
    case TT_ATTN_ERR_NULL: return "a required pointer is NULL";
    case TT_ATTN_ERR_DTYPE: return "unsupported dtype (expected 0=Float32, 1=Float16, 2=BFloat16)";
    case TT_ATTN_ERR_SHAPE: return "invalid shape";
    case TT_ATTN_ERR_HEAD_DIM: return "head dimension must be 64 or 128";
    case TT_ATTN_ERR_ALIGN: return "pointers and strides must be 16-byte aligned";
    case TT_ATTN_ERR_WORKSPACE: return "workspace too small, or allocator hook missing / returned NULL";
    case TT_ATTN_ERR_LAUNCH: return "CUDA launch error (see tt_attn_last_cuda_error)";
    case TT_ATTN_ERR_STRUCT: return "parameter struct size mismatch";
    case TT_ATTN_ERR_NO_DEVICE: return "invalid device or CUDA driver entry point unavailable";
    case TT_ATTN_ERR_TOO_LARGE: return "size beyond a fixed limit of this library";
    default: return "unknown status";
  }
}

}  // extern "C"

namespace {
// Validates the optional mask of a prefill call.
int take_mask(const void* ptr, int kind, const int64_t st[3], MaskArgs* m) {
  *m = MaskArgs{};
  if (kind == TT_ATTN_MASK_NONE || !ptr) return (kind == TT_ATTN_MASK_NONE) ? TT_ATTN_OK : TT_ATTN_ERR_NULL;
  if (kind < 0 || kind > TT_ATTN_MASK_ADD_F32) return TT_ATTN_ERR_DTYPE;
  if (st[0] < 0 || st[1] < 0 || st[2] < 0) return TT_ATTN_ERR_SHAPE;
  m->ptr = ptr, m->kind = kind, m->sb = st[0], m->sh = st[1], m->sl = st[2];
  const int64_t esz = kind == TT_ATTN_MASK_BOOL ? 1 : (kind == TT_ATTN_MASK_ADD_F32 ? 4 : 2);
  m->wide = ((reinterpret_cast<uintptr_t>(ptr) | (m->sb * esz) | (m->sh * esz) | (m->sl * esz)) & 15) == 0;
  return TT_ATTN_OK;
}
// Whether the lengths that a padding mask comes to have a place in the scratch memory (of `room` bytes, `used` of them taken);
// a caller who knows of the work counter only, or whose mask is of another kind, needs 256 bytes.
bool mask_lens_fit(const MaskArgs& m, int causal, int B, size_t room, size_t used) {
  return is_padding_mask(m, causal) && room >= used + round256(scratch_words(B) * sizeof(int));
}

// The fused decode step on the tensor-core path, beside the scan's scratch: the rotated q and the new lengths.
size_t append_bytes(int dtype, int B, int Hq, int Hkv, int D) {
  DecodeArgs probe{};
  probe.Hq = Hq, probe.Hkv = Hkv;
  if (!decode_tc_applies(dtype, D, probe)) return 0;
  return round256(static_cast<size_t>(B) * Hq * D * elem_size(dtype)) + round256(static_cast<size_t>(B) * 4);
}
}  // namespace

// The backward, and how the fp32 one comes to dQ: as planned, as the selftest says, or not at all (kAsked: the plan is asked for).
enum BwdPath { kPlanned, kAsked, kRecompute, kStore };
static int bwd_call(const tt_attn_bwd_params* p, BwdPath path, int32_t* planned) {
  if (!p) return TT_ATTN_ERR_NULL;
  const bool v2 = p->struct_size == sizeof(tt_attn_bwd_params);
  if (!v2 && p->struct_size != offsetof(tt_attn_bwd_params, mask)) return TT_ATTN_ERR_STRUCT;
  if (int rc = check_common(p->dtype, p->B, p->Hq, p->Hkv, p->Lq, p->Skv, p->D)) return rc;
  if (!p->q || !p->k || !p->v || !p->o || !p->d_o || !p->lse) return TT_ATTN_ERR_NULL;
  if (path != kPlanned && p->dtype != TT_ATTN_F32) return TT_ATTN_ERR_DTYPE;
  if (path == kStore && !(p->dq && (p->dk || p->dv))) return TT_ATTN_ERR_SHAPE;
  if (path == kAsked) *planned = 0;
  if (!p->dq && !p->dk && !p->dv) return TT_ATTN_OK;
  const size_t es = elem_size(p->dtype);
  BwdArgs a{};
  a.q = p->q, a.k = p->k, a.v = p->v, a.o = p->o, a.d_o = p->d_o, a.lse = p->lse;
  a.dq = p->dq, a.dk = p->dk, a.dv = p->dv;
  a.qs = dense_or(p->q_strides, p->Hq, p->Lq, p->D);
  a.ks = dense_or(p->k_strides, p->Hkv, p->Skv, p->D);
  a.vs = dense_or(p->v_strides, p->Hkv, p->Skv, p->D);
  a.os = dense_or(p->o_strides, p->Hq, p->Lq, p->D);
  a.dos = dense_or(p->do_strides, p->Hq, p->Lq, p->D);
  a.dqs = dense_or(p->dq_strides, p->Hq, p->Lq, p->D);
  a.dks = dense_or(p->dk_strides, p->Hkv, p->Skv, p->D);
  a.dvs = dense_or(p->dv_strides, p->Hkv, p->Skv, p->D);
  const void* ptrs[] = {p->q, p->k, p->v, p->o, p->d_o, p->dq, p->dk, p->dv, p->lse};
  for (const void* q : ptrs)
    if (!aligned16(q)) return TT_ATTN_ERR_ALIGN;
  const Str3* sts[] = {&a.qs, &a.ks, &a.vs, &a.os, &a.dos, &a.dqs, &a.dks, &a.dvs};
  for (const Str3* s : sts)
    if (!strides_ok(*s, es)) return TT_ATTN_ERR_ALIGN;
  a.B = p->B, a.Hq = p->Hq, a.Hkv = p->Hkv, a.Lq = p->Lq, a.Skv = p->Skv;
  if (p->is_causal < 0 || p->is_causal > TT_ATTN_CAUSAL_BOTTOM_RIGHT) return TT_ATTN_ERR_SHAPE;
  a.causal = p->is_causal;
  a.scale = p->scale;
  a.kv_lens = p->kv_lens;
  a.status = p->status;
  if (v2)
    if (int rc = take_mask(p->mask, p->mask_kind, p->mask_strides, &a.mask)) return rc;
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  Workspace ws;
  // delta | dQ accumulator | shares of dK / dV | work counter and, if they fit, a padding mask's lengths; fp32: delta | dS | rows' maxima and sums
  const size_t rows = static_cast<size_t>(p->B) * p->Hq * p->Lq, delta = round256(rows * sizeof(float));
  const size_t accum = round256(rows * p->D * sizeof(float)), room = p->workspace ? p->workspace_bytes : SIZE_MAX;
  size_t need = delta, part = 0;
  bool lens = false;
  // fp32: dS tiles on their way from dK / dV to dQ, where dQ and at least one of the others are asked for and there is room
  size_t ds = p->dtype == TT_ATTN_F32 && p->dq && (p->dk || p->dv) ? round256(bwd_ds_bytes(p->B, p->Hq, p->Hkv, p->Lq, p->Skv, p->D)) : 0;
  if (path == kStore) ds = round256(static_cast<size_t>(bwd_ds_bytes_of(p->B, p->Hq, p->Lq, p->Skv)));
  if (path == kRecompute || delta + ds > room) ds = 0;
  if (path == kStore && ds == 0) return TT_ATTN_ERR_WORKSPACE;
  // ... and, with an additive mask, maxima and sums of the rows whose log-sum-exp is too large to say both
  size_t stats = p->dtype == TT_ATTN_F32 && a.mask.ptr && a.mask.kind != TT_ATTN_MASK_BOOL ? round256(rows * sizeof(float2)) : 0;
  if (delta + ds + stats > room) stats = 0;
  if (p->dtype != TT_ATTN_F32) {
    // a buffer that is too small for the division (a small batch is divided further than a large one): fewer shares
    a.parts = bwd_parts(p->B, p->Hq, p->Hkv, p->Lq, p->Skv, p->D, p->is_causal != 0);
    while (a.parts > 1 && delta + accum + round256(bwd_part_bytes_of(a.parts, p->B, p->Hkv, p->Skv, p->D)) + 256 > room) --a.parts;
    part = round256(bwd_part_bytes_of(a.parts, p->B, p->Hkv, p->Skv, p->D));
    need = delta + accum + part;
    lens = mask_lens_fit(a.mask, a.causal, p->B, room, need);
    need += lens ? round256(scratch_words(p->B) * sizeof(int)) : 256;
  }
  if (path == kAsked) {
    *planned = ds > 0 && bwd_f32_takes_ds(p->D, a, p->device);
    return TT_ATTN_OK;
  }
  if (ds + stats == 0 || ws.acquire(need + ds + stats, p->workspace, p->workspace_bytes, p->alloc, p->device) != TT_ATTN_OK) {
    ds = stats = 0;  // (an allocator that has no more than before)
    if (int rc = ws.acquire(need, p->workspace, p->workspace_bytes, p->alloc, p->device)) return rc;
  }
  a.delta = static_cast<float*>(ws.ptr);
  if (ds > 0) a.ds = reinterpret_cast<float*>(static_cast<char*>(ws.ptr) + delta);
  if (stats > 0) a.row_stats = reinterpret_cast<float2*>(static_cast<char*>(ws.ptr) + delta + ds);
  if (p->dtype != TT_ATTN_F32) {
    a.dq_accum = reinterpret_cast<float*>(static_cast<char*>(ws.ptr) + delta);
    a.dkv_part = reinterpret_cast<float*>(static_cast<char*>(ws.ptr) + delta + accum);
    a.sched = reinterpret_cast<int*>(static_cast<char*>(ws.ptr) + delta + accum + part);
    a.mask_lens = lens ? a.sched + 1 : nullptr;
  }
  if (path == kStore && ds == 0) return TT_ATTN_ERR_WORKSPACE;
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  cudaError_t e = p->dtype == TT_ATTN_F32 ? launch_bwd_f32(p->D, a, path == kStore, p->device, stream)
                                          : launch_bwd_tc(p->dtype, p->D, a, p->device, stream);
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

extern "C" {

size_t tt_attn_workspace_bytes(int kind, int dtype, int B, int Hq, int Hkv, int Lq, int Skv, int D) {
  if (B <= 0 || Hq <= 0 || D <= 0) return 0;
  // fp16 / bf16 forward: one work counter for the persistent kernel's scheduler, and the lengths that a padding mask
  // comes to (a call without such a mask takes 256 bytes of it)
  if (kind == TT_ATTN_KIND_FWD) return dtype == TT_ATTN_F32 ? 0 : round256(scratch_words(B) * sizeof(int));
  if (kind == TT_ATTN_KIND_BWD) {
    // delta [B,Hq,Lq] fp32; the fp16 / bf16 path adds an fp32 dQ accumulator [B,Hq,Lq,D]
    const size_t rows = static_cast<size_t>(B) * Hq * (Lq > 0 ? Lq : 0);
    // and the persistent kernel's work counter
    if (dtype == TT_ATTN_F32) {
      const size_t ds = round256(bwd_ds_bytes(B, Hq, Hkv, Lq, Skv, D));
      return round256(rows * sizeof(float)) + ds + (ds > 0 ? round256(rows * sizeof(float2)) : 0);
    }
    // (and, where few key tiles are divided among several work items, their partial dK / dV)
    return round256(rows * sizeof(float)) + round256(rows * D * sizeof(float)) +
           round256(bwd_part_bytes(B, Hq, Hkv, Lq, Skv, D)) + round256(scratch_words(B) * sizeof(int));
  }
  if (kind == TT_ATTN_KIND_DECODE_APPEND) {
    // the decode scratch; on the grouped-query tensor-core path also the rotated q and the new lengths
    const size_t base = tt_attn_workspace_bytes(TT_ATTN_KIND_DECODE, dtype, B, Hq, Hkv, Lq, Skv, D);
    return base + (Skv > 0 ? append_bytes(dtype, B, Hq, Hkv, D) : 0);
  }
  if (kind == TT_ATTN_KIND_DECODE) {
    if (Skv <= 0) return 0;
    int nsplit, chunk;
    decode_plan_for(dtype, D, B, Hq, Hkv, Skv, &nsplit, &chunk);
    return decode_scratch_bytes(dtype, D, B, Hq, Hkv, nsplit);
  }
  return 0;
}

int tt_attn_fwd(const tt_attn_fwd_params* p) {
  if (!p) return TT_ATTN_ERR_NULL;
  const bool v2 = p->struct_size == sizeof(tt_attn_fwd_params);
  if (!v2 && p->struct_size != offsetof(tt_attn_fwd_params, mask)) return TT_ATTN_ERR_STRUCT;
  if (int rc = check_common(p->dtype, p->B, p->Hq, p->Hkv, p->Lq, p->Skv, p->D)) return rc;
  if (!p->q || !p->k || !p->v || !p->o) return TT_ATTN_ERR_NULL;
  const size_t es = elem_size(p->dtype);
  FwdArgs a{};
  a.q = p->q, a.k = p->k, a.v = p->v, a.o = p->o, a.lse = p->lse;
  a.qs = dense_or(p->q_strides, p->Hq, p->Lq, p->D);
  a.ks = dense_or(p->k_strides, p->Hkv, p->Skv, p->D);
  a.vs = dense_or(p->v_strides, p->Hkv, p->Skv, p->D);
  a.os = dense_or(p->o_strides, p->Hq, p->Lq, p->D);
  if (!aligned16(p->q) || !aligned16(p->k) || !aligned16(p->v) || !aligned16(p->o) || !strides_ok(a.qs, es) ||
      !strides_ok(a.ks, es) || !strides_ok(a.vs, es) || !strides_ok(a.os, es))
    return TT_ATTN_ERR_ALIGN;
  a.B = p->B, a.Hq = p->Hq, a.Hkv = p->Hkv, a.Lq = p->Lq, a.Skv = p->Skv;
  if (p->is_causal < 0 || p->is_causal > TT_ATTN_CAUSAL_BOTTOM_RIGHT) return TT_ATTN_ERR_SHAPE;
  a.causal = p->is_causal;
  a.scale = p->scale;
  a.kv_lens = p->kv_lens;
  a.status = p->status;
  if (v2)
    if (int rc = take_mask(p->mask, p->mask_kind, p->mask_strides, &a.mask)) return rc;
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  Workspace ws;
  const size_t room = p->workspace ? p->workspace_bytes : SIZE_MAX;
  const bool lens = p->dtype != TT_ATTN_F32 && mask_lens_fit(a.mask, a.causal, p->B, room, 0);
  const size_t need = p->dtype == TT_ATTN_F32 ? 0 : (lens ? round256(scratch_words(p->B) * sizeof(int)) : 256);
  if (int rc = ws.acquire(need, p->workspace, p->workspace_bytes, p->alloc, p->device)) return rc;
  a.sched = static_cast<int*>(ws.ptr);
  a.mask_lens = lens ? a.sched + 1 : nullptr;
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  cudaError_t e = p->dtype == TT_ATTN_F32 ? launch_fwd_f32(p->D, a, p->device, stream)
                                          : launch_fwd_tc(p->dtype, p->D, a, p->device, stream);
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

int tt_attn_bwd(const tt_attn_bwd_params* p) { return bwd_call(p, kPlanned, nullptr); }

int tt_attn_bwd_selftest(const tt_attn_bwd_params* p, int32_t path, int32_t* planned) {
  if (path < -1 || path > 1) return TT_ATTN_ERR_SHAPE;
  if (path < 0 && !planned) return TT_ATTN_ERR_NULL;
  return bwd_call(p, path < 0 ? kAsked : (path == 0 ? kRecompute : kStore), planned);
}

int tt_attn_decode(const tt_attn_decode_params* p) {
  if (!p) return TT_ATTN_ERR_NULL;
  if (p->struct_size != sizeof(tt_attn_decode_params)) return TT_ATTN_ERR_STRUCT;
  if (int rc = check_common(p->dtype, p->B, p->Hq, p->Hkv, 1, p->capacity, p->D)) return rc;
  if (!p->q || !p->k || !p->v || !p->o) return TT_ATTN_ERR_NULL;
  const size_t es = elem_size(p->dtype);
  DecodeArgs a{};
  a.q = p->q, a.k = p->k, a.v = p->v, a.o = p->o, a.lse = p->lse;
  a.qs = dense_or(p->q_strides, p->Hq, 1, p->D);
  a.ks = dense_or(p->k_strides, p->Hkv, p->capacity, p->D);
  a.vs = dense_or(p->v_strides, p->Hkv, p->capacity, p->D);
  a.os = dense_or(p->o_strides, p->Hq, 1, p->D);
  if (!aligned16(p->q) || !aligned16(p->k) || !aligned16(p->v) || !aligned16(p->o) || !strides_ok(a.qs, es) ||
      !strides_ok(a.ks, es) || !strides_ok(a.vs, es) || !strides_ok(a.os, es))
    return TT_ATTN_ERR_ALIGN;
  a.B = p->B, a.Hq = p->Hq, a.Hkv = p->Hkv, a.capacity = p->capacity;
  a.scale = p->scale;
  a.kv_lens = p->kv_lens;
  const size_t need = decode_plan_within(p->dtype, p->D, p->B, p->Hq, p->Hkv, p->capacity,
                                         p->workspace ? p->workspace_bytes : SIZE_MAX, &a.nsplit, &a.chunk);
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  Workspace ws;
  if (int rc = ws.acquire(need, p->workspace, p->workspace_bytes, p->alloc, p->device)) return rc;
  a.partial = static_cast<float*>(ws.ptr);
  // the tensor-core path's work counter sits in the last 256 bytes (unused by the scan kernel)
  a.sched = need >= 256 ? reinterpret_cast<int*>(static_cast<char*>(ws.ptr) + need - 256) : nullptr;
  a.status = p->status;
  cudaError_t e = launch_decode(p->dtype, p->D, a, static_cast<cudaStream_t>(p->stream));
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

int tt_attn_decode_append(const tt_attn_decode_append_params* p) {
  if (!p) return TT_ATTN_ERR_NULL;
  if (p->struct_size != sizeof(tt_attn_decode_append_params)) return TT_ATTN_ERR_STRUCT;
  if (int rc = check_common(p->dtype, p->B, p->Hq, p->Hkv, 1, p->capacity, p->D)) return rc;
  if (!p->q || !p->k_new || !p->v_new || !p->k_cache || !p->v_cache || !p->o || !p->kv_lens) return TT_ATTN_ERR_NULL;
  if ((p->rope_cos == nullptr) != (p->rope_sin == nullptr)) return TT_ATTN_ERR_NULL;
  if (p->rope_cos && p->rope_positions <= 0) return TT_ATTN_ERR_SHAPE;
  if (p->new_lens && p->new_lens == p->kv_lens) return TT_ATTN_ERR_SHAPE;
  const size_t es = elem_size(p->dtype);
  DecodeArgs a{};
  a.q = p->q, a.k = p->k_cache, a.v = p->v_cache, a.o = p->o, a.lse = p->lse;
  a.k_new = p->k_new, a.v_new = p->v_new;
  a.qs = dense_or(p->q_strides, p->Hq, 1, p->D);
  a.ks = dense_or(p->k_strides, p->Hkv, p->capacity, p->D);
  a.vs = dense_or(p->v_strides, p->Hkv, p->capacity, p->D);
  a.os = dense_or(p->o_strides, p->Hq, 1, p->D);
  const Str3 kn = dense_or(p->k_new_strides, p->Hkv, 1, p->D), vn = dense_or(p->v_new_strides, p->Hkv, 1, p->D);
  a.kn_b = kn.b, a.kn_h = kn.h, a.vn_b = vn.b, a.vn_h = vn.h;
  const void* ptrs[] = {p->q, p->k_new, p->v_new, p->k_cache, p->v_cache, p->o};
  for (const void* q : ptrs)
    if (!aligned16(q)) return TT_ATTN_ERR_ALIGN;
  const Str3* sts[] = {&a.qs, &a.ks, &a.vs, &a.os, &kn, &vn};
  for (const Str3* s : sts)
    if (!strides_ok(*s, es)) return TT_ATTN_ERR_ALIGN;
  a.B = p->B, a.Hq = p->Hq, a.Hkv = p->Hkv, a.capacity = p->capacity;
  a.scale = p->scale;
  a.kv_lens = p->kv_lens;
  a.new_lens = p->new_lens;
  a.rope_cos = p->rope_cos, a.rope_sin = p->rope_sin;
  a.rope_positions = p->rope_positions, a.rope_interleaved = p->rope_interleaved;
  a.status = p->status;
  const size_t more = append_bytes(p->dtype, p->B, p->Hq, p->Hkv, p->D);
  const size_t room = !p->workspace ? SIZE_MAX : (p->workspace_bytes > more ? p->workspace_bytes - more : 0);
  const size_t base = decode_plan_within(p->dtype, p->D, p->B, p->Hq, p->Hkv, p->capacity, room, &a.nsplit, &a.chunk);
  const size_t need = base + more;
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  Workspace ws;
  if (int rc = ws.acquire(need, p->workspace, p->workspace_bytes, p->alloc, p->device)) return rc;
  a.partial = static_cast<float*>(ws.ptr);
  a.sched = base >= 256 ? reinterpret_cast<int*>(static_cast<char*>(ws.ptr) + base - 256) : nullptr;
  if (need > base) {
    a.q_rot = static_cast<char*>(ws.ptr) + base;
    a.lens_scratch = reinterpret_cast<int32_t*>(static_cast<char*>(ws.ptr) + need - round256(static_cast<size_t>(p->B) * 4));
  }
  cudaError_t e = launch_decode_append(p->dtype, p->D, a, static_cast<cudaStream_t>(p->stream));
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

int tt_attn_decode_static(const tt_attn_decode_params* p) {
  if (!p) return TT_ATTN_ERR_NULL;
  if (p->struct_size != sizeof(tt_attn_decode_params)) return TT_ATTN_ERR_STRUCT;
  if (int rc = check_common(p->dtype, p->B, p->Hq, p->Hkv, 1, p->capacity, p->D)) return rc;
  if (!p->q || !p->k || !p->v || !p->o) return TT_ATTN_ERR_NULL;
  const size_t es = elem_size(p->dtype);
  DecodeArgs a{};
  a.q = p->q, a.k = p->k, a.v = p->v, a.o = p->o, a.lse = p->lse;
  a.qs = dense_or(p->q_strides, p->Hq, 1, p->D);
  a.ks = dense_or(p->k_strides, p->Hkv, p->capacity, p->D);
  a.vs = dense_or(p->v_strides, p->Hkv, p->capacity, p->D);
  a.os = dense_or(p->o_strides, p->Hq, 1, p->D);
  if (!aligned16(p->q) || !aligned16(p->k) || !aligned16(p->v) || !aligned16(p->o) || !strides_ok(a.qs, es) ||
      !strides_ok(a.ks, es) || !strides_ok(a.vs, es) || !strides_ok(a.os, es))
    return TT_ATTN_ERR_ALIGN;
  a.B = p->B, a.Hq = p->Hq, a.Hkv = p->Hkv, a.capacity = p->capacity;
  a.scale = p->scale;
  a.kv_lens = p->kv_lens;
  a.status = p->status;
  const size_t need = decode_plan_within(p->dtype, p->D, p->B, p->Hq, p->Hkv, p->capacity, TT_ATTN_STATIC_SCRATCH_BYTES,
                                         &a.nsplit, &a.chunk);
  if (need > TT_ATTN_STATIC_SCRATCH_BYTES) return TT_ATTN_ERR_TOO_LARGE;
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  bool too_large = false;
  cudaError_t e =
      launch_decode_static(p->dtype, p->D, a, need, p->device, static_cast<cudaStream_t>(p->stream), &too_large);
  if (too_large) return TT_ATTN_ERR_TOO_LARGE;
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

int tt_attn_selftest_wait_expiry(int device, void* stream, uint64_t limit_ns, int32_t* status,
                                 unsigned long long* waited_ns) {
  if (!status) return TT_ATTN_ERR_NULL;
  if (limit_ns == 0 || limit_ns > 2000000000ull) return TT_ATTN_ERR_SHAPE;  // the kernels' own limit is 2 s
  DeviceGuard guard(device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  cudaError_t e = launch_wait_expiry(status, limit_ns, waited_ns, static_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

int tt_fused_add_rms_norm(const tt_fused_add_rms_norm_params* p) {
  if (!p) return TT_ATTN_ERR_NULL;
  if (p->struct_size != sizeof(tt_fused_add_rms_norm_params)) return TT_ATTN_ERR_STRUCT;
  if (p->dtype < TT_ATTN_F32 || p->dtype > TT_ATTN_BF16) return TT_ATTN_ERR_DTYPE;
  if (p->rows < 0 || p->dim <= 0 || p->rows > 0x7fffffff) return TT_ATTN_ERR_SHAPE;
  if (p->rows == 0) return TT_ATTN_OK;  // an empty tensor has no storage to point to
  if (!p->input || !p->residual || !p->weight) return TT_ATTN_ERR_NULL;
  const size_t es = elem_size(p->dtype);
  if (reinterpret_cast<uintptr_t>(p->input) % es || reinterpret_cast<uintptr_t>(p->residual) % es ||
      reinterpret_cast<uintptr_t>(p->weight) % es)
    return TT_ATTN_ERR_ALIGN;
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  cudaError_t e = launch_fused_add_rms_norm(p->dtype, p->input, p->residual, p->weight, p->rows, p->dim, p->eps,
                                            static_cast<cudaStream_t>(p->stream));
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

int tt_silu_mul(const tt_silu_mul_params* p) {
  if (!p) return TT_ATTN_ERR_NULL;
  if (p->struct_size != sizeof(tt_silu_mul_params)) return TT_ATTN_ERR_STRUCT;
  if (p->dtype < TT_ATTN_F32 || p->dtype > TT_ATTN_BF16) return TT_ATTN_ERR_DTYPE;
  if (p->rows < 0 || p->d <= 0) return TT_ATTN_ERR_SHAPE;
  if (p->rows == 0) return TT_ATTN_OK;
  if (!p->x || !p->out) return TT_ATTN_ERR_NULL;
  const size_t es = elem_size(p->dtype);
  if (reinterpret_cast<uintptr_t>(p->x) % es || reinterpret_cast<uintptr_t>(p->out) % es) return TT_ATTN_ERR_ALIGN;
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  cudaError_t e = launch_silu_mul(p->dtype, p->out, p->x, p->rows, p->d, static_cast<cudaStream_t>(p->stream));
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

int tt_linear(const tt_linear_params* p) {
  LinearCall c;
  bool sums_only;
  if (int rc = linear_call(p, &c, &sums_only)) return rc;
  if (c.M == 0) return TT_ATTN_OK;
  void* x_sum = p->struct_size == sizeof(tt_linear_params) ? p->x_sum : nullptr;
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  bool persistent = false;
  cudaError_t e = sums_only ? cudaSuccess : launch_linear_tc(c, &persistent);
  if (e == cudaSuccess && x_sum) e = launch_column_sums(c.dtype, c.x, x_sum, c.K, c.M, c.ldx, persistent, c.stream);
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

int tt_linear_selftest(const tt_linear_params* p, int32_t shape, int32_t* planned) {
  LinearCall c;
  bool sums_only;
  if (int rc = linear_call(p, &c, &sums_only)) return rc;
  const bool pair = shape < 0;
  const int bn = shape < -1024 ? 0 : (pair ? -shape : shape);
  if (sums_only || c.M == 0 || (shape != 0 && !linear_tile_fits(c, pair, bn))) return TT_ATTN_ERR_SHAPE;
  if (shape == 0 && !planned) return TT_ATTN_ERR_NULL;
  DeviceGuard guard(p->device);
  if (!guard.ok) return TT_ATTN_ERR_NO_DEVICE;
  if (planned) *planned = linear_shape(c);
  cudaError_t e = shape != 0 ? launch_linear_tile(c, pair, bn) : cudaSuccess;
  return e == cudaSuccess ? TT_ATTN_OK : launch_failed(e);
}

}  // extern "C"
