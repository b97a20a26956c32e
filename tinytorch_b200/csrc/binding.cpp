// Python binding of libtt_attn.so for torch tensors: argument checks, output and scratch allocation, the C ABI calls
// and the autograd nodes, in one extension module (tinytorch_b200._native) instead of in Python.
//
// Why native: a call on small tensors is bound by the host, not by the GPU.  Filling the parameter structs through
// ctypes, calling back into Python for scratch memory and going through Python autograd functions took 16-50 us per
// operator (150-220 us for a forward and backward pass) while the kernels of such a call run for 2-20 us.
//
// The Python layer (op.py, function.py, fused.py) keeps the public signatures and hands its arguments on; its autograd
// functions take the calls that need more than reverse mode (needs_python_function).  The GIL is
// released around every launch.  Scratch memory comes from torch's caching allocator on the current stream, the
// stand-in for the reference's getCUDACachedAllocator(device) (src/Tensor/Allocator.cpp:117-139).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <cmath>
#include <cstdarg>
#include <optional>

#include "../../include/tt_fused.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------------------------- library --
struct Api {
  int (*fwd)(const tt_attn_fwd_params*);
  int (*bwd)(const tt_attn_bwd_params*);
  int (*decode)(const tt_attn_decode_params*);
  int (*decode_append)(const tt_attn_decode_append_params*);
  int (*add_rms_norm)(const tt_fused_add_rms_norm_params*);
  int (*silu_mul)(const tt_silu_mul_params*);
  int (*linear)(const tt_linear_params*);
  const char* (*strerror)(int);
  const char* (*last_cuda_error)();
} api;
PyObject* attn_error = nullptr;  // _capi.AttnError

// Called with or without the GIL (the backward nodes run in the engine's threads).
[[noreturn]] void raise(PyObject* type, const char* fmt, ...) {
  const PyGILState_STATE st = PyGILState_Ensure();
  python_error err;
  va_list ap;
  va_start(ap, fmt);
  PyErr_FormatV(type, fmt, ap);
  va_end(ap);
  err.persist();
  PyGILState_Release(st);
  throw err;
}

// As above.
void check(int rc) {
  if (rc == TT_ATTN_OK) return;
  std::string text = api.strerror(rc);
  if (rc == TT_ATTN_ERR_LAUNCH) text += std::string(" [") + api.last_cuda_error() + "]";
  const PyGILState_STATE st = PyGILState_Ensure();
  python_error err;
  if (PyObject* args = Py_BuildValue("(is)", rc, text.c_str())) {
    if (PyObject* exc = PyObject_CallObject(attn_error, args)) {
      PyErr_SetObject(attn_error, exc);
      Py_DECREF(exc);
    }
    Py_DECREF(args);
  }
  err.persist();
  PyGILState_Release(st);
  throw err;
}

struct NoGil {
  PyThreadState* st = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(st); }
};

// ------------------------------------------------------------------------------------------------- scratch --
void* hook_alloc(void*, size_t bytes, int device) {
  try {
    return c10::cuda::CUDACachingAllocator::raw_alloc_with_stream(bytes, c10::cuda::getCurrentCUDAStream(device));
  } catch (...) {  // (out of memory: the C ABI reports it as a status)
    return nullptr;
  }
}
void hook_free(void*, void* ptr, int) { c10::cuda::CUDACachingAllocator::raw_delete(ptr); }
const tt_attn_alloc_hook hook = {hook_alloc, hook_free, nullptr};

// ------------------------------------------------------------------------------------------------- tensors --
int dtype_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return TT_ATTN_F32;
    case at::kHalf: return TT_ATTN_F16;
    case at::kBFloat16: return TT_ATTN_BF16;
    default: return -1;
  }
}

const Tensor& tensor_of(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) raise(PyExc_TypeError, "%s must be a tensor", name);
  return THPVariable_Unpack(o);
}
Tensor optional_of(PyObject* o, const char* name) { return o == Py_None ? Tensor() : tensor_of(o, name); }

void check_attn_tensor(const Tensor& t, const char* name) {
  if (!t.is_cuda()) raise(PyExc_ValueError, "%s must be a CUDA tensor (this op has no CPU path)", name);
  if (t.dim() != 4) raise(PyExc_ValueError, "%s must be [B, H, S, D]", name);
  if (t.stride(3) != 1) raise(PyExc_ValueError, "%s: innermost dimension must be contiguous", name);
  if (dtype_of(t.scalar_type()) < 0) raise(PyExc_ValueError, "%s: dtype %s not supported", name, c10::toString(t.scalar_type()));
}

// The C ABI sees the sizes of q (and the key heads and rows of k) only; every other operand has to have at least what a
// kernel will take from it, in q's dtype and on its device.
void check_operand(const Tensor& t, const char* name, const Tensor& q, int64_t B, int64_t H, int64_t S) {
  if (t.scalar_type() != q.scalar_type() || t.device() != q.device())
    raise(PyExc_ValueError, "%s must have the dtype and device of q", name);
  if (t.size(0) < B || t.size(1) < H || t.size(2) < S || t.size(3) < q.size(3))
    raise(PyExc_ValueError, "%s is smaller than [%lld, %lld, %lld, %lld], which q and the keys ask for", name, (long long)B,
          (long long)H, (long long)S, (long long)q.size(3));
}
// `grads`: gradients of the same shapes are to be written, every element of them
void check_kv(const Tensor& q, const Tensor& k, const Tensor& v, bool grads) {
  check_operand(k, "k", q, q.size(0), 1, 0);
  check_operand(v, "v", q, q.size(0), k.size(1), k.size(2));
  if (grads && (k.size(0) != q.size(0) || k.size(3) != q.size(3) || v.sizes() != k.sizes()))
    raise(PyExc_ValueError, "gradients need k and v of one shape, with the batch and head dimension of q");
}

tt_attn_strides strides_of(const Tensor& t) { return {t.stride(0), t.stride(1), t.stride(2)}; }

Tensor empty(at::IntArrayRef sizes, at::ScalarType dt, const at::Device& dev) {
  return Tensor(at::detail::empty_cuda(sizes, dt, dev, c10::nullopt));
}

// The reference's default scale 1/sqrt(D) (src/Function/FuncNNLayer.h:235) where the caller gave none.
float scale_or_default(const std::optional<double>& scale, int64_t D) {
  return static_cast<float>(scale ? *scale : 1.0 / std::sqrt(static_cast<double>(D)));
}

template <typename P>
void set_common(P* p, const Tensor& ref) {
  p->struct_size = sizeof(P);
  p->device = ref.get_device();
  p->stream = c10::cuda::getCurrentCUDAStream(ref.get_device()).stream();
}

// attnMask of the reference (src/Function/FuncNNLayer.h:249-256): Bool -> keys that participate, otherwise added to
// the scaled scores; any shape that broadcasts against [B, Hq, L, S] by trailing-dimension alignment.
struct Mask {
  Tensor t;
  int kind = TT_ATTN_MASK_NONE;
  int64_t strides[3] = {0, 0, 0};
};

Mask mask_of(const Tensor& mask, const Tensor& q, int64_t S) {
  Mask r;
  if (!mask.defined()) return r;
  Tensor m = mask;
  if (m.requires_grad()) m = m.detach();
  if (!m.is_cuda() || m.device() != q.device()) raise(PyExc_ValueError, "attnMask must be on the device of q");
  if (m.dim() > 4) raise(PyExc_ValueError, "attnMask has more than 4 dimensions");
  const int64_t want[4] = {q.size(0), q.size(1), q.size(2), S};
  if (m.dim() < 4) {
    at::DimVector shape(4 - m.dim(), 1);
    shape.append(m.sizes().begin(), m.sizes().end());
    m = m.reshape(shape);
  }
  for (int i = 0; i < 4; ++i)
    if (m.size(i) != want[i] && m.size(i) != 1)
      raise(PyExc_ValueError, "attnMask shape does not broadcast against (%lld, %lld, %lld, %lld)", (long long)want[0],
            (long long)want[1], (long long)want[2], (long long)want[3]);
  if (m.scalar_type() == at::kBool) {
    r.kind = TT_ATTN_MASK_BOOL;
  } else if (m.scalar_type() == q.scalar_type() && q.scalar_type() != at::kFloat) {
    r.kind = TT_ATTN_MASK_ADD;
  } else {
    if (m.scalar_type() != at::kFloat) m = m.to(at::kFloat);
    r.kind = TT_ATTN_MASK_ADD_F32;
  }
  // keys must be contiguous in memory; a mask broadcast over keys is expanded
  if (m.size(3) != S || m.stride(3) != 1) m = m.expand({m.size(0), m.size(1), m.size(2), S}).contiguous();
  for (int i = 0; i < 3; ++i) r.strides[i] = m.size(i) == 1 ? 0 : m.stride(i);
  r.t = std::move(m);
  return r;
}

template <typename P>
void set_mask(P* p, const Mask& m) {
  p->mask = m.t.defined() ? m.t.data_ptr() : nullptr, p->mask_kind = m.kind;
  for (int i = 0; i < 3; ++i) p->mask_strides[i] = m.strides[i];
}

// Integers that a kernel reads or writes: lengths [B], a status word.  Pinned host memory is reachable as well.
void check_ints(const Tensor& t, const char* name, int64_t n, const Tensor& q) {
  if (!t.defined()) return;
  if (t.scalar_type() != at::kInt || !t.is_contiguous() || t.numel() < n || !(t.is_cuda() ? t.device() == q.device() : t.is_pinned()))
    raise(PyExc_ValueError, "%s must be a contiguous int32 tensor of %lld elements or more on the device of q", name, (long long)n);
}
void check_ints(const Tensor& kv_lens, const Tensor& status, const Tensor& q) {
  check_ints(kv_lens, "kvLens", q.size(0), q);
  check_ints(status, "status", 1, q);
}
int32_t* ints_ptr(const Tensor& t) { return t.defined() ? static_cast<int32_t*>(t.data_ptr()) : nullptr; }

// --------------------------------------------------------------------------------------------- attention --
// The output's gradient; zeros where what follows gave none, so that the inputs get gradients of zeros and not none.
Tensor gradient_of(const torch::autograd::Node& node, const variable_list& grads) {
  return grads[0].defined() ? grads[0] : node.input_metadata(0).zeros_like();
}

Tensor same_memory(const Tensor& t) { return t.defined() ? t.variable_data() : Tensor(); }

struct FwdResult {
  Tensor o, lse;
};

FwdResult attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, int mode, float scale, const Tensor& kv_lens,
                   bool need_lse, const Tensor& status, const Mask& mask) {
  check_ints(kv_lens, status, q);
  FwdResult r;
  const int64_t B = q.size(0), Hq = q.size(1), L = q.size(2), D = q.size(3);
  tt_attn_fwd_params p{};
  set_common(&p, q);
  r.o = empty({B, Hq, L, D}, q.scalar_type(), q.device());
  if (need_lse) r.lse = empty({B, Hq, L}, at::kFloat, q.device());
  p.dtype = dtype_of(q.scalar_type());
  p.B = B, p.Hq = Hq, p.Hkv = k.size(1), p.Lq = L, p.Skv = k.size(2), p.D = D;
  p.q = q.data_ptr(), p.k = k.data_ptr(), p.v = v.data_ptr(), p.o = r.o.data_ptr();
  p.lse = need_lse ? static_cast<float*>(r.lse.data_ptr()) : nullptr;
  p.q_strides = strides_of(q), p.k_strides = strides_of(k), p.v_strides = strides_of(v), p.o_strides = strides_of(r.o);
  p.is_causal = mode, p.scale = scale, p.kv_lens = ints_ptr(kv_lens);
  p.alloc = &hook;
  p.status = ints_ptr(status);
  set_mask(&p, mask);
  check(api.fwd(&p));
  return r;
}

struct BwdResult {
  Tensor g[3];
};

BwdResult attn_bwd(const Tensor& dO, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                   int mode, float scale, const Tensor& kv_lens, const bool (&needs)[3], const Mask& mask) {
  check_ints(kv_lens, Tensor(), q);
  BwdResult r;
  const Tensor* like[3] = {&q, &k, &v};
  for (int i = 0; i < 3; ++i)
    if (needs[i]) r.g[i] = empty(like[i]->sizes(), like[i]->scalar_type(), like[i]->device());
  tt_attn_bwd_params p{};
  set_common(&p, q);
  p.dtype = dtype_of(q.scalar_type());
  p.B = q.size(0), p.Hq = q.size(1), p.Hkv = k.size(1), p.Lq = q.size(2), p.Skv = k.size(2), p.D = q.size(3);
  p.q = q.data_ptr(), p.k = k.data_ptr(), p.v = v.data_ptr(), p.o = o.data_ptr(), p.d_o = dO.data_ptr();
  p.lse = static_cast<const float*>(lse.data_ptr());
  p.q_strides = strides_of(q), p.k_strides = strides_of(k), p.v_strides = strides_of(v);
  p.o_strides = strides_of(o), p.do_strides = strides_of(dO);
  void** out[3] = {&p.dq, &p.dk, &p.dv};
  tt_attn_strides* st[3] = {&p.dq_strides, &p.dk_strides, &p.dv_strides};
  for (int i = 0; i < 3; ++i)
    if (needs[i]) *out[i] = r.g[i].data_ptr(), *st[i] = strides_of(r.g[i]);
  p.is_causal = mode, p.scale = scale, p.kv_lens = ints_ptr(kv_lens);
  p.alloc = &hook;
  set_mask(&p, mask);
  check(api.bwd(&p));
  return r;
}

void check_bwd(const Tensor& dO, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse) {
  check_kv(q, k, v, true);
  check_operand(dO, "dO", q, q.size(0), q.size(1), q.size(2));
  check_operand(o, "o", q, q.size(0), q.size(1), q.size(2));
  if (lse.scalar_type() != at::kFloat || lse.device() != q.device() || !lse.is_contiguous() ||
      lse.numel() < q.size(0) * q.size(1) * q.size(2))
    raise(PyExc_ValueError, "lse must be a contiguous float32 tensor [B, Hq, L] on the device of q");
}

// What FuncSDPAttention::backward (src/Function/FuncNNLayer.h:267) leaves unimplemented: the forward saves (O, LSE)
// and hands dQ, dK, dV to autograd.  What it saves goes through saved-tensor hooks, but for the mask and the lengths, which
// receive no gradient.
struct AttentionBackward : public torch::autograd::Node {
  SavedVariable q, k, v, o, lse;
  Tensor kv_lens;  // as the mask: over the caller's memory, not the caller's tensor, which may be pointed elsewhere meanwhile
  Mask mask;
  int mode;
  float scale;
  std::string name() const override { return "FuncSDPAttentionBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    q.reset_data(), k.reset_data(), v.reset_data(), o.reset_data(), lse.reset_data();
    kv_lens.reset(), mask = Mask();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(3);
    Tensor dO = gradient_of(*this, grads);
    std::lock_guard<std::mutex> lock(mutex_);
    at::NoGradGuard no_grad;
    const Tensor qt = q.unpack(), kt = k.unpack(), vt = v.unpack(), ot = o.unpack(shared_from_this()), lt = lse.unpack();
    if (dO.stride(3) != 1) dO = dO.contiguous();
    check_bwd(dO, qt, kt, vt, ot, lt);
    const bool needs[3] = {task_should_compute_output(0), task_should_compute_output(1), task_should_compute_output(2)};
    BwdResult r = attn_bwd(dO, qt, kt, vt, ot, lt, mode, scale, kv_lens, needs, mask);
    for (int i = 0; i < 3; ++i) out[i] = std::move(r.g[i]);
    return out;
  }
};

void check_qkv(const Tensor& q, const Tensor& k, const Tensor& v, bool grads) {
  check_attn_tensor(q, "q");
  check_attn_tensor(k, "k");
  check_attn_tensor(v, "v");
  if (!(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type() && q.device() == k.device() &&
        k.device() == v.device()))
    raise(PyExc_ValueError, "q, k, v must share dtype and device");
  check_kv(q, k, v, grads);
}
bool wants_grad(const Tensor& q, const Tensor& k, const Tensor& v) {
  return at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
}

// ------------------------------------------------------------------------------------------------- linear --
// Row stride of a matrix with contiguous columns (a single row's stride may be anything).
int64_t row_stride(const Tensor& t) { return t.size(0) > 1 ? t.stride(0) : t.size(1); }

// y[M, N] (dense memory) = x[M, K] w[N, K]^T + bias; x_t / w_t: the operand is given as [K, M] / [K, N]; without y only x_sum
void linear_raw(const Tensor& x, bool x_t, const Tensor& w, bool w_t, const Tensor& bias, const Tensor& y, const Tensor& status,
                const Tensor& x_sum) {
  tt_linear_params p{};
  set_common(&p, x);
  p.dtype = dtype_of(x.scalar_type());
  p.M = x.size(x_t ? 1 : 0), p.K = x.size(x_t ? 0 : 1), p.N = w.size(w_t ? 1 : 0);
  p.x = x.data_ptr(), p.w = y.defined() ? w.data_ptr() : nullptr, p.y = y.defined() ? y.data_ptr() : nullptr;
  p.bias = bias.defined() ? bias.data_ptr() : nullptr;
  p.ldx = row_stride(x), p.ldw = row_stride(w), p.ldy = p.N;
  p.status = ints_ptr(status);
  p.x_t = x_t, p.w_t = w_t;
  p.x_sum = x_sum.defined() ? x_sum.data_ptr() : nullptr;
  check(api.linear(&p));
}

Tensor rows_of(const Tensor& t) {  // [.., C] as [rows, C] with contiguous columns
  Tensor r = t.dim() == 2 ? t : t.reshape({-1, t.size(-1)});
  if (r.stride(1) != 1 || (r.size(0) > 1 && r.stride(0) < r.size(1))) r = r.clone(at::MemoryFormat::Contiguous);
  return r;
}

// ... that start on 16 bytes, as the kernels read them: a gradient may be a part of a larger one (the split of a projection,
// a concatenation), at any offset and row stride, and is copied then
Tensor aligned_rows_of(const Tensor& t) {
  Tensor r = rows_of(t);
  const bool aligned = reinterpret_cast<uintptr_t>(r.data_ptr()) % 16 == 0 && (r.size(0) <= 1 || r.stride(0) % 8 == 0);
  return aligned ? r : r.clone(at::MemoryFormat::Contiguous);
}

// function::FuncLinear::backward (src/Function/FuncNNLayer.h:20-34)
struct LinearGrads {
  Tensor g[3];
};
LinearGrads linear_bwd(const Tensor& dy, const Tensor& x2, const Tensor& w, at::IntArrayRef dx_shape, const bool (&needs)[3]) {
  LinearGrads r;
  const Tensor g2 = aligned_rows_of(dy);
  if (g2.size(0) == 0) {  // sums of nothing
    const at::IntArrayRef shapes[3] = {dx_shape, w.sizes(), w.sizes().slice(0, 1)};
    for (int i = 0; i < 3; ++i)
      if (needs[i]) r.g[i] = at::zeros(shapes[i], g2.options());
    return r;
  }
  // the products contract over the slow dimension of W, and of dY and X: read as they are stored
  if (needs[0]) {  // dX[M,K] = dY[M,N] W[N,K]
    r.g[0] = empty(dx_shape, g2.scalar_type(), g2.device());
    linear_raw(g2, false, w, true, Tensor(), r.g[0], Tensor(), Tensor());
  }
  if (needs[2]) r.g[2] = empty({g2.size(1)}, g2.scalar_type(), g2.device());
  if (needs[1]) {  // dW[N,K] = dY[M,N]^T X[M,K], with db[N] = sum of dY over its rows
    r.g[1] = empty({g2.size(1), x2.size(1)}, g2.scalar_type(), g2.device());
    linear_raw(g2, true, x2, true, Tensor(), r.g[1], Tensor(), r.g[2]);
  } else if (needs[2]) {
    linear_raw(g2, true, x2, true, Tensor(), Tensor(), Tensor(), r.g[2]);  // (the sums alone)
  }
  return r;
}

struct LinearBackward : public torch::autograd::Node {
  SavedVariable x2, w;
  at::DimVector in_shape;
  bool has_bias;
  std::string name() const override { return "FuncLinearBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    x2.reset_data(), w.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(3);
    const Tensor dY = gradient_of(*this, grads);
    std::lock_guard<std::mutex> lock(mutex_);
    bool needs[3] = {task_should_compute_output(0), task_should_compute_output(1), has_bias && task_should_compute_output(2)};
    if (needs[2] && at::GradMode::is_enabled() && dY.requires_grad()) {
      // create_graph: db is linear in dY and can be differentiated again (dX and dW cannot)
      out[2] = dY.reshape({-1, dY.size(-1)}).to(at::kFloat).sum(0).to(dY.scalar_type());
      needs[2] = false;
    }
    at::NoGradGuard no_grad;
    LinearGrads r = linear_bwd(dY, x2.unpack(), w.unpack(), in_shape, needs);
    for (int i = 0; i < 3; ++i)
      if (needs[i]) out[i] = std::move(r.g[i]);
    return out;
  }
};

// [N] values in the dtype and on the device of x, contiguous
Tensor bias_of(const Tensor& bias, const Tensor& x, int64_t N) {
  if (!bias.defined()) return bias;
  if (bias.dim() != 1 || bias.size(0) != N || bias.scalar_type() != x.scalar_type())
    raise(PyExc_AssertionError, "bias must be [N] (OpLinalg.cpp:261-263)");
  if (bias.device() != x.device()) raise(PyExc_ValueError, "bias must be on the device of input");
  return bias.contiguous();
}

Tensor linear_autograd(const Tensor& x, const Tensor& w, const Tensor& bias) {
  if (!x.is_cuda() || (x.scalar_type() != at::kHalf && x.scalar_type() != at::kBFloat16))
    raise(PyExc_ValueError, "linear needs CUDA float16 / bfloat16 tensors (float32 stays on the library gemm; no CPU path)");
  if (w.dim() != 2 || w.scalar_type() != x.scalar_type() || w.device() != x.device())
    raise(PyExc_ValueError, "weight must be [N, K] with the dtype and device of input");
  if (x.size(-1) != w.size(1)) raise(PyExc_AssertionError, "matmul error: shape not aligned (OpLinalg.cpp:251-254)");
  const Tensor b = bias_of(bias, x, w.size(0));
  NoGil nogil;
  const bool grad = at::GradMode::is_enabled() &&
                    (x.requires_grad() || w.requires_grad() || (bias.defined() && bias.requires_grad()));
  Tensor x2, wc, y;
  {
    at::NoGradGuard no_grad;
    x2 = rows_of(x);
    wc = rows_of(w);
    at::DimVector shape(x.sizes().begin(), x.sizes().end());
    shape.back() = w.size(0);
    y = empty(shape, x.scalar_type(), x.device());
    linear_raw(x2, false, wc, false, b, y, Tensor(), Tensor());
  }
  if (grad) {
    auto node = std::shared_ptr<LinearBackward>(new LinearBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, w, bias));
    node->x2 = SavedVariable(x2, false);
    node->w = SavedVariable(wc, false);
    node->in_shape.assign(x.sizes().begin(), x.sizes().end());
    node->has_bias = bias.defined();
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ------------------------------------------------------------------------------------------ python methods --
// The nodes here know reverse mode only.  A trace has to record the operator, forward-mode derivatives and functorch's
// transforms have to reach torch, which refuses them: the Python autograd functions (function.py, fused.py) see to that.
bool needs_python_function(std::initializer_list<const Tensor*> inputs) {
  if (torch::jit::tracer::isTracing() || c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode))
    return true;
  for (const Tensor* t : inputs)
    if (t->defined() && t->_fw_grad(0).defined()) return true;
  return false;
}
std::optional<double> scale_arg(PyObject* o) {
  if (o == Py_None) return std::nullopt;
  const double d = PyFloat_AsDouble(o);
  if (d == -1.0 && PyErr_Occurred()) throw python_error();
  return d;
}
int int_arg(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return static_cast<int>(v);
}
bool bool_arg(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
void expect(Py_ssize_t n, Py_ssize_t want) {
  if (n != want) raise(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
}
PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
PyObject* tuple_of(std::initializer_list<const Tensor*> ts) {
  PyObject* r = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
  if (!r) throw python_error();
  Py_ssize_t i = 0;
  for (const Tensor* t : ts) PyTuple_SET_ITEM(r, i++, wrap(*t));
  return r;
}

// sdp_attention(q, k, v, mode, kvLens, scale, mask) -> O, with an autograd node where one is needed; NotImplemented where
// the call is for the Python autograd function
PyObject* py_sdp_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 7);
  const Tensor &q = tensor_of(a[0], "q"), &k = tensor_of(a[1], "k"), &v = tensor_of(a[2], "v");
  if (needs_python_function({&q, &k, &v})) Py_RETURN_NOTIMPLEMENTED;
  const bool grad = wants_grad(q, k, v);
  check_qkv(q, k, v, grad);
  const int mode = int_arg(a[3]);
  const Tensor kv_lens = optional_of(a[4], "kvLens");
  const float scale = scale_or_default(scale_arg(a[5]), q.size(3));
  const Mask mask = mask_of(optional_of(a[6], "attnMask"), q, k.size(2));
  FwdResult r;
  {
    NoGil nogil;
    r = attn_fwd(q, k, v, mode, scale, kv_lens, grad, Tensor(), mask);
    if (grad) {
      auto node = std::shared_ptr<AttentionBackward>(new AttentionBackward(), torch::autograd::deleteNode);
      node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
      node->q = SavedVariable(q, false), node->k = SavedVariable(k, false), node->v = SavedVariable(v, false);
      node->lse = SavedVariable(r.lse, false), node->kv_lens = same_memory(kv_lens), node->mask = mask;
      node->mask.t = same_memory(mask.t), node->mode = mode, node->scale = scale;
      torch::autograd::set_history(r.o, node);
      node->o = SavedVariable(r.o, true);
    }
  }
  return wrap(r.o);
  END_HANDLE_TH_ERRORS
}

// attn_fwd(q, k, v, mode, scale, kvLens, needLse, status, mask) -> (O, LSE or None)
PyObject* py_attn_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 9);
  const Tensor &q = tensor_of(a[0], "q"), &k = tensor_of(a[1], "k"), &v = tensor_of(a[2], "v");
  check_qkv(q, k, v, false);
  const int mode = int_arg(a[3]);
  const float scale = scale_or_default(scale_arg(a[4]), q.size(3));
  const Tensor kv_lens = optional_of(a[5], "kvLens"), status = optional_of(a[7], "status");
  const bool need_lse = bool_arg(a[6]);
  const Mask mask = mask_of(optional_of(a[8], "attnMask"), q, k.size(2));
  FwdResult r;
  {
    NoGil nogil;
    r = attn_fwd(q, k, v, mode, scale, kv_lens, need_lse, status, mask);
  }
  return tuple_of({&r.o, &r.lse});
  END_HANDLE_TH_ERRORS
}

// attn_bwd(dO, q, k, v, o, lse, mode, scale, kvLens, need_dq, need_dk, need_dv, mask) -> (dQ, dK, dV), None where not needed
PyObject* py_attn_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 13);
  const Tensor &dO = tensor_of(a[0], "dO"), &q = tensor_of(a[1], "q"), &k = tensor_of(a[2], "k"), &v = tensor_of(a[3], "v"),
               &o = tensor_of(a[4], "o"), &lse = tensor_of(a[5], "lse");
  check_attn_tensor(dO, "dO");
  check_attn_tensor(q, "q");
  check_attn_tensor(k, "k");
  check_attn_tensor(v, "v");
  check_attn_tensor(o, "o");
  check_bwd(dO, q, k, v, o, lse);
  const int mode = int_arg(a[6]);
  const float scale = scale_or_default(scale_arg(a[7]), q.size(3));
  const Tensor kv_lens = optional_of(a[8], "kvLens");
  const bool needs[3] = {bool_arg(a[9]), bool_arg(a[10]), bool_arg(a[11])};
  const Mask mask = mask_of(optional_of(a[12], "attnMask"), q, k.size(2));
  BwdResult r;
  {
    NoGil nogil;
    r = attn_bwd(dO, q, k, v, o, lse, mode, scale, kv_lens, needs, mask);
  }
  return tuple_of({&r.g[0], &r.g[1], &r.g[2]});
  END_HANDLE_TH_ERRORS
}

// decode(q, kCache, vCache, kvLens, scale, needLse, workspace) -> (O, LSE or None)
PyObject* py_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 7);
  const Tensor &q = tensor_of(a[0], "q"), &k = tensor_of(a[1], "kCache"), &v = tensor_of(a[2], "vCache");
  check_attn_tensor(q, "q");
  check_attn_tensor(k, "kCache");
  check_attn_tensor(v, "vCache");
  if (q.size(2) != 1) raise(PyExc_ValueError, "decode takes exactly one query per sequence");
  check_kv(q, k, v, false);
  const Tensor kv_lens = optional_of(a[3], "kvLens"), ws = optional_of(a[6], "workspace");
  check_ints(kv_lens, Tensor(), q);
  if (ws.defined() && (ws.device() != q.device() || !ws.is_contiguous()))
    raise(PyExc_ValueError, "workspace must be a contiguous tensor on the device of q");
  const float scale = scale_or_default(scale_arg(a[4]), q.size(3));
  const bool need_lse = bool_arg(a[5]);
  Tensor o, lse;
  {
    NoGil nogil;
    const int64_t B = q.size(0), Hq = q.size(1), D = q.size(3);
    tt_attn_decode_params p{};
    set_common(&p, q);
    o = empty({B, Hq, 1, D}, q.scalar_type(), q.device());
    if (need_lse) lse = empty({B, Hq}, at::kFloat, q.device());
    p.dtype = dtype_of(q.scalar_type());
    p.B = B, p.Hq = Hq, p.Hkv = k.size(1), p.capacity = k.size(2), p.D = D;
    p.q = q.data_ptr(), p.k = k.data_ptr(), p.v = v.data_ptr(), p.o = o.data_ptr();
    p.lse = need_lse ? static_cast<float*>(lse.data_ptr()) : nullptr;
    p.q_strides = strides_of(q), p.k_strides = strides_of(k), p.v_strides = strides_of(v), p.o_strides = strides_of(o);
    p.scale = scale, p.kv_lens = ints_ptr(kv_lens);
    p.alloc = &hook;
    if (ws.defined()) p.workspace = ws.data_ptr(), p.workspace_bytes = ws.numel() * ws.element_size();
    check(api.decode(&p));
  }
  return tuple_of({&o, &lse});
  END_HANDLE_TH_ERRORS
}

// decode_append(q, kNew, vNew, kCache, vCache, kvLens, ropeCos, ropeSin, interleaved, scale, needLse, status)
// -> (O, LSE or None, newLens)
PyObject* py_decode_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 12);
  const Tensor &q = tensor_of(a[0], "q"), &kn = tensor_of(a[1], "kNew"), &vn = tensor_of(a[2], "vNew"),
               &kc = tensor_of(a[3], "kCache"), &vc = tensor_of(a[4], "vCache");
  check_attn_tensor(q, "q");
  check_attn_tensor(kn, "kNew");
  check_attn_tensor(vn, "vNew");
  check_attn_tensor(kc, "kCache");
  check_attn_tensor(vc, "vCache");
  const int64_t B = q.size(0), Hq = q.size(1), Hkv = kc.size(1), D = q.size(3);
  const at::DimVector row = {B, Hkv, 1, D};
  if (q.size(2) != 1 || kn.sizes() != at::IntArrayRef(row) || vn.sizes() != at::IntArrayRef(row))
    raise(PyExc_ValueError, "decode-append takes one query and one new key / value row per sequence");
  check_kv(q, kc, vc, false);
  check_operand(kn, "kNew", q, B, Hkv, 1);
  check_operand(vn, "vNew", q, B, Hkv, 1);
  const Tensor kv_lens = optional_of(a[5], "kvLens");
  if (!kv_lens.defined() || !kv_lens.is_cuda()) raise(PyExc_ValueError, "kvLens (int32 [B] on the device of q) is required");
  const Tensor cos = optional_of(a[6], "ropeCos"), sin = optional_of(a[7], "ropeSin"), status = optional_of(a[11], "status");
  check_ints(kv_lens, status, q);
  if (cos.defined() && (!sin.defined() || cos.scalar_type() != at::kFloat || cos.sizes() != sin.sizes() || cos.dim() != 2 ||
                        cos.size(1) != D / 2 || !cos.is_contiguous() || !sin.is_contiguous() || sin.scalar_type() != at::kFloat ||
                        cos.device() != q.device() || sin.device() != q.device()))
    raise(PyExc_ValueError, "rope tables must be contiguous fp32 [positions, D/2] on the device of q");
  const bool interleaved = bool_arg(a[8]), need_lse = bool_arg(a[10]);
  const float scale = scale_or_default(scale_arg(a[9]), D);
  Tensor o, lse, new_lens;
  {
    NoGil nogil;
    tt_attn_decode_append_params p{};
    set_common(&p, q);
    o = empty({B, Hq, 1, D}, q.scalar_type(), q.device());
    if (need_lse) lse = empty({B, Hq}, at::kFloat, q.device());
    new_lens = empty(kv_lens.sizes(), at::kInt, kv_lens.device());
    p.dtype = dtype_of(q.scalar_type());
    p.B = B, p.Hq = Hq, p.Hkv = Hkv, p.capacity = kc.size(2), p.D = D;
    p.q = q.data_ptr(), p.k_new = kn.data_ptr(), p.v_new = vn.data_ptr();
    p.k_cache = kc.data_ptr(), p.v_cache = vc.data_ptr(), p.o = o.data_ptr();
    p.lse = need_lse ? static_cast<float*>(lse.data_ptr()) : nullptr;
    p.q_strides = strides_of(q), p.k_new_strides = strides_of(kn), p.v_new_strides = strides_of(vn);
    p.k_strides = strides_of(kc), p.v_strides = strides_of(vc), p.o_strides = strides_of(o);
    p.scale = scale, p.kv_lens = ints_ptr(kv_lens), p.new_lens = static_cast<int32_t*>(new_lens.data_ptr());
    if (cos.defined()) {
      p.rope_cos = static_cast<const float*>(cos.data_ptr()), p.rope_sin = static_cast<const float*>(sin.data_ptr());
      p.rope_positions = cos.size(0);
    }
    p.rope_interleaved = interleaved ? 1 : 0;
    p.alloc = &hook;
    p.status = ints_ptr(status);
    check(api.decode_append(&p));
  }
  return tuple_of({&o, &lse, &new_lens});
  END_HANDLE_TH_ERRORS
}

// silu_mul(x [.., 2d]) -> [.., d]
PyObject* py_silu_mul(PyObject*, PyObject* x_obj) {
  HANDLE_TH_ERRORS
  Tensor x = tensor_of(x_obj, "x");
  if (!x.is_cuda() || dtype_of(x.scalar_type()) < 0)
    raise(PyExc_ValueError, "siluMul needs a CUDA tensor of dtype float32 / float16 / bfloat16 (no CPU path)");
  if (x.size(-1) % 2 != 0) raise(PyExc_AssertionError, "last dimension must be even (OpFusedCpu.h:16)");
  Tensor out;
  {
    NoGil nogil;
    at::NoGradGuard no_grad;
    x = x.contiguous();
    const int64_t d = x.size(-1) / 2;
    at::DimVector shape(x.sizes().begin(), x.sizes().end());
    shape.back() = d;
    out = empty(shape, x.scalar_type(), x.device());
    tt_silu_mul_params p{};
    set_common(&p, x);
    p.dtype = dtype_of(x.scalar_type());
    p.rows = d ? x.numel() / (2 * d) : 0, p.d = d;
    p.x = x.data_ptr(), p.out = out.data_ptr();
    check(api.silu_mul(&p));
  }
  return wrap(out);
  END_HANDLE_TH_ERRORS
}

// add_rms_norm(input, residual, weight, eps): in place
PyObject* py_add_rms_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 4);
  const Tensor &input = tensor_of(a[0], "input"), &residual = tensor_of(a[1], "residual"), &weight = tensor_of(a[2], "weight");
  for (const Tensor* t : {&input, &residual, &weight})
    if (!t->is_cuda() || t->device() != input.device() || t->scalar_type() != input.scalar_type() || dtype_of(t->scalar_type()) < 0)
      raise(PyExc_ValueError, "fusedAddRmsNorm needs tensors of one dtype (float32 / float16 / bfloat16) on one CUDA device");
  if (input.sizes() != residual.sizes())
    raise(PyExc_AssertionError, "input and residual must have the same shape (OpFusedCpu.h:44)");
  if (!(input.is_contiguous() && residual.is_contiguous() && weight.is_contiguous()))
    raise(PyExc_ValueError, "fusedAddRmsNorm works in place on dense tensors");
  const int64_t dim = input.size(-1);
  if (weight.numel() != dim) raise(PyExc_ValueError, "weight must have input.size(-1) elements");
  const double eps = PyFloat_AsDouble(a[3]);
  if (eps == -1.0 && PyErr_Occurred()) throw python_error();
  {
    NoGil nogil;
    tt_fused_add_rms_norm_params p{};
    set_common(&p, input);
    p.dtype = dtype_of(input.scalar_type());
    p.rows = dim ? input.numel() / dim : 0, p.dim = dim;
    p.input = input.data_ptr(), p.residual = residual.data_ptr(), p.weight = weight.data_ptr();
    p.eps = static_cast<float>(eps);
    check(api.add_rms_norm(&p));
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// linear(input, weight, bias or None); NotImplemented as sdp_attention
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 3);
  const Tensor &x = tensor_of(a[0], "input"), &w = tensor_of(a[1], "weight"), bias = optional_of(a[2], "bias");
  if (needs_python_function({&x, &w, &bias})) Py_RETURN_NOTIMPLEMENTED;
  return wrap(linear_autograd(x, w, bias));
  END_HANDLE_TH_ERRORS
}

// linear_bwd(dY [.., N], x2 [M, K], w [N, K], need_dx, need_dw, need_db) -> (dX [M, K], dW, db), None where not needed
PyObject* py_linear_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 6);
  const Tensor &dy = tensor_of(a[0], "dY"), &x2 = tensor_of(a[1], "x2"), &w = tensor_of(a[2], "w");
  for (const Tensor* t : {&x2, &w})
    if (t->dim() != 2 || (t->size(1) > 1 && t->stride(1) != 1) || t->scalar_type() != dy.scalar_type() || t->device() != dy.device())
      raise(PyExc_ValueError, "x2 [M, K] and w [N, K] must be matrices of dY's dtype and device with contiguous columns");
  if (!dy.is_cuda() || dy.dim() < 1 || dy.size(-1) != w.size(0) || x2.size(1) != w.size(1) || dy.numel() != x2.size(0) * w.size(0))
    raise(PyExc_ValueError, "dY must be a CUDA tensor [.., N] with the rows of x2");
  const bool needs[3] = {bool_arg(a[3]), bool_arg(a[4]), bool_arg(a[5])};
  LinearGrads g;
  {
    NoGil nogil;
    at::NoGradGuard no_grad;
    g = linear_bwd(dy, x2, w, x2.sizes(), needs);
  }
  return tuple_of({&g.g[0], &g.g[1], &g.g[2]});
  END_HANDLE_TH_ERRORS
}

// linear_raw(x2 [M, K], w [N, K], bias or None, status or None) -> [M, N], no autograd
PyObject* py_linear_raw(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 4);
  const Tensor &x = tensor_of(a[0], "x"), &w = tensor_of(a[1], "w");
  const Tensor status = optional_of(a[3], "status");
  if (x.dim() != 2 || w.dim() != 2 || x.size(1) != w.size(1) || w.scalar_type() != x.scalar_type() || !x.is_cuda() ||
      w.device() != x.device() || (x.size(1) > 1 && (x.stride(1) != 1 || w.stride(1) != 1)))
    raise(PyExc_ValueError, "x [M, K] and w [N, K] must be CUDA matrices of one dtype and device with contiguous columns");
  const Tensor bias = bias_of(optional_of(a[2], "bias"), x, w.size(0));
  check_ints(status, "status", 1, x);
  Tensor y;
  {
    NoGil nogil;
    y = empty({x.size(0), w.size(0)}, x.scalar_type(), x.device());
    linear_raw(x, false, w, false, bias, y, status, Tensor());
  }
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// bind(path of libtt_attn.so, exception class): the library the calls go to
PyObject* py_bind(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  const char* path;
  PyObject* exc;
  if (!PyArg_ParseTuple(args, "sO", &path, &exc)) return nullptr;
  void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!h) raise(PyExc_ImportError, "%s", dlerror());
  auto sym = [&](auto*& fn, const char* name) {
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(dlsym(h, name));
    if (!fn) raise(PyExc_ImportError, "%s lacks %s", path, name);
  };
  sym(api.fwd, "tt_attn_fwd");
  sym(api.bwd, "tt_attn_bwd");
  sym(api.decode, "tt_attn_decode");
  sym(api.decode_append, "tt_attn_decode_append");
  sym(api.add_rms_norm, "tt_fused_add_rms_norm");
  sym(api.silu_mul, "tt_silu_mul");
  sym(api.linear, "tt_linear");
  sym(api.strerror, "tt_attn_strerror");
  sym(api.last_cuda_error, "tt_attn_last_cuda_error");
  Py_INCREF(exc);
  Py_XDECREF(attn_error);
  attn_error = exc;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyCFunction fast(PyObject* (*f)(PyObject*, PyObject* const*, Py_ssize_t)) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, nullptr},
    {"sdp_attention", fast(py_sdp_attention), METH_FASTCALL, nullptr},
    {"attn_fwd", fast(py_attn_fwd), METH_FASTCALL, nullptr},
    {"attn_bwd", fast(py_attn_bwd), METH_FASTCALL, nullptr},
    {"decode", fast(py_decode), METH_FASTCALL, nullptr},
    {"decode_append", fast(py_decode_append), METH_FASTCALL, nullptr},
    {"silu_mul", py_silu_mul, METH_O, nullptr},
    {"add_rms_norm", fast(py_add_rms_norm), METH_FASTCALL, nullptr},
    {"linear", fast(py_linear), METH_FASTCALL, nullptr},
    {"linear_bwd", fast(py_linear_bwd), METH_FASTCALL, nullptr},
    {"linear_raw", fast(py_linear_raw), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module_def); }
