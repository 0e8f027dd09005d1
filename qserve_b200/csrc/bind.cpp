// qserve_b200 -- CPython binding of the operators a decode step calls one by one (linear layers, decode attention, norms, quantisation, activation).
//
// Each function checks its tensors, takes the current stream of their device and calls the C ABI (include/qserve_b200.h).  The checks, the argument
// conversion and the current-stream lookup cost 5 us per linear layer and 20 us per attention call as Python over ctypes -- more than most of these
// kernels run; here a call takes about 3 us with its launch.  What is called, what is taken (whatever int(), float() and bool() take) and what is refused is
// as it was there: an argument that is no tensor raises TypeError, everything else what torch's own functions raise.  The Python functions of backend.py
// keep the names, argument orders and defaults and pass everything on by position.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <stdexcept>
#include <string>
#include <tuple>
#include <type_traits>
#include <vector>

#include "../../include/qserve_b200.h"

namespace {

struct Args {
  PyObject* const* a;
  Py_ssize_t n;
  const at::Tensor& tensor(int i) const {
    if (!THPVariable_Check(a[i])) {
      PyErr_Format(PyExc_TypeError, "argument %d must be a tensor, not %s", i + 1, Py_TYPE(a[i])->tp_name);
      throw python_error();
    }
    return THPVariable_Unpack(a[i]);
  }
  bool none(int i) const { return a[i] == Py_None; }
  void* ptr(int i) const { return tensor(i).data_ptr(); }
  void* ptr_or_none(int i) const { return none(i) ? nullptr : ptr(i); }
  int small(int i) const {  // whatever int() takes, in the low bits of a C int
    if (PyLong_Check(a[i])) return static_cast<int>(PyLong_AsUnsignedLongLongMask(a[i]));
    PyObject* n = PyNumber_Long(a[i]);
    if (n == nullptr) throw python_error();
    const int v = static_cast<int>(PyLong_AsUnsignedLongLongMask(n));
    Py_DECREF(n);
    return v;
  }
  float real(int i) const {  // whatever float() takes
    if (PyFloat_Check(a[i])) return static_cast<float>(PyFloat_AS_DOUBLE(a[i]));
    PyObject* n = PyNumber_Float(a[i]);
    if (n == nullptr) throw python_error();
    const float v = static_cast<float>(PyFloat_AS_DOUBLE(n));
    Py_DECREF(n);
    return v;
  }
  int truth(int i) const {
    const int v = PyObject_IsTrue(a[i]);
    if (v < 0) throw python_error();
    return v;
  }
};

void require(bool ok, const char* what) {
  if (!ok) throw std::runtime_error(what);
}
void require_cuda(const at::Tensor& t, const char* name) {
  if (!t.is_cuda()) throw std::runtime_error(std::string(name) + " must be on CUDA");
}

// fn(stream) with t's device current, on that device's current stream, without the interpreter lock
template <typename F>
void launch(const at::Tensor& t, F fn) {
  const int dev = t.get_device();
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != dev) guard.set_index(static_cast<c10::DeviceIndex>(dev));
  void* stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS rc = fn(stream);
  Py_END_ALLOW_THREADS if (rc != 0) throw std::runtime_error("qserve_b200 [" + std::to_string(rc) + "]: " + qs_last_error());
}

// ---- work spaces: one per device and kind, zeroed once, then owned by the library (self-cleaning counters).  A work space that was handed out is never
//      freed -- a captured CUDA graph may hold its address -- so outgrown ones stay in `retired`; the objects are left to the process's end ----
struct Workspaces {
  std::vector<at::Tensor> gemm, attention, retired;
};
Workspaces& workspaces() {
  static Workspaces* w = new Workspaces();
  return *w;
}
at::Tensor& grown(std::vector<at::Tensor>& v, int dev, size_t need) {
  require(dev >= 0 && dev < c10::cuda::device_count(), "no such CUDA device");
  if (static_cast<int>(v.size()) <= dev) v.resize(dev + 1);
  at::Tensor& ws = v[dev];
  if (!ws.defined() || static_cast<size_t>(ws.numel()) < need) {
    const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(dev));
    at::Tensor next = at::zeros({static_cast<int64_t>(need)}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev));
    if (ws.defined()) workspaces().retired.push_back(ws);
    ws = std::move(next);
  }
  return ws;
}
at::Tensor& gemm_ws(int dev) {
  static const size_t need = qs_gemm_workspace_bytes();
  return grown(workspaces().gemm, dev, need);
}
at::Tensor& attention_ws(int dev, int batch, int heads, int dim) { return grown(workspaces().attention, dev, qs_attention_workspace_bytes(batch, heads, dim)); }

PyObject* none() { Py_RETURN_NONE; }

// ---- linear layers ----
struct Gemm {
  int M, N, K;
};
Gemm gemm_common(const at::Tensor& x, const at::Tensor& w, const at::Tensor& out, int k_div) {
  require_cuda(x, "in_feats");
  require_cuda(w, "kernel");
  require_cuda(out, "out_feats");
  require(x.scalar_type() == at::kChar && w.scalar_type() == at::kChar, "in_feats and kernel must be int8");
  require(out.scalar_type() == at::kHalf, "out_feats must be float16");
  require(x.is_contiguous() && w.is_contiguous() && out.is_contiguous(), "GEMM operands must be contiguous");
  const int64_t M = x.size(0), K = x.size(1), N = out.size(-1);
  require(out.size(-2) == M, "out_feats rows must match in_feats rows");
  if (w.size(0) != N || w.size(1) * k_div != K) {
    std::string shape;
    for (const int64_t n : w.sizes()) shape += (shape.empty() ? "" : ", ") + std::to_string(n);
    throw std::runtime_error("kernel shape (" + shape + ") does not match N=" + std::to_string(N) + ", K=" + std::to_string(K));
  }
  return {static_cast<int>(M), static_cast<int>(N), static_cast<int>(K)};
}
int8_t* s8(void* p) { return static_cast<int8_t*>(p); }

PyObject* w4a8_per_chn(const Args& a) {  // in_feats, kernel, wscales, ascales, w_szs, a_ssums, out_feats, acc_out
  const at::Tensor &x = a.tensor(0), &w = a.tensor(1), &out = a.tensor(6);
  const Gemm g = gemm_common(x, w, out, 2);
  if (g.M == 0) return none();
  void *p[8];
  for (int i = 0; i < 7; ++i) p[i] = a.ptr(i);
  p[7] = a.ptr_or_none(7);
  at::Tensor& ws = gemm_ws(x.get_device());
  void* wp = ws.data_ptr();
  const size_t wn = ws.numel();
  launch(x, [&](void* s) { return qs_w4a8_gemm_per_chn(s8(p[0]), s8(p[1]), p[2], p[3], p[4], p[5], p[6], static_cast<int32_t*>(p[7]), g.M, g.N, g.K, wp, wn, s); });
  return none();
}
PyObject* w4a8_per_group(const Args& a) {  // in_feats, kernel, zeros, scales_i8, wscales, ascales, out_feats, acc_out
  const at::Tensor &x = a.tensor(0), &w = a.tensor(1), &z = a.tensor(2), &s2 = a.tensor(3), &out = a.tensor(6);
  const Gemm g = gemm_common(x, w, out, 2);
  require(z.scalar_type() == at::kChar && s2.scalar_type() == at::kChar, "zeros and scales_i8 must be int8");
  auto fits = [&](const at::Tensor& t) { return t.dim() == 2 && t.size(0) == g.K / 128 && t.size(1) == g.N; };
  require(fits(z) && fits(s2), "level-2 params must be [K/128, N]");
  if (g.M == 0) return none();
  void *p[8];
  for (int i = 0; i < 7; ++i) p[i] = a.ptr(i);
  p[7] = a.ptr_or_none(7);
  at::Tensor& ws = gemm_ws(x.get_device());
  void* wp = ws.data_ptr();
  const size_t wn = ws.numel();
  launch(x, [&](void* s) { return qs_w4a8_gemm_per_group(s8(p[0]), s8(p[1]), s8(p[2]), s8(p[3]), p[4], p[5], p[6], static_cast<int32_t*>(p[7]), g.M, g.N, g.K, wp, wn, s); });
  return none();
}
PyObject* w8a8(const Args& a) {  // in_feats, kernel, wscales, ascales, out_feats, acc_out
  const at::Tensor &x = a.tensor(0), &w = a.tensor(1), &out = a.tensor(4);
  const Gemm g = gemm_common(x, w, out, 1);
  require(a.tensor(2).scalar_type() == at::kHalf && a.tensor(3).scalar_type() == at::kHalf, "wscales and ascales must be float16 (w8a8_linear.py:99-101 casts them)");
  if (g.M == 0) return none();
  void *p[6];
  for (int i = 0; i < 5; ++i) p[i] = a.ptr(i);
  p[5] = a.ptr_or_none(5);
  at::Tensor& ws = gemm_ws(x.get_device());
  void* wp = ws.data_ptr();
  const size_t wn = ws.numel();
  launch(x, [&](void* s) { return qs_w8a8_gemm(s8(p[0]), s8(p[1]), p[2], p[3], p[4], static_cast<int32_t*>(p[5]), g.M, g.N, g.K, wp, wn, s); });
  return none();
}

// ---- decode attention ----
PyObject* single_query_attention(const Args& a) {  // the 15 arguments of the operator
  const at::Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &kvp = a.tensor(3);
  require_cuda(q, "q");
  require_cuda(k, "k");
  require_cuda(v, "v");
  require_cuda(kvp, "kv_pointers");
  require(q.scalar_type() == at::kHalf && k.scalar_type() == at::kHalf && v.scalar_type() == at::kHalf,
          "single_query_attention: only float16 is supported (fused_attention.cpp:24-30)");
  const int64_t batch = kvp.size(0), heads = q.size(1), heads_kv = k.size(1), dim = k.size(-1);
  require(k.stride(2) == 1 && k.stride(1) == dim, "k must have stride(2) == 1 and stride(1) == head_dim");
  require(v.stride(2) == 1 && v.stride(1) == dim, "v must have stride(2) == 1 and stride(1) == head_dim");
  require(q.stride(2) == 1 && q.stride(1) == dim, "q must have stride(2) == 1 and stride(1) == head_dim");
  require(kvp.is_contiguous() && kvp.scalar_type() == at::kLong, "kv_pointers must be contiguous int64");
  void* lens = nullptr;
  if (!a.none(4)) {
    const at::Tensor& l = a.tensor(4);
    require_cuda(l, "length_per_sample");
    require(l.dim() == 1 && l.size(0) == batch, "length_per_sample must have shape (batch_size)");
    require(l.is_contiguous(), "length_per_sample must be contiguous");
    require(l.scalar_type() == at::kInt, "length_per_sample must be int32");
    lens = l.data_ptr();
  }
  if (!a.none(5)) {  // accepted, validated and ignored, exactly like the reference (:192-199, :91)
    const at::Tensor& s = a.tensor(5);
    require_cuda(s, "alibi_slopes");
    require(s.dim() == 1 && s.size(0) == heads && s.scalar_type() == at::kFloat, "alibi_slopes must be float32 [nheads]");
  }
  const int max_seqlen = a.small(6), tpb = a.small(7), spt = a.small(8), timestep = a.small(9), rot = a.small(10);
  const float base = a.real(11);
  const int neox = a.truth(12), int4 = a.truth(13), zeros = a.truth(14);
  at::Tensor out = at::empty({q.size(0), heads, dim}, q.options().requires_grad(false));
  at::Tensor& ws = attention_ws(q.get_device(), static_cast<int>(batch), static_cast<int>(heads), static_cast<int>(dim));
  void *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr(), *tp = kvp.data_ptr(), *op = out.data_ptr(), *wp = ws.data_ptr();
  const int64_t qs = q.stride(0), ks = k.stride(0), vs = v.stride(0), blocks = kvp.size(-1);
  const size_t wn = ws.numel();
  launch(q, [&](void* s) {
    return qs_single_query_attention(qp, kp, vp, qs, ks, vs, static_cast<const int64_t*>(tp), static_cast<const int32_t*>(lens), op, static_cast<int>(batch),
                                     static_cast<int>(heads), static_cast<int>(heads_kv), static_cast<int>(dim), static_cast<int>(blocks), max_seqlen, tpb, spt,
                                     timestep, rot, base, neox, int4, zeros, wp, wn, s);
  });
  return THPVariable_Wrap(std::move(out));
}
PyObject* single_query_attention_quant(const Args& a) {  // the 16 arguments of the operator
  const at::Tensor &q = a.tensor(0), &k = a.tensor(1), &v = a.tensor(2), &kvp = a.tensor(3);
  const int64_t batch = kvp.size(0);
  if (batch == 0) return none();
  const int64_t heads = q.size(1), heads_kv = k.size(1), dim = k.size(-1);
  require(q.scalar_type() == at::kHalf && q.stride(2) == 1 && q.stride(1) == dim, "q must be float16 with stride(1) == head_dim");
  require(k.stride(1) == dim && v.stride(1) == dim && kvp.is_contiguous(), "k, v, kv_pointers layout");
  const at::Tensor& oq = a.tensor(13);
  require(oq.scalar_type() == at::kChar && oq.is_contiguous() && oq.numel() == batch * heads * dim, "out_q must be int8 [B, Hq*D]");
  const int max_seqlen = a.small(5), tpb = a.small(6), spt = a.small(7), timestep = a.small(8), rot = a.small(9);
  const float base = a.real(10);
  const int int4 = a.truth(11), zeros = a.truth(12);
  require_cuda(q, "q");
  at::Tensor& ws = attention_ws(q.get_device(), static_cast<int>(batch), static_cast<int>(heads), static_cast<int>(dim));
  void *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr(), *tp = kvp.data_ptr(), *lens = a.tensor(4).data_ptr(), *op = oq.data_ptr(), *sp = a.tensor(14).data_ptr(),
       *up = a.ptr_or_none(15), *wp = ws.data_ptr();
  const int64_t qs = q.stride(0), ks = k.stride(0), vs = v.stride(0), blocks = kvp.size(-1);
  const size_t wn = ws.numel();
  launch(q, [&](void* s) {
    return qs_single_query_attention_quant(qp, kp, vp, qs, ks, vs, static_cast<const int64_t*>(tp), static_cast<const int32_t*>(lens), s8(op), sp, up,
                                           static_cast<int>(batch), static_cast<int>(heads), static_cast<int>(heads_kv), static_cast<int>(dim),
                                           static_cast<int>(blocks), max_seqlen, tpb, spt, timestep, rot, base, int4, zeros, wp, wn, s);
  });
  return none();
}

// ---- row operators ----
struct Rows {
  int tokens, width;
};
Rows rows_of(const at::Tensor& t) {
  const int64_t w = t.size(-1);
  return {static_cast<int>(w ? t.numel() / w : 0), static_cast<int>(w)};
}
void half_only(const at::Tensor& t, const char* op) {
  if (t.scalar_type() != at::kHalf)
    throw std::runtime_error(std::string(op) + ": only float16 activations are supported by qserve_b200 (models run .half(), model_runner.py:148)");
}
PyObject* rms_norm_general(const Args& a) {  // out, input, weight, scaling, epsilon, use_per_token_quant
  const at::Tensor& x = a.tensor(1);
  require_cuda(x, "input");
  half_only(x, "rms_norm_general");
  if (x.numel() == 0) return none();
  const Rows r = rows_of(x);
  void *o = a.tensor(0).data_ptr(), *xp = x.data_ptr(), *w = a.tensor(2).data_ptr(), *sc = a.tensor(3).data_ptr();
  const float eps = a.real(4);
  const int quant = a.truth(5);
  launch(x, [&](void* s) { return qs_rms_norm_general(s8(o), xp, w, sc, eps, quant, r.tokens, r.width, s); });
  return none();
}
PyObject* rms_norm_general_fuse_sum(const Args& a) {  // out, input, weight, input_sum, scaling, epsilon, use_per_token_quant
  const at::Tensor& x = a.tensor(1);
  require_cuda(x, "input");
  half_only(x, "rms_norm_general_fuse_sum");
  if (x.numel() == 0) return none();
  const Rows r = rows_of(x);
  void *o = a.tensor(0).data_ptr(), *xp = x.data_ptr(), *w = a.tensor(2).data_ptr(), *sum = a.tensor(3).data_ptr(), *sc = a.tensor(4).data_ptr();
  const float eps = a.real(5);
  const int quant = a.truth(6);
  launch(x, [&](void* s) { return qs_rms_norm_general_fuse_sum(s8(o), xp, w, sum, sc, eps, quant, r.tokens, r.width, s); });
  return none();
}
PyObject* quant(const at::Tensor& o, const at::Tensor& x, const at::Tensor* sum, const at::Tensor& scale, const char* op, const char* layout) {
  require_cuda(x, "input");
  half_only(x, op);
  require(x.is_contiguous() && o.is_contiguous(), layout);
  if (x.numel() == 0) return none();
  const Rows r = rows_of(x);
  void *op_ = o.data_ptr(), *xp = x.data_ptr(), *sc = scale.data_ptr(), *su = sum != nullptr ? sum->data_ptr() : nullptr;
  launch(x, [&](void* s) { return sum != nullptr ? qs_invoke_quant_fuse_sum(s8(op_), xp, su, sc, r.tokens, r.width, s) : qs_invoke_quant(s8(op_), xp, sc, r.tokens, r.width, s); });
  return none();
}
PyObject* invoke_quant(const Args& a) {  // out, input, scale tensor
  return quant(a.tensor(0), a.tensor(1), nullptr, a.tensor(2), "invoke_quant", "invoke_quant: input and out must be contiguous");
}
PyObject* invoke_quant_fuse_sum(const Args& a) {  // out, input, input_sum, scale tensor
  return quant(a.tensor(0), a.tensor(1), &a.tensor(2), a.tensor(3), "invoke_quant_fuse_sum", "invoke_quant_fuse_sum: input and out must be contiguous");
}
PyObject* silu_and_mul(const Args& a) {  // out, input
  const at::Tensor& x = a.tensor(1);
  require_cuda(x, "input");
  half_only(x, "silu_and_mul");
  if (x.numel() == 0) return none();
  const Rows r = rows_of(x);
  void *o = a.tensor(0).data_ptr(), *xp = x.data_ptr();
  launch(x, [&](void* s) { return qs_silu_and_mul(o, xp, r.tokens, r.width / 2, s); });
  return none();
}
PyObject* silu_and_mul_quant(const Args& a) {  // out, input, input_sum or None, scale
  const at::Tensor& x = a.tensor(1);
  require_cuda(x, "input");
  half_only(x, "silu_and_mul_quant");
  if (x.numel() == 0) return none();
  const Rows r = rows_of(x);
  void *o = a.tensor(0).data_ptr(), *xp = x.data_ptr(), *su = a.ptr_or_none(2), *sc = a.tensor(3).data_ptr();
  launch(x, [&](void* s) { return qs_silu_and_mul_quant(s8(o), xp, su, sc, r.tokens, r.width / 2, s); });
  return none();
}
PyObject* add_rms_norm_general(const Args& a) {  // out, hidden_out, x, delta, weight, input_sum or None, scaling, epsilon
  const at::Tensor& x = a.tensor(2);
  require_cuda(x, "x");
  half_only(x, "add_rms_norm_general");
  half_only(a.tensor(3), "add_rms_norm_general");
  if (x.numel() == 0) return none();
  const Rows r = rows_of(x);
  void *o = a.tensor(0).data_ptr(), *h = a.tensor(1).data_ptr(), *xp = x.data_ptr(), *d = a.tensor(3).data_ptr(), *w = a.tensor(4).data_ptr(), *su = a.ptr_or_none(5),
       *sc = a.tensor(6).data_ptr();
  const float eps = a.real(7);
  launch(x, [&](void* s) { return qs_add_rms_norm_general(s8(o), h, xp, d, w, su, sc, eps, r.tokens, r.width, s); });
  return none();
}

// ---- work spaces, for the operators that stay in Python ----
PyObject* gemm_workspace(const Args& a) { return THPVariable_Wrap(gemm_ws(a.small(0))); }
PyObject* attention_workspace(const Args& a) { return THPVariable_Wrap(attention_ws(a.small(0), a.small(1), a.small(2), a.small(3))); }

template <PyObject* (*Fn)(const Args&), int N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != N) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
    return nullptr;
  }
  try {
    return Fn(Args{args, n});
  } catch (...) {  // as torch's own functions raise them: IndexError for a missing dimension, OutOfMemoryError, RuntimeError for the rest
    torch::translate_exception_to_python(std::current_exception());
  }
  return nullptr;
}

// ---- functions of the C ABI as they are declared: conversions in the order and of the types of the declaration (pointers: an address or None;
//      integers: whatever has an __index__, as ctypes takes them), then the call without the interpreter lock; returns its status.  The attention and state
//      functions of the hybrid decoders have 25 to 40 arguments, a layer of short prompts five such calls: 79 us through ctypes, 69 here; a prompt's attention
//      block 56 and 50 ----
template <typename T>
T converted(PyObject* o) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) return nullptr;
    if (PyLong_Check(o)) {
      void* const p = PyLong_AsVoidPtr(o);
      if (p == nullptr && PyErr_Occurred()) throw python_error();
      return static_cast<T>(p);
    }
  } else if constexpr (std::is_floating_point_v<T>) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return static_cast<T>(v);
  } else {
    static_assert(std::is_integral_v<T>);
    if (PyLong_Check(o)) return static_cast<T>(PyLong_AsUnsignedLongLongMask(o));
    if (PyIndex_Check(o)) {  // numbers of numpy, tensors of one integer: sizes that a program read out of an array
      PyObject* const i = PyNumber_Index(o);
      if (i == nullptr) throw python_error();
      const T v = static_cast<T>(PyLong_AsUnsignedLongLongMask(i));
      Py_DECREF(i);
      return v;
    }
  }
  PyErr_Format(PyExc_TypeError, "%s expected, not %s", std::is_pointer_v<T> ? "an address or None" : "an integer", Py_TYPE(o)->tp_name);
  throw python_error();
}
template <auto Fn>
struct Abi;
template <typename... A, int (*Fn)(A...)>
struct Abi<Fn> {
  static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != static_cast<Py_ssize_t>(sizeof...(A))) {
      PyErr_Format(PyExc_TypeError, "expected %zu arguments, got %zd", sizeof...(A), n);
      return nullptr;
    }
    try {
      Py_ssize_t i = 0;
      const std::tuple<A...> a{converted<A>(args[i++])...};  // in order: a braced list
      int rc;
      Py_BEGIN_ALLOW_THREADS rc = std::apply(Fn, a);
      Py_END_ALLOW_THREADS return PyLong_FromLong(rc);
    } catch (...) {
      torch::translate_exception_to_python(std::current_exception());
    }
    return nullptr;
  }
};
#define QS_ABI(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&Abi<&name>::call)), METH_FASTCALL, nullptr}
#define QS_ENTRY(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&entry<name, n>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {QS_ENTRY(w4a8_per_chn, 8),
                         QS_ENTRY(w4a8_per_group, 8),
                         QS_ENTRY(w8a8, 6),
                         QS_ENTRY(single_query_attention, 15),
                         QS_ENTRY(single_query_attention_quant, 16),
                         QS_ENTRY(rms_norm_general, 6),
                         QS_ENTRY(rms_norm_general_fuse_sum, 7),
                         QS_ENTRY(invoke_quant, 3),
                         QS_ENTRY(invoke_quant_fuse_sum, 4),
                         QS_ENTRY(silu_and_mul, 2),
                         QS_ENTRY(silu_and_mul_quant, 4),
                         QS_ENTRY(add_rms_norm_general, 8),
                         QS_ENTRY(gemm_workspace, 1),
                         QS_ENTRY(attention_workspace, 4),
                         QS_ABI(qs_apply_bias_rope_update_kv_cache),
                         QS_ABI(qs_compute_padding_offsets),
                         QS_ABI(qs_prefill_attention),
                         QS_ABI(qs_hyb_attention),
                         QS_ABI(qs_hyb_attention_fast),
                         QS_ABI(qs_hyb_bias_gated_act),
                         QS_ABI(qs_hyb_bias_gelu_tanh),
                         QS_ABI(qs_hyb_branch_norm_mean),
                         QS_ABI(qs_hyb_cast_rows),
                         QS_ABI(qs_hyb_embed),
                         QS_ABI(qs_hyb_gate_recurrence),
                         QS_ABI(qs_hyb_gated_delta),
                         QS_ABI(qs_hyb_gated_linear),
                         QS_ABI(qs_hyb_gated_norm_update),
                         QS_ABI(qs_hyb_gelu_tanh_mul),
                         QS_ABI(qs_hyb_latent_attention),
                         QS_ABI(qs_hyb_latent_attention_fast),
                         QS_ABI(qs_hyb_latent_gate_out),
                         QS_ABI(qs_hyb_latent_prepare),
                         QS_ABI(qs_hyb_latent_query),
                         QS_ABI(qs_hyb_lru_conv),
                         QS_ABI(qs_hyb_lru_scan),
                         QS_ABI(qs_hyb_moe_act),
                         QS_ABI(qs_hyb_moe_combine),
                         QS_ABI(qs_hyb_moe_gather),
                         QS_ABI(qs_hyb_moe_plan),
                         QS_ABI(qs_hyb_moe_router),
                         QS_ABI(qs_hyb_post_norm_update),
                         QS_ABI(qs_hyb_qk_prepare_append),
                         QS_ABI(qs_hyb_qk_row_norm_append),
                         QS_ABI(qs_hyb_retention),
                         QS_ABI(qs_hyb_rms_norm),
                         QS_ABI(qs_hyb_rope_append),
                         QS_ABI(qs_hyb_softcap),
                         QS_ABI(qs_hyb_state_space),
                         QS_ABI(qs_hyb_stream_norm),
                         QS_ABI(qs_hyb_stream_update_norm),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_bind", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__bind(void) { return PyModule_Create(&module); }
