// native_ops.cpp — the differentiable operators of ops/functional.py that a training or serving layer calls most, as autograd
// functions in C++ over the same C entry points of libsxb200.so.
//
// What bounds small layers is the host: a Python autograd function costs 30 to 40 us per direction (context, views, ctypes), so one
// decoder layer of a small model on a ragged micro-batch of 662 tokens took 940 us of host time for 250 us of kernels, and a
// projection of a decode batch 14.5 us for a kernel of 10.  With these functions the layer
// takes 440 us, 2 x 300 rows of attention forward and backward 70 (150 before), the host side of a projection 7 (14.5).
//
// A weight's marks are read again in backward, where they decide who takes the gradient.
//
// Every function here looks at what it is given and returns None for anything that is not the plain case: another device, type or layout,
// tensor subclasses, forward-mode levels, tracing, function transforms, dispatch modes, weights that carry the main-grad
// protocol (attributes ops/functional.py reads).  The Python operator then goes its own way, errors included.  Tensors are saved through
// the autograd context, so hooks on saved tensors and version checks see them as before.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>
#include <string>

#include "sxb200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------------------------ the C library
struct Lib {                                   // (typed by the header, which the kernels' sources are checked against)
  decltype(&sxb_gemm_bf16) gemm_bf16;
  decltype(&sxb_rmsnorm_fwd) rmsnorm_fwd;
  decltype(&sxb_rmsnorm_bwd) rmsnorm_bwd;
  decltype(&sxb_norm_bwd_scratch_elems) norm_bwd_scratch_elems;
  decltype(&sxb_rope) rope;
  decltype(&sxb_rope_copy) rope_copy;
  decltype(&sxb_gated_act_fwd) gated_act_fwd;
  decltype(&sxb_gated_act_bwd) gated_act_bwd;
  decltype(&sxb_attn_fwd) attn_fwd;
  decltype(&sxb_attn_bwd) attn_bwd;
};
Lib g_lib;
bool g_bound = false;                          // written once, under the GIL
PyObject* g_error = nullptr;                   // the exception type of the Python binding, once bound
std::atomic<long long> g_calls{0};             // entry points called since they were last taken
PyObject* g_marks[3];                          // attributes of the main-grad protocol
// What backward passes ask of Python: the gradients through marked weights, and the number of ranks told to the library.
PyObject *g_linear_bwd = nullptr, *g_rms_norm_bwd = nullptr, *g_know_ranks = nullptr;

// A refused or failed call raises the binding's error, in a backward pass too: as a Python exception that the autograd engine hands on.
[[noreturn]] void refuse(const std::string& what) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(g_error, what.c_str());
  python_error e;
  e.persist();
  throw e;
}

void check(const char* name, int rc) {
  g_calls.fetch_add(1, std::memory_order_relaxed);
  if (rc == 0) return;
  std::string what = std::string("sxb_") + name;
  if (rc > 0) {
    what += " failed: cudaError " + std::to_string(rc);
  } else {
    const char* why = rc == -1 ? "bad argument" : rc == -2 ? "unsupported shape/alignment" : rc == -3 ? "size beyond limit"
                    : rc == -4 ? "driver entry point unavailable" : "error";
    what += std::string(" rejected the call: ") + why + " (" + std::to_string(rc) + ")";
  }
  refuse(what);
}

bool marked(PyObject* o) {                     // carries the main-grad protocol, or may
  PyObject** d = _PyObject_GetDictPtr(o);
  if (d == nullptr || *d == nullptr) return false;
  for (PyObject* m : g_marks)
    if (PyDict_Contains(*d, m) != 0) return true;
  return false;
}
// Calls f of the Python side; what it raises goes on to whoever runs the backward pass.  The GIL is held.
pybind11::object ask(PyObject* f, const pybind11::tuple& args) {
  PyObject* r = PyObject_CallObject(f, args.ptr());
  if (r == nullptr) {
    python_error e;
    e.persist();
    throw e;
  }
  return pybind11::reinterpret_steal<pybind11::object>(r);
}
pybind11::object py(const Tensor& t) {
  return t.defined() ? pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(t)) : pybind11::object(pybind11::none());
}
// Where the weight has come under the main-grad protocol since the forward pass: the gradients as Python's function f returns or
// delivers them (a tuple of tensors and None) for what args() gives.  False where it carries no mark.
template <typename Args>
bool through_python(PyObject* f, const Tensor& weight, variable_list& grads, Args&& args) {
  pybind11::gil_scoped_acquire gil;
  if (!marked(py(weight).ptr())) return false;
  const pybind11::object r = ask(f, args());
  for (size_t i = 0; i < grads.size(); ++i) {
    PyObject* g = PyTuple_GET_ITEM(r.ptr(), i);
    if (g != Py_None) grads[i] = THPVariable_Unpack(g);
  }
  return true;
}

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return 0;
    case at::kHalf: return 1;
    case at::kBFloat16: return 2;
    default: return -1;
  }
}

Tensor rows_of(const Tensor& t, int64_t width) {           // [rows, width], contiguous
  Tensor r = t.dim() == 2 ? t : t.reshape({-1, width});
  return r.is_contiguous() ? r : r.contiguous();
}

bool aligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

enum { kNT, kNN, kTN };
void gemm(const Tensor& a, const Tensor& b, const Tensor& out, int64_t M, int64_t N, int64_t K, int layout) {
  check("gemm_bf16", g_lib.gemm_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, layout, (int)a.stride(0),
                                     (int)b.stride(0), (int)N, 2, 0, 1.f, 0, stream()));
}

// ------------------------------------------------------------------------------------------------ operators
Tensor linear_fwd(const Tensor& x, const Tensor& w) {
  const int64_t K = w.size(1), N = w.size(0);
  std::vector<int64_t> shape = x.sizes().vec();
  shape.back() = N;
  Tensor y = at::empty(shape, x.options());
  // x is contiguous: its rows are K apart whatever its shape
  check("gemm_bf16", g_lib.gemm_bf16(x.data_ptr(), w.data_ptr(), y.data_ptr(), (int)(x.numel() / K), (int)N, (int)K, kNT, (int)K,
                                     (int)w.stride(0), (int)N, 2, 0, 1.f, 0, stream()));
  return y;
}

struct Linear : Function<Linear> {
  static Variable forward(AutogradContext* ctx, const Variable& x, const Variable& w) {
    Tensor y = linear_fwd(x, w);
    ctx->save_for_backward({x, w});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    const int64_t K = w.size(1), N = w.size(0);
    const Tensor dy = rows_of(grads[0], N);
    const int64_t M = dy.size(0);
    const bool want_x = ctx->needs_input_grad(0), want_w = ctx->needs_input_grad(1);
    variable_list delivered(2);
    if (through_python(g_linear_bwd, w, delivered, [&] { return pybind11::make_tuple(py(rows_of(x, K)), py(w), py(dy), want_x, want_w); }))
      return {want_x ? delivered[0].view(x.sizes()) : Tensor(), delivered[1]};
    Tensor dx, dw;
    if (want_x) {
      dx = at::empty(x.sizes(), dy.options());
      gemm(dy, w, dx, M, K, N, kNN);
    }
    if (want_w) {
      dw = at::empty({N, K}, w.options());
      const Tensor x2 = rows_of(x, K);
      gemm(dy, x2, dw, N, K, M, kTN);
    }
    return {dx, dw};
  }
};

// y, and the sum with the residual where there is one; rstd may be undefined
variable_list rms_norm_fwd(const Tensor& x, const Tensor& w, double eps, const std::optional<Tensor>& res, const Tensor& rstd) {
  const int64_t H = x.size(-1);
  Tensor y = at::empty(x.sizes(), x.options()), h;
  if (res) h = at::empty(x.sizes(), x.options());
  check("rmsnorm_fwd", g_lib.rmsnorm_fwd(x.data_ptr(), res ? res->data_ptr() : nullptr, w.data_ptr(), y.data_ptr(),
                                         res ? h.data_ptr() : nullptr, rstd.defined() ? rstd.data_ptr() : nullptr, x.numel() / H,
                                         (int)H, (float)eps, dtype_code(x), stream()));
  if (res) return {y, h};
  return {y};
}

struct RmsNorm : Function<RmsNorm> {
  static variable_list forward(AutogradContext* ctx, const Variable& x, const Variable& w, double eps,
                               const std::optional<Variable>& res) {
    const Tensor rstd = at::empty({x.numel() / x.size(-1)}, x.options().dtype(at::kFloat));
    variable_list out = rms_norm_fwd(x, w, eps, res, rstd);
    ctx->save_for_backward({res ? out[1] : x, w, rstd});
    ctx->saved_data["res"] = res.has_value();
    ctx->set_materialize_grads(false);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &src = saved[0], &w = saved[1], &rstd = saved[2];
    const bool res = ctx->saved_data["res"].toBool();
    const int64_t H = src.size(-1), rows = src.numel() / H;
    const Tensor dy = grads[0].defined() ? rows_of(grads[0], H) : at::zeros(src.sizes(), src.options());
    Tensor dres;
    if (res && grads[1].defined()) dres = rows_of(grads[1], H);
    variable_list delivered(2);
    if (through_python(g_rms_norm_bwd, w, delivered,
                       [&] { return pybind11::make_tuple(py(rows_of(src, H)), py(w), py(rstd), py(rows_of(dy, H)), py(dres)); })) {
      const Tensor dx = delivered[0].view(src.sizes());
      return {dx, delivered[1], Variable(), res ? dx : Variable()};
    }
    Tensor dx = at::empty(src.sizes(), src.options()), dw = at::empty(w.sizes(), w.options());
    // (its own scratch: passes on other streams may run at the same time)
    const Tensor scratch = at::empty({g_lib.norm_bwd_scratch_elems(rows, (int)H, 0)}, src.options().dtype(at::kFloat));
    check("rmsnorm_bwd", g_lib.rmsnorm_bwd(dy.data_ptr(), src.data_ptr(), w.data_ptr(), rstd.data_ptr(),
                                           dres.defined() ? dres.data_ptr() : nullptr, dx.data_ptr(), dw.data_ptr(),
                                           scratch.data_ptr(), rows, (int)H, dtype_code(src), 0, stream()));
    return {dx, dw, Variable(), res ? dx : Variable()};
  }
};

void rope_kernel(const Tensor& x, const Tensor& pos, const Tensor& cos, const Tensor& sin, int64_t heads, int64_t dim, int inverse) {
  const int64_t C = x.size(-1);
  check("rope", g_lib.rope(x.data_ptr(), pos.defined() ? pos.data_ptr() : nullptr, cos.data_ptr(), sin.data_ptr(), x.numel() / C,
                           (int)heads, (int)dim, C, inverse, dtype_code(x), stream()));
}

struct Rope : Function<Rope> {                 // in place
  static Variable forward(AutogradContext* ctx, const Variable& x, const std::optional<Variable>& pos, const Variable& cos,
                          const Variable& sin, int64_t heads, int64_t dim) {
    ctx->mark_dirty({x});
    rope_kernel(x, pos ? *pos : Tensor(), cos, sin, heads, dim, 0);
    ctx->save_for_backward({pos ? *pos : Tensor(), cos, sin});
    ctx->saved_data["heads"] = heads;
    ctx->saved_data["dim"] = dim;
    return x;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const int64_t heads = ctx->saved_data["heads"].toInt(), dim = ctx->saved_data["dim"].toInt();
    const Tensor& dy = grads[0];
    const int64_t C = dy.size(-1);
    // never rotate autograd's buffer in place
    if (dy.is_contiguous() && dim % 16 == 0 && C % 8 == 0 && (C - heads * dim) % 16 == 0 && aligned(dy) && C < (int64_t(1) << 31)) {
      Tensor dx = at::empty(dy.sizes(), dy.options());
      check("rope_copy", g_lib.rope_copy(dy.data_ptr(), dx.data_ptr(), saved[0].defined() ? saved[0].data_ptr() : nullptr,
                                         saved[1].data_ptr(), saved[2].data_ptr(), dy.numel() / C, (int)heads, (int)dim, (int)C, 1,
                                         dtype_code(dy), stream()));
      return {dx, Variable(), Variable(), Variable(), Variable(), Variable()};
    }
    const Tensor dx = dy.clone(at::MemoryFormat::Contiguous);
    rope_kernel(dx, saved[0], saved[1], saved[2], heads, dim, 1);
    return {dx, Variable(), Variable(), Variable(), Variable(), Variable()};
  }
};

Tensor gated_fwd(const Tensor& x, int64_t act) {
  const int64_t F = x.size(-1) / 2;
  std::vector<int64_t> shape = x.sizes().vec();
  shape.back() = F;
  Tensor y = at::empty(shape, x.options());
  check("gated_act_fwd", g_lib.gated_act_fwd(x.data_ptr(), nullptr, y.data_ptr(), x.numel() / (2 * F), (int)F, (int)act,
                                             dtype_code(x), stream()));
  return y;
}

struct Gated : Function<Gated> {
  static Variable forward(AutogradContext* ctx, const Variable& x, int64_t act) {
    ctx->save_for_backward({x});
    ctx->saved_data["act"] = act;
    return gated_fwd(x, act);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor& x = saved[0];
    const int64_t F = x.size(-1) / 2;
    const Tensor dy = rows_of(grads[0], F);
    Tensor dx = at::empty(x.sizes(), x.options());
    check("gated_act_bwd", g_lib.gated_act_bwd(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), dy.size(0), (int)F,
                                               (int)ctx->saved_data["act"].toInt(), dtype_code(x), stream()));
    return {dx, Variable()};
  }
};

struct Heads {
  int64_t Hq, Hk, D;
  bool causal;
  double scale;
};
const void* column(const Tensor& t, int64_t c) { return (const char*)t.data_ptr() + c * 2; }

Tensor attention_fwd(const Tensor& qkv, const Heads& a, const Tensor& lse) {
  const int64_t B = qkv.size(0), S = qkv.size(1), C = qkv.size(2);
  Tensor out = at::empty({B, S, a.Hq, a.D}, qkv.options());
  check("attn_fwd", g_lib.attn_fwd(qkv.data_ptr(), column(qkv, a.Hq * a.D), column(qkv, (a.Hq + a.Hk) * a.D), out.data_ptr(),
                                   lse.data_ptr(), (int)B, (int)S, (int)a.Hq, (int)a.Hk, (int)a.D, C, C, C, out.stride(1), a.causal,
                                   (float)a.scale, stream()));
  return out;
}

struct Attention : Function<Attention> {
  static Variable forward(AutogradContext* ctx, const Variable& qkv, int64_t Hq, int64_t Hk, int64_t D, bool causal, double scale) {
    const Heads a{Hq, Hk, D, causal, scale};
    const Tensor lse = at::empty({qkv.size(0), Hq, qkv.size(1)}, qkv.options().dtype(at::kFloat));
    Tensor out = attention_fwd(qkv, a, lse);
    ctx->save_for_backward({qkv, out, lse});
    ctx->saved_data["Hk"] = Hk;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &qkv = saved[0], &out = saved[1], &lse = saved[2];
    const int64_t B = out.size(0), S = out.size(1), Hq = out.size(2), D = out.size(3), C = qkv.size(2);
    const int64_t Hk = ctx->saved_data["Hk"].toInt();
    Tensor dout = grads[0];
    if (dout.stride(3) != 1 || dout.stride(2) != D || dout.stride(0) != S * dout.stride(1)) dout = dout.contiguous();
    Tensor dqkv = at::empty(qkv.sizes(), qkv.options());
    const Tensor delta = at::empty({B, Hq, S}, qkv.options().dtype(at::kFloat));
    const int64_t k0 = Hq * D, v0 = (Hq + Hk) * D;
    {
      pybind11::gil_scoped_acquire gil;        // a process group may have come about since the forward pass
      ask(g_know_ranks, pybind11::tuple());
    }
    check("attn_bwd", g_lib.attn_bwd(qkv.data_ptr(), column(qkv, k0), column(qkv, v0), out.data_ptr(), dout.data_ptr(),
                                     lse.data_ptr(), delta.data_ptr(), dqkv.data_ptr(), (void*)column(dqkv, k0),
                                     (void*)column(dqkv, v0), (int)B, (int)S, (int)Hq, (int)Hk, (int)D, C, C, C, out.stride(1),
                                     dout.stride(1), C, C, C, ctx->saved_data["causal"].toBool(),
                                     (float)ctx->saved_data["scale"].toDouble(), stream()));
    return {dqkv, Variable(), Variable(), Variable(), Variable(), Variable()};
  }
};

// ------------------------------------------------------------------------------------------------ Python side
// Nothing but autograd watches what happens here.
bool unwatched() {
  return g_bound && g_know_ranks != nullptr && torch::autograd::ForwardADLevel::try_get_by_idx(0) == nullptr && !torch::jit::tracer::isTracing() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) && c10::impl::TorchDispatchModeTLS::stack_len() == 0;
}
// A tensor or parameter itself (no subclass), dense and on the GPU; null if it is something else.
const Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && !t.is_neg() && !t.is_conj() ? &t : nullptr;
}
bool tape(const Tensor& a) { return a.requires_grad(); }

constexpr int64_t kMost = int64_t(1) << 31;

// Runs f without the GIL and wraps what it returns.
template <typename F>
PyObject* run(F&& f) {
  HANDLE_TH_ERRORS                             // (hooks on saved tensors may raise too: a checkpoint stops its recomputation so)
  variable_list out;
  {
    pybind11::gil_scoped_release no_gil;
    out = f();
  }
  if (out.size() == 1) return THPVariable_Wrap(out[0]);
  PyObject* a = THPVariable_Wrap(out[0]);
  PyObject* b = THPVariable_Wrap(out[1]);
  PyObject* r = a && b ? PyTuple_Pack(2, a, b) : nullptr;
  Py_XDECREF(a);
  Py_XDECREF(b);
  return r;
  END_HANDLE_TH_ERRORS
}

// linear(x, weight)
PyObject* py_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) Py_RETURN_NONE;
  const Tensor *x = plain(args[0]), *w = plain(args[1]);
  if (!x || !w || !unwatched() || marked(args[1])) Py_RETURN_NONE;
  if (x->scalar_type() != at::kBFloat16 || w->scalar_type() != at::kBFloat16 || w->dim() != 2 || x->dim() < 1 || x->numel() == 0 ||
      x->size(-1) != w->size(1) || x->size(-1) % 8 || w->size(0) % 8 || w->size(0) == 0 || w->stride(1) != 1 || w->stride(0) % 8 ||
      w->stride(0) < w->size(1) || !x->is_contiguous() || !aligned(*x) || !aligned(*w) || x->device() != w->device() ||
      x->numel() / x->size(-1) >= kMost || w->stride(0) >= kMost || w->size(0) >= kMost)
    Py_RETURN_NONE;
  const bool grad = at::GradMode::is_enabled() && (tape(*x) || tape(*w));
  return run([&]() -> variable_list { return {grad ? Linear::apply(*x, *w) : linear_fwd(*x, *w)}; });
}

// rms_norm(x, weight, eps, residual or None) -> norm, or (norm, x + residual)
PyObject* py_rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4 || !PyFloat_CheckExact(args[2])) Py_RETURN_NONE;
  const Tensor *x = plain(args[0]), *w = plain(args[1]), *r = args[3] == Py_None ? nullptr : plain(args[3]);
  if (!x || !w || (!r && args[3] != Py_None) || !unwatched() || marked(args[1])) Py_RETURN_NONE;
  if (dtype_code(*x) < 0 || w->scalar_type() != x->scalar_type() || x->dim() < 1 || x->numel() == 0 || w->dim() != 1 ||
      w->size(0) != x->size(-1) || !w->is_contiguous() || !x->is_contiguous() || x->size(-1) >= kMost || w->device() != x->device())
    Py_RETURN_NONE;
  if (r && (r->scalar_type() != x->scalar_type() || r->sizes() != x->sizes() || !r->is_contiguous() || r->device() != x->device()))
    Py_RETURN_NONE;
  const double eps = PyFloat_AS_DOUBLE(args[2]);
  const bool grad = at::GradMode::is_enabled() && (tape(*x) || tape(*w) || (r && tape(*r)));
  const std::optional<Tensor> res = r ? std::optional<Tensor>(*r) : std::nullopt;
  return run([&]() -> variable_list { return grad ? RmsNorm::apply(*x, *w, eps, res) : rms_norm_fwd(*x, *w, eps, res, Tensor()); });
}

// rope(x, positions or None, cos, sin, heads, head size), in place
PyObject* py_rope(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6) Py_RETURN_NONE;
  const Tensor *x = plain(args[0]), *p = args[1] == Py_None ? nullptr : plain(args[1]), *c = plain(args[2]), *s = plain(args[3]);
  if (!x || (!p && args[1] != Py_None) || !c || !s || !unwatched()) Py_RETURN_NONE;
  const long heads = PyLong_AsLong(args[4]), dim = PyLong_AsLong(args[5]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (dtype_code(*x) < 0 || x->dim() < 1 || x->numel() == 0 || !x->is_contiguous() || x->is_inference() ||
      (p && (p->scalar_type() != at::kLong || !p->is_contiguous())) || c->scalar_type() != at::kFloat || s->scalar_type() != at::kFloat ||
      !c->is_contiguous() || !s->is_contiguous() || tape(*c) || tape(*s) || heads < 1 || dim < 1 || heads * dim > x->size(-1))
    Py_RETURN_NONE;
  if (!(at::GradMode::is_enabled() && tape(*x))) Py_RETURN_NONE;      // without a tape the Python function's bookkeeping is kept
  const std::optional<Tensor> pos = p ? std::optional<Tensor>(*p) : std::nullopt;
  return run([&]() -> variable_list { return {Rope::apply(*x, pos, *c, *s, (int64_t)heads, (int64_t)dim)}; });
}

// gated_act(x, code)
PyObject* py_gated(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) Py_RETURN_NONE;
  const Tensor* x = plain(args[0]);
  if (!x || !unwatched()) Py_RETURN_NONE;
  const long act = PyLong_AsLong(args[1]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (dtype_code(*x) < 0 || x->dim() < 2 || x->numel() == 0 || x->size(-1) % 2 || !x->is_contiguous() || x->size(-1) >= kMost)
    Py_RETURN_NONE;
  const bool grad = at::GradMode::is_enabled() && tape(*x);
  return run([&]() -> variable_list { return {grad ? Gated::apply(*x, (int64_t)act) : gated_fwd(*x, act)}; });
}

// attention_qkv(qkv, query heads, key heads, head size, causal, scale)
PyObject* py_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6) Py_RETURN_NONE;
  const Tensor* x = plain(args[0]);
  if (!x || !unwatched()) Py_RETURN_NONE;
  const long hq = PyLong_AsLong(args[1]), hk = PyLong_AsLong(args[2]), d = PyLong_AsLong(args[3]);
  const int causal = PyObject_IsTrue(args[4]);
  const double scale = PyFloat_AsDouble(args[5]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (x->scalar_type() != at::kBFloat16 || (d != 64 && d != 128) || hq < 1 || hk < 1 || hq % hk || x->dim() != 3 || x->numel() == 0 ||
      x->size(2) != (hq + 2 * hk) * d || !x->is_contiguous() || !aligned(*x) || x->size(0) >= kMost || x->size(1) >= kMost)
    Py_RETURN_NONE;
  const bool grad = at::GradMode::is_enabled() && tape(*x);
  return run([&]() -> variable_list {
    if (grad) return {Attention::apply(*x, (int64_t)hq, (int64_t)hk, (int64_t)d, (bool)causal, scale)};
    const Tensor lse = at::empty({x->size(0), hq, x->size(1)}, x->options().dtype(at::kFloat));
    return {attention_fwd(*x, Heads{hq, hk, d, (bool)causal, scale}, lse)};
  });
}

// bind(dlopen handle of libsxb200.so, exception type) -> whether every entry point is there
PyObject* py_bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) return PyErr_Format(PyExc_TypeError, "bind(handle, error)");
  void* h = PyLong_AsVoidPtr(args[0]);
  if (PyErr_Occurred()) return nullptr;
  Lib l{};
  bool all = true;
  auto get = [&](auto& f, const char* name) {
    f = reinterpret_cast<std::remove_reference_t<decltype(f)>>(dlsym(h, name));
    all = all && f != nullptr;
  };
  get(l.gemm_bf16, "sxb_gemm_bf16");
  get(l.rmsnorm_fwd, "sxb_rmsnorm_fwd");
  get(l.rmsnorm_bwd, "sxb_rmsnorm_bwd");
  get(l.norm_bwd_scratch_elems, "sxb_norm_bwd_scratch_elems");
  get(l.rope, "sxb_rope");
  get(l.rope_copy, "sxb_rope_copy");
  get(l.gated_act_fwd, "sxb_gated_act_fwd");
  get(l.gated_act_bwd, "sxb_gated_act_bwd");
  get(l.attn_fwd, "sxb_attn_fwd");
  get(l.attn_bwd, "sxb_attn_bwd");
  if (all) {
    Py_INCREF(args[1]);
    g_error = args[1];
    g_lib = l;
    g_bound = true;
  }
  return PyBool_FromLong(all);
}

// backward_side(gradients of a product, gradients of a norm, telling the library its ranks): see through_python
PyObject* py_backward_side(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) return PyErr_Format(PyExc_TypeError, "backward_side(linear, rms_norm, know_ranks)");
  PyObject** to[3] = {&g_linear_bwd, &g_rms_norm_bwd, &g_know_ranks};
  for (int i = 0; i < 3; ++i) {
    Py_INCREF(args[i]);
    *to[i] = args[i];
  }
  Py_RETURN_NONE;
}

PyObject* py_calls(PyObject*, PyObject*) { return PyLong_FromLongLong(g_calls.load(std::memory_order_relaxed)); }

PyMethodDef kMethods[] = {
    {"linear", (PyCFunction)(void*)py_linear, METH_FASTCALL, "linear(x, weight) -> tensor, or None: not the plain case"},
    {"rms_norm", (PyCFunction)(void*)py_rms_norm, METH_FASTCALL, "rms_norm(x, weight, eps, residual or None)"},
    {"rope", (PyCFunction)(void*)py_rope, METH_FASTCALL, "rope(x, positions or None, cos, sin, heads, head size), in place"},
    {"gated_act", (PyCFunction)(void*)py_gated, METH_FASTCALL, "gated_act(x, activation code)"},
    {"attention_qkv", (PyCFunction)(void*)py_attention, METH_FASTCALL, "attention_qkv(qkv, hq, hk, d, causal, scale)"},
    {"bind", (PyCFunction)(void*)py_bind, METH_FASTCALL, "bind(handle of libsxb200.so, exception type)"},
    {"backward_side", (PyCFunction)(void*)py_backward_side, METH_FASTCALL, "backward_side(linear, rms_norm, know_ranks)"},
    {"calls", py_calls, METH_NOARGS, "entry points called so far"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_sxb_ops", "Differentiable operators over libsxb200.so", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__sxb_ops() {
  const char* marks[3] = {"_sxb_main_grad", "_sxb_gate", "_sxb_grad_ready"};
  for (int i = 0; i < 3; ++i)
    if ((g_marks[i] = PyUnicode_InternFromString(marks[i])) == nullptr) return nullptr;
  return PyModule_Create(&kModule);
}
