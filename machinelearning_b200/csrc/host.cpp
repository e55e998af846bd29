// The call path between torch and the C ABI, in C++: what flash_cuda.py, qk_prologue.py and value_gate.py do per
// call -- checks, casts, output allocation, the autograd node, the launch -- without Python in it.
//
// Why: the kernels of a small call are a few microseconds, and with the Python forms of these functions (ctypes
// marshalling, autograd.Function, a backward that needs the interpreter lock in the engine's thread) the host was
// what took the time: forward + backward of B=2 T=100 H=4/2 D=64 was 133 us, back to back, with under 30 us of
// kernels.  The Python forms stay for what a compiler traces and for callers that replace `flash_cuda.fwd`.
//
// Every function that may decline returns None; the Python caller then takes the general path, which
// raises the documented error or handles the case.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/csrc/utils/pybind.h>

#include <cmath>

#include "../../include/nlfa.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

bool g_tensor_cores = false;                       // the load-time self-test passed
bool g_watched[64] = {};                           // devices whose status word the host can read
PyObject* g_check = nullptr;                       // _lib.check: raises for a non-zero status

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return NLFA_DTYPE_F32;
    case at::kHalf: return NLFA_DTYPE_F16;
    case at::kBFloat16: return NLFA_DTYPE_BF16;
    default: return -1;
  }
}

// Raises what _lib.check raises (its NlfaError names the status), from any thread.
void check(const char* fn, int status) {
  if (status == NLFA_OK) return;
  py::gil_scoped_acquire gil;
  PyObject* r = PyObject_CallFunction(g_check, "si", fn, status);
  Py_XDECREF(r);
  python_error err;
  err.persist();
  throw err;
}

// A CUDA tensor this file may take by its data pointer: no subclass with a dispatch of its own, no transform, no
// forward-mode gradient.
bool plain(const Tensor& t) {
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && !t.unsafeGetTensorImpl()->is_python_dispatch() &&
         !t.key_set().has(c10::DispatchKey::FuncTorchBatched) && !t.key_set().has(c10::DispatchKey::FuncTorchGradWrapper) &&
         !t._fw_grad(0).defined();
}
bool watched(const Tensor& t) { return g_watched[t.device().index() & 63]; }

Tensor empty(at::IntArrayRef size, at::ScalarType dtype, const Tensor& like) {
  return Tensor(at::detail::empty_cuda(size, dtype, like.device(), std::nullopt));
}
Tensor empty_as(const Tensor& t) { return empty(t.sizes(), t.scalar_type(), t); }

Tensor contiguous(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
Tensor cast(const Tensor& t, at::ScalarType dtype) { return t.scalar_type() == dtype ? t : t.to(dtype); }
Tensor f32(const Tensor& t) { return contiguous(cast(t.requires_grad() ? t.detach() : t, at::kFloat)); }

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

bool recording(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

template <typename N>
std::shared_ptr<N> make_node() {
  return std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
}

// What once_differentiable does: gradients of a backward that was itself differentiated raise when used.
variable_list once(variable_list grads, const Tensor& dout) {
  if (!(at::GradMode::is_enabled() && dout.requires_grad())) return grads;
  auto err = std::make_shared<torch::autograd::DelayedError>(
      "trying to differentiate twice a function that was marked with @once_differentiable",
      static_cast<int64_t>(grads.size()));
  for (Tensor& g : grads) g.set_requires_grad(true);      // so that what comes back has an edge to the error
  return err->apply(std::move(grads));
}

// ------------------------------------------------------------------------------------------ attention core

struct Mask {
  int window, sinks, block;
};

struct Shape {
  int B, T, H, Hkv, D, dtype;
};
Shape shape_of(const Tensor& q, const Tensor& k) {
  return {static_cast<int>(q.size(0)), static_cast<int>(q.size(1)), static_cast<int>(q.size(2)),
          static_cast<int>(k.size(2)), static_cast<int>(q.size(3)), dtype_code(q.scalar_type())};
}

std::pair<Tensor, Tensor> attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, double scale, bool tensor_cores,
                                       Mask m) {
  const c10::cuda::CUDAGuard guard(q.device());
  const Shape s = shape_of(q, k);
  Tensor o = empty_as(q), lse = empty({s.B, s.H, s.T}, at::kFloat, q);
  check("nlfa_fwd", nlfa_fwd_masked(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
                                    static_cast<float*>(lse.data_ptr()), s.B, s.T, s.H, s.Hkv, s.D,
                                    static_cast<float>(scale), m.window, m.sinks, m.block, s.dtype,
                                    tensor_cores ? NLFA_PATH_TENSOR : NLFA_PATH_SIMT, stream_of(q)));
  return {o, lse};
}

variable_list attn_backward(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o,
                            const Tensor& lse, double scale, bool tensor_cores, bool fused, Mask m) {
  const c10::cuda::CUDAGuard guard(q.device());
  const Shape s = shape_of(q, k);
  const int path = tensor_cores ? NLFA_PATH_TENSOR : NLFA_PATH_SIMT;
  const size_t bytes = fused ? nlfa_bwd_fused_scratch_bytes(s.B, s.T, s.H, s.D)
                             : nlfa_bwd_workspace_bytes(s.B, s.T, s.H, s.Hkv, s.D, m.window, m.sinks, m.block, s.dtype, path);
  Tensor dq = empty_as(q), dk = empty_as(k), dv = empty_as(v);
  Tensor scratch;
  try {
    scratch = empty({static_cast<int64_t>(bytes > 16 ? bytes : 16)}, at::kByte, q);
  } catch (const c10::OutOfMemoryError&) {
    // room for dS is a matter of speed: with the tape alone the backward recomputes it, to the same bits
    const size_t least = nlfa_bwd_scratch_bytes(s.B, s.T, s.H);
    if (fused || bytes <= least) throw;
    scratch = empty({static_cast<int64_t>(least > 16 ? least : 16)}, at::kByte, q);
  }
  check("nlfa_bwd_masked",
        nlfa_bwd_masked(dout.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
                        static_cast<const float*>(lse.data_ptr()), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                        scratch.data_ptr(), static_cast<size_t>(scratch.numel()), s.B, s.T, s.H, s.Hkv, s.D,
                        static_cast<float>(scale), m.window, m.sinks, m.block, s.dtype, path,
                        fused ? (NLFA_PASS_DELTA | NLFA_PASS_FUSED) : NLFA_PASS_ALL, stream_of(q)));
  return {dq, dk, dv};
}

struct FlashAttnBackward : public Node {
  SavedVariable q, k, v, o, lse;
  double scale;
  bool tensor_cores;
  Mask mask;
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    Tensor q_ = q.unpack(), o_ = o.unpack(shared_from_this());
    Tensor dout = grads[0].defined() ? contiguous(grads[0]) : at::zeros_like(o_);
    return once(attn_backward(dout, q_, k.unpack(), v.unpack(), o_, lse.unpack(), scale, tensor_cores, false, mask), dout);
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&q, &k, &v, &o, &lse}) s->reset_data();
  }
  std::string name() const override { return "FlashAttnBackward"; }
};

// ------------------------------------------------------------------------------------------ q/k prologue

struct QkPrologueBackward : public Node {
  SavedVariable x, w, c, s, rstd;
  bool has_weight, has_rope;
  at::ScalarType weight_dtype;
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    Tensor x_ = x.unpack(), w_ = has_weight ? w.unpack() : Tensor(), c_ = has_rope ? c.unpack() : Tensor(),
           s_ = has_rope ? s.unpack() : Tensor(), rstd_ = rstd.unpack();
    const c10::cuda::CUDAGuard guard(x_.device());
    Tensor gy = grads[0].defined() ? contiguous(grads[0]) : at::zeros_like(x_);
    const int B = x_.size(0), T = x_.size(1), H = x_.size(2), D = x_.size(3);
    Tensor gx = empty_as(x_), gw, scratch;
    if (has_weight) {
      gw = empty({D}, at::kFloat, x_);
      scratch = empty({static_cast<int64_t>(nlfa_qk_prologue_scratch_bytes(D))}, at::kByte, x_);
    } else {
      scratch = empty({4}, at::kByte, x_);
    }
    check("nlfa_qk_prologue_bwd",
          nlfa_qk_prologue_bwd(gy.data_ptr(), dtype_code(gy.scalar_type()), x_.data_ptr(), dtype_code(x_.scalar_type()),
                               has_weight ? static_cast<float*>(w_.data_ptr()) : nullptr,
                               has_rope ? static_cast<float*>(c_.data_ptr()) : nullptr,
                               has_rope ? static_cast<float*>(s_.data_ptr()) : nullptr,
                               static_cast<float*>(rstd_.data_ptr()), gx.data_ptr(),
                               has_weight ? static_cast<float*>(gw.data_ptr()) : nullptr,
                               static_cast<float*>(scratch.data_ptr()), static_cast<size_t>(scratch.numel()), B, T, H, D,
                               stream_of(x_)));
    if (has_weight) gw = cast(gw, weight_dtype);
    variable_list out = once(has_weight ? variable_list{gx, gw} : variable_list{gx}, gy);
    out.resize(2);
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&x, &w, &c, &s, &rstd}) v->reset_data();
  }
  std::string name() const override { return "QkPrologueBackward"; }
};

Tensor prologue(const Tensor& x_in, const Tensor& weight, const Tensor& cos, const Tensor& sin, double eps,
                at::ScalarType out_dtype) {
  const c10::cuda::CUDAGuard guard(x_in.device());
  const bool rec = recording({&x_in, &weight});
  const Tensor x = contiguous(x_in);
  const bool has_weight = weight.defined(), has_rope = cos.defined();
  const Tensor w = has_weight ? f32(weight) : Tensor(), c = has_rope ? f32(cos) : Tensor(), s = has_rope ? f32(sin) : Tensor();
  const int B = x.size(0), T = x.size(1), H = x.size(2), D = x.size(3);
  Tensor y = empty(x.sizes(), out_dtype, x);
  Tensor rstd = empty({has_weight ? static_cast<int64_t>(B) * T * H : 1}, at::kFloat, x);
  check("nlfa_qk_prologue_fwd",
        nlfa_qk_prologue_fwd(x.data_ptr(), dtype_code(x.scalar_type()), has_weight ? static_cast<float*>(w.data_ptr()) : nullptr,
                             has_rope ? static_cast<float*>(c.data_ptr()) : nullptr,
                             has_rope ? static_cast<float*>(s.data_ptr()) : nullptr, y.data_ptr(), dtype_code(out_dtype),
                             static_cast<float*>(rstd.data_ptr()), B, T, H, D, static_cast<float>(eps), stream_of(x)));
  if (rec) {
    auto node = make_node<QkPrologueBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(x, weight));
    node->x = SavedVariable(x, false);
    if (has_weight) {
      node->w = SavedVariable(w, false);
      node->weight_dtype = weight.scalar_type();
    }
    if (has_rope) {
      node->c = SavedVariable(c, false);
      node->s = SavedVariable(s, false);
    }
    node->rstd = SavedVariable(rstd, false);
    node->has_weight = has_weight;
    node->has_rope = has_rope;
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ----------------------------------------------------------------------------- value blend and head gate

struct ValueBlendBackward : public Node {
  SavedVariable v, v0, lam;
  at::ScalarType lam_dtype;
  std::vector<int64_t> lam_shape;
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    Tensor v_ = v.unpack(), v0_ = v0.unpack(), lam_ = lam.unpack();
    const c10::cuda::CUDAGuard guard(v_.device());
    Tensor g = grads[0].defined() ? contiguous(grads[0]) : at::zeros_like(v_);
    Tensor dv = empty_as(v_), dv0 = empty_as(v0_);
    Tensor dlam = lam_dtype == at::kFloat ? empty(lam_shape, at::kFloat, v_) : empty({1}, at::kFloat, v_);
    Tensor scratch = empty({static_cast<int64_t>(nlfa_value_blend_scratch_bytes())}, at::kByte, v_);
    check("nlfa_value_blend_bwd",
          nlfa_value_blend_bwd(g.data_ptr(), dtype_code(g.scalar_type()), v_.data_ptr(), v0_.data_ptr(),
                               dtype_code(v_.scalar_type()), static_cast<float*>(lam_.data_ptr()), dv.data_ptr(),
                               dv0.data_ptr(), static_cast<float*>(dlam.data_ptr()), scratch.data_ptr(),
                               static_cast<size_t>(scratch.numel()), v_.numel(), stream_of(v_)));
    if (lam_dtype != at::kFloat) dlam = dlam.to(lam_dtype).reshape(lam_shape);
    return once({dv, dv0, dlam}, g);
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&v, &v0, &lam}) s->reset_data();
  }
  std::string name() const override { return "ValueBlendBackward"; }
};

Tensor blend(const Tensor& v_in, const Tensor& v0_in, const Tensor& lam, at::ScalarType out_dtype) {
  const c10::cuda::CUDAGuard guard(v_in.device());
  const bool rec = recording({&v_in, &v0_in, &lam});
  const Tensor v = contiguous(v_in), v0 = contiguous(v0_in), lam32 = f32(lam);
  Tensor out = empty(v.sizes(), out_dtype, v);
  check("nlfa_value_blend_fwd",
        nlfa_value_blend_fwd(v.data_ptr(), v0.data_ptr(), dtype_code(v.scalar_type()), static_cast<float*>(lam32.data_ptr()),
                             out.data_ptr(), dtype_code(out_dtype), v.numel(), stream_of(v)));
  if (rec) {
    auto node = make_node<ValueBlendBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(v, v0, lam));
    node->v = SavedVariable(v, false);
    node->v0 = SavedVariable(v0, false);
    node->lam = SavedVariable(lam32, false);
    node->lam_dtype = lam.scalar_type();
    node->lam_shape = lam.sizes().vec();
    torch::autograd::set_history(out, node);
  }
  return out;
}

struct HeadGateBackward : public Node {
  SavedVariable y, gate;
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    Tensor y_ = y.unpack(), gate_ = gate.unpack();
    const c10::cuda::CUDAGuard guard(y_.device());
    Tensor g = grads[0].defined() ? cast(contiguous(grads[0]), y_.scalar_type()) : at::zeros_like(y_);
    Tensor dy = empty_as(y_), dgate = empty_as(gate_);
    const int D = y_.size(3);
    check("nlfa_head_gate_bwd",
          nlfa_head_gate_bwd(g.data_ptr(), y_.data_ptr(), dtype_code(y_.scalar_type()), gate_.data_ptr(),
                             dtype_code(gate_.scalar_type()), dy.data_ptr(), dgate.data_ptr(), y_.numel() / D, D,
                             stream_of(y_)));
    return once({dy, dgate}, g);
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    y.reset_data();
    gate.reset_data();
  }
  std::string name() const override { return "HeadGateBackward"; }
};

Tensor head_gate(const Tensor& y_in, const Tensor& gate_in) {
  const c10::cuda::CUDAGuard guard(y_in.device());
  const bool rec = recording({&y_in, &gate_in});
  const Tensor y = contiguous(y_in), gate = contiguous(gate_in);
  Tensor out = empty_as(y);
  const int D = y.size(3);
  check("nlfa_head_gate_fwd",
        nlfa_head_gate_fwd(y.data_ptr(), dtype_code(y.scalar_type()), gate.data_ptr(), dtype_code(gate.scalar_type()),
                           out.data_ptr(), y.numel() / D, D, stream_of(y)));
  if (rec) {
    auto node = make_node<HeadGateBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(y, gate));
    node->y = SavedVariable(y, false);
    node->gate = SavedVariable(gate, false);
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ------------------------------------------------------------------------------------------- Python entries

bool is_tensor(PyObject* o) { return THPVariable_Check(o); }
bool tensor_or_none(PyObject* o) { return o == Py_None || THPVariable_Check(o); }
const Tensor& tensor(PyObject* o) { return THPVariable_Unpack(o); }
Tensor maybe(PyObject* o) { return o == Py_None ? Tensor() : THPVariable_Unpack(o); }
// What int(o), float(o) and bool(o) give, as the general path takes these arguments (a window of 4.0, a scale tensor).
int integer(PyObject* o) {
  THPObjectPtr i(PyLong_Check(o) ? Py_NewRef(o) : PyNumber_Long(o));
  const long v = i ? PyLong_AsLong(i.get()) : -1;
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return static_cast<int>(v);
}
double number(PyObject* o) {
  THPObjectPtr f(PyFloat_Check(o) ? Py_NewRef(o) : PyNumber_Float(o));
  if (!f) throw python_error();
  return PyFloat_AsDouble(f.get());
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v == 1;
}
void require_tensors(const char* fn, PyObject* const* a, int n) {
  for (int i = 0; i < n; ++i)
    TORCH_CHECK_TYPE(is_tensor(a[i]), fn, ": argument ", i + 1, " must be a tensor, not ", Py_TYPE(a[i])->tp_name);
}
PyObject* decline() { Py_RETURN_NONE; }

bool head_dim(int64_t D) { return D == 32 || D == 64 || D == 128; }
bool valid_mask(const Mask& m) {
  if (m.block < 0 || m.window < 0 || (m.block && m.window)) return false;
  return m.window == 0 ? m.sinks == 0 : m.sinks >= 0 && m.sinks < m.window;
}
std::optional<at::ScalarType> autocast_dtype() {
  if (!at::autocast::is_autocast_enabled(at::kCUDA)) return std::nullopt;
  return at::autocast::get_autocast_dtype(at::kCUDA);
}

// attn(q, k, v, scale | None, use_mma | None, window, sinks, block) -> [B,T,H,D] | None
PyObject* py_attn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8 || !is_tensor(a[0]) || !is_tensor(a[1]) || !is_tensor(a[2])) return decline();
  Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]);
  const Mask m{integer(a[5]), integer(a[6]), integer(a[7])};
  if (!plain(q) || !plain(k) || !plain(v) || q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || !watched(q) ||
      k.device() != q.device() || v.device() != q.device() || !valid_mask(m))
    return decline();
  const auto ac = autocast_dtype();
  if (!ac && (k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type())) return decline();
  const at::ScalarType dtype = ac ? *ac : q.scalar_type();
  if (dtype_code(dtype) < 0 || dtype_code(q.scalar_type()) < 0 || dtype_code(k.scalar_type()) < 0 ||
      dtype_code(v.scalar_type()) < 0)
    return decline();
  const auto qs = q.sizes(), ks = k.sizes();
  if (!head_dim(qs[3]) || ks != v.sizes() || ks[0] != qs[0] || ks[1] != qs[1] || ks[3] != qs[3] || ks[2] == 0 ||
      qs[2] % ks[2] != 0)
    return decline();
  bool tensor_cores = dtype != at::kFloat && g_tensor_cores;
  if (a[4] != Py_None) {
    if (truth(a[4]) && !tensor_cores) return decline();
    tensor_cores = truth(a[4]);
  }
  const double scale = a[3] == Py_None ? 1.0 / std::sqrt(static_cast<double>(qs[3])) : number(a[3]);
  Tensor o;
  {
    py::gil_scoped_release no_gil;
    q = contiguous(cast(q, dtype));
    k = contiguous(cast(k, dtype));
    v = contiguous(cast(v, dtype));
    Tensor lse;
    std::tie(o, lse) = attn_forward(q, k, v, scale, tensor_cores, m);
    if (recording({&q, &k, &v})) {
      auto node = make_node<FlashAttnBackward>();
      node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
      node->q = SavedVariable(q, false);
      node->k = SavedVariable(k, false);
      node->v = SavedVariable(v, false);
      node->lse = SavedVariable(lse, false);
      node->scale = scale;
      node->tensor_cores = tensor_cores;
      node->mask = m;
      torch::autograd::set_history(o, node);
      node->o = SavedVariable(o, true);
    }
  }
  return THPVariable_Wrap(o);
  END_HANDLE_TH_ERRORS
}

// attn_fwd(q, k, v, scale, use_mma, window, sinks, block) -> (o, lse): contiguous tensors of one dtype
PyObject* py_attn_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 8, "attn_fwd takes 8 arguments");
  require_tensors("attn_fwd", a, 3);
  const Mask m{integer(a[5]), integer(a[6]), integer(a[7])};
  const double scale = number(a[3]);
  const bool tc = truth(a[4]);
  const Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]);
  std::pair<Tensor, Tensor> r;
  {
    py::gil_scoped_release no_gil;
    r = attn_forward(q, k, v, scale, tc, m);
  }
  return Py_BuildValue("NN", THPVariable_Wrap(r.first), THPVariable_Wrap(r.second));
  END_HANDLE_TH_ERRORS
}

// attn_bwd(dout, q, k, v, o, lse, scale, use_mma, fused, window, sinks, block) -> (dq, dk, dv)
PyObject* py_attn_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 12, "attn_bwd takes 12 arguments");
  require_tensors("attn_bwd", a, 6);
  const Mask m{integer(a[9]), integer(a[10]), integer(a[11])};
  const double scale = number(a[6]);
  const bool tc = truth(a[7]), fused = truth(a[8]);
  const Tensor dout = tensor(a[0]), q = tensor(a[1]), k = tensor(a[2]), v = tensor(a[3]), o = tensor(a[4]), lse = tensor(a[5]);
  variable_list r;
  {
    py::gil_scoped_release no_gil;
    r = attn_backward(dout, q, k, v, o, lse, scale, tc, fused, m);
  }
  return Py_BuildValue("NNN", THPVariable_Wrap(r[0]), THPVariable_Wrap(r[1]), THPVariable_Wrap(r[2]));
  END_HANDLE_TH_ERRORS
}

// attn_cached(q, k, v, scale | None, qpos | None, kpos | None, causal, window, sinks, return_lse, use_mma | None)
//   -> o | (o, lse) | None
PyObject* py_attn_cached(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 11 || !is_tensor(a[0]) || !is_tensor(a[1]) || !is_tensor(a[2]) || !tensor_or_none(a[4]) || !tensor_or_none(a[5]))
    return decline();
  Tensor q = tensor(a[0]), k = tensor(a[1]), v = tensor(a[2]), qpos = maybe(a[4]), kpos = maybe(a[5]);
  const bool causal = truth(a[6]), want_lse = truth(a[9]);
  const Mask m{integer(a[7]), integer(a[8]), 0};
  if (!plain(q) || !plain(k) || !plain(v) || q.dim() != 4 || k.dim() != 4 || k.sizes() != v.sizes() ||
      k.device() != q.device() || v.device() != q.device() || k.scalar_type() != q.scalar_type() ||
      v.scalar_type() != q.scalar_type() || dtype_code(q.scalar_type()) < 0 || !valid_mask(m) || (m.window && !causal))
    return decline();
  const auto qs = q.sizes(), ks = k.sizes();
  if (!head_dim(qs[3]) || ks[0] != qs[0] || ks[3] != qs[3] || ks[1] == 0 || qs[2] % ks[1] != 0) return decline();
  const int B = qs[0], T = qs[1], H = qs[2], D = qs[3], Hkv = ks[1], L = ks[2];
  if (!qpos.defined() && T > L) return decline();
  if ((qpos.defined() && (!plain(qpos) || qpos.numel() != T)) || (kpos.defined() && (!plain(kpos) || kpos.numel() != L)))
    return decline();
  const int path = a[10] == Py_None ? NLFA_PATH_AUTO : truth(a[10]) ? NLFA_PATH_TENSOR : NLFA_PATH_SIMT;
  const double scale = a[3] == Py_None ? 1.0 / std::sqrt(static_cast<double>(D)) : number(a[3]);
  Tensor o, lse;
  {
    py::gil_scoped_release no_gil;
    const c10::cuda::CUDAGuard guard(q.device());
    auto detached = [](const Tensor& t) { return contiguous(t.requires_grad() ? t.detach() : t); };
    q = detached(q);
    k = detached(k);
    v = detached(v);
    const auto kind = [](const Tensor& t) { return t.defined() ? t.scalar_type() : at::kLong; };
    const bool wide = kind(qpos) == at::kLong && kind(kpos) == at::kLong;        // read as they are
    auto positions = [&](const Tensor& t) {
      return !t.defined() ? t : contiguous((t.device() == q.device() ? t : t.to(q.device())).to(wide ? at::kLong : at::kInt));
    };
    qpos = positions(qpos);
    kpos = positions(kpos);
    o = empty_as(q);
    if (want_lse) lse = empty({B, H, T}, at::kFloat, q);
    const int st = nlfa_fwd_cached_positions(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), want_lse ? static_cast<float*>(lse.data_ptr()) : nullptr,
        qpos.defined() ? qpos.data_ptr() : nullptr, kpos.defined() ? kpos.data_ptr() : nullptr, wide ? 8 : 4, B, T, H, Hkv, L, D, static_cast<float>(scale),
        causal ? 1 : 0, m.window, m.sinks, dtype_code(q.scalar_type()), path, nullptr, 0, stream_of(q));
    if (st == NLFA_ERR_UNSUPPORTED_PATH && path == NLFA_PATH_TENSOR)
      TORCH_CHECK_VALUE(false, "flash_attn_cached: use_mma=True but the tensor-core kernel does not apply to these inputs");
    check("nlfa_fwd_cached", st);
  }
  if (want_lse) return Py_BuildValue("NN", THPVariable_Wrap(o), THPVariable_Wrap(lse));
  return THPVariable_Wrap(o);
  END_HANDLE_TH_ERRORS
}

// qk_prologue(x, weight | None, cos | None, sin | None, eps, out_dtype | None) -> y | None
PyObject* py_qk_prologue(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !is_tensor(a[0])) return decline();
  for (int i = 1; i < 4; ++i)
    if (!tensor_or_none(a[i])) return decline();
  const Tensor x = tensor(a[0]), w = maybe(a[1]), c = maybe(a[2]), s = maybe(a[3]);
  if (!plain(x) || x.dim() != 4 || dtype_code(x.scalar_type()) < 0 || !head_dim(x.size(3))) return decline();
  const int64_t T = x.size(1), D = x.size(3);
  for (const Tensor* t : {&w, &c, &s})
    if (t->defined() && (!plain(*t) || t->device() != x.device())) return decline();
  if (w.defined() && (w.dim() != 1 || w.size(0) != D)) return decline();
  if (c.defined() != s.defined()) return decline();
  if (c.defined() && (c.dim() != 2 || c.size(0) != T || c.size(1) != D || s.sizes() != c.sizes())) return decline();
  at::ScalarType out = x.scalar_type();
  if (a[5] != Py_None) {
    if (!THPDtype_Check(a[5])) return decline();
    out = reinterpret_cast<THPDtype*>(a[5])->scalar_type;
  } else if (const auto ac = autocast_dtype()) {
    out = *ac;
  }
  if (dtype_code(out) < 0) return decline();
  const double eps = number(a[4]);
  Tensor y;
  {
    py::gil_scoped_release no_gil;
    y = prologue(x, w, c, s, eps, out);
  }
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// value_blend(v, v0, lam, out_dtype | None) -> out | None
PyObject* py_value_blend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || !is_tensor(a[0]) || !is_tensor(a[1]) || !is_tensor(a[2])) return decline();
  const Tensor v = tensor(a[0]), v0 = tensor(a[1]), lam = tensor(a[2]);
  if (!plain(v) || !plain(v0) || !plain(lam) || v0.device() != v.device() || lam.device() != v.device() ||
      dtype_code(v.scalar_type()) < 0 || v0.scalar_type() != v.scalar_type() || v.sizes() != v0.sizes() ||
      v.numel() % 8 != 0 || lam.numel() != 1)
    return decline();
  at::ScalarType out = v.scalar_type();
  if (a[3] != Py_None) {
    if (!THPDtype_Check(a[3])) return decline();
    out = reinterpret_cast<THPDtype*>(a[3])->scalar_type;
  } else if (const auto ac = autocast_dtype()) {
    out = *ac;
  }
  if (dtype_code(out) < 0) return decline();
  Tensor r;
  {
    py::gil_scoped_release no_gil;
    r = blend(v, v0, lam, out);
  }
  return THPVariable_Wrap(r);
  END_HANDLE_TH_ERRORS
}

// head_gate(y, gate) -> out | None
PyObject* py_head_gate(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2 || !is_tensor(a[0]) || !is_tensor(a[1])) return decline();
  const Tensor y = tensor(a[0]), gate = tensor(a[1]);
  if (!plain(y) || !plain(gate) || gate.device() != y.device() || y.dim() != 4 || gate.dim() != 3 ||
      dtype_code(y.scalar_type()) < 0 || dtype_code(gate.scalar_type()) < 0 || !head_dim(y.size(3)) ||
      gate.sizes() != y.sizes().slice(0, 3))
    return decline();
  Tensor r;
  {
    py::gil_scoped_release no_gil;
    r = head_gate(y, gate);
  }
  return THPVariable_Wrap(r);
  END_HANDLE_TH_ERRORS
}

// configure(check, tensor_cores): _lib.check and whether the self-test passed;  watch(device index)
PyObject* py_configure(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 2, "configure takes 2 arguments");
  Py_INCREF(a[0]);
  Py_XSETREF(g_check, a[0]);
  g_tensor_cores = truth(a[1]);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
PyObject* py_watch(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 1, "watch takes 1 argument");
  const int i = integer(a[0]);
  TORCH_CHECK(i >= 0 && i < 64, "device index out of range");
  g_watched[i] = true;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

#define NLFA_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {NLFA_METHOD(attn),        NLFA_METHOD(attn_fwd),    NLFA_METHOD(attn_bwd),  NLFA_METHOD(attn_cached),
                           NLFA_METHOD(qk_prologue), NLFA_METHOD(value_blend), NLFA_METHOD(head_gate), NLFA_METHOD(configure),
                           NLFA_METHOD(watch),       {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_host", "torch-facing call path of libnlfa (host.cpp)", -1, g_methods};

}  // namespace

#ifndef NLFA_HOST_STAMP
#define NLFA_HOST_STAMP ""
#endif

// What this was compiled against (_build.py looks for the text in the file before it is loaded).
PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&g_module);
  if (m != nullptr) PyModule_AddStringConstant(m, "built_for", NLFA_HOST_STAMP);
  return m;
}
