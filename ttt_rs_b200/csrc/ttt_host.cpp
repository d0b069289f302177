// Native host path between the Python operator and the C ABI (include/ttt_b200.h): argument checks, output and workspace
// allocation, stream lookup and the launch of one call without returning to the interpreter, and the autograd nodes of
// the two inner loops.
//
// Why it exists: through ctypes a call costs 20 us (one-token step of the TTT-Linear inner model, whose kernel takes 4 us)
// to 300 us (forward + backward through a Python autograd function) of interpreter time; here it costs 4 to 40 us.
//
// Every function takes what the call needs and returns its results, or None where the arguments are not the plain case
// (not contiguous, another dtype or shape, not on a GPU, an error code from the library): the Python code then walks
// through its own checks, which convert or raise.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/autocast_mode.h>
#include <torch/csrc/Exceptions.h>
#include <torch/torch.h>

#include "../../include/ttt_b200.h"
#include "ttt_internal.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int kMaxDevices = 64;
Tensor g_status[kMaxDevices];   // the status words of each device, handed over by the Python side when it creates them
PyObject* g_error_type = nullptr;  // TttError(code, message)

[[noreturn]] void throw_error(int rc) {
  pybind11::gil_scoped_acquire gil;
  PyObject* args = Py_BuildValue("(is)", rc, ttt_b200_last_error());
  PyObject* exc = args ? PyObject_CallObject(g_error_type, args) : nullptr;
  Py_XDECREF(args);
  if (exc) {
    PyErr_SetObject(g_error_type, exc);
    Py_DECREF(exc);
  }
  throw python_error();
}

bool on_16_bytes(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0; }
bool is(const Tensor& t, at::ScalarType dt, const c10::Device& dev, c10::IntArrayRef sizes) {
  return t.defined() && t.is_cuda() && t.device() == dev && t.scalar_type() == dt && t.sizes() == sizes &&
         t.is_contiguous() && t.layout() == c10::kStrided;
}

struct Dims {
  ttt_dims d;
  int64_t B, H, T, F;
  at::ScalarType dt = at::kBFloat16;
  c10::Device dev = c10::Device(c10::kCPU);
  Tensor status;
  // false: not the plain case
  bool set(const Tensor& xq, int64_t head_dim, int64_t mb, int64_t K, int64_t eps_scaled) {
    if (!xq.defined() || !xq.is_cuda() || xq.dim() != 4 || mb <= 0) return false;
    dt = xq.scalar_type();
    if (dt != at::kBFloat16 && dt != at::kFloat) return false;
    dev = xq.device();
    B = xq.size(0), H = xq.size(1), T = xq.size(2), F = xq.size(3);
    if (F != head_dim || dev.index() >= kMaxDevices || B > INT32_MAX || H > INT32_MAX || T > INT32_MAX) return false;
    status = g_status[dev.index()];
    d.batch = (int32_t)B;
    d.heads = (int32_t)H;
    d.seq_len = (int32_t)T;
    d.head_dim = (int32_t)F;
    d.mini_batch = (int32_t)mb;
    d.checkpoint_interval = (int32_t)K;
    d.epsilon = (float)eps_scaled * 1e-9f;  // float32 arithmetic, as FusedTttConfig.epsilon
    d.dtype = dt == at::kBFloat16 ? TTT_BF16 : TTT_F32;
    return true;
  }
  at::TensorOptions opt() const { return at::TensorOptions().dtype(dt).device(dev); }
  at::TensorOptions opt(at::ScalarType t) const { return at::TensorOptions().dtype(t).device(dev); }
  void* stream() const { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
};

struct LinIn {  // xq, xk, xv, weight, bias, token_eta, ttt_lr_eta, ln_weight, ln_bias
  Tensor t[9];
  bool plain(const Dims& m) const {
    const int64_t B = m.B, H = m.H, T = m.T, F = m.F;
    return is(t[0], m.dt, m.dev, {B, H, T, F}) && is(t[1], m.dt, m.dev, {B, H, T, F}) &&
           is(t[2], m.dt, m.dev, {B, H, T, F}) && is(t[3], m.dt, m.dev, {B, H, F, F}) && is(t[4], m.dt, m.dev, {B, H, F}) &&
           is(t[5], m.dt, m.dev, {T}) && is(t[6], m.dt, m.dev, {B, H, T}) && is(t[7], m.dt, m.dev, {H, F}) &&
           is(t[8], m.dt, m.dev, {H, F});
  }
  const void* p(int i) const { return t[i].const_data_ptr(); }
};

// ---- TTT-Linear --------------------------------------------------------------------------------------------------
struct LinOut {
  Tensor out, w, b, wck, bck;
};
int linear_forward(const Dims& m, const LinIn& in, bool save, LinOut& o) {
  c10::cuda::CUDAGuard guard(m.dev);
  if (save) {
    const size_t wb = ttt_linear_weight_ckpt_bytes(&m.d), bb = ttt_linear_bias_ckpt_bytes(&m.d);
    if (wb == 0 || bb == 0) return TTT_ERR_SHAPE;
    o.wck = at::empty({(int64_t)(wb / (64 * 64 * 4)), 64, 64}, m.opt(at::kFloat));
    o.bck = at::empty({(int64_t)bb}, m.opt(at::kByte));
  }
  o.out = at::empty({m.B, m.H, m.T, m.F}, m.opt());
  o.w = at::empty({m.B, m.H, m.F, m.F}, m.opt());
  o.b = at::empty({m.B, m.H, m.F}, m.opt());
  return ttt_linear_forward(&m.d, in.p(0), in.p(1), in.p(2), in.p(3), in.p(4), in.p(5), in.p(6), in.p(7), in.p(8),
                            o.out.data_ptr(), o.w.data_ptr(), o.b.data_ptr(), save ? o.wck.data_ptr() : nullptr,
                            save ? o.bck.data_ptr() : nullptr, m.status.data_ptr(), m.stream());
}

// gradients in the order of the inputs
int linear_backward(const Dims& m, const LinIn& in, const Tensor& wck, const Tensor& bck, const Tensor& go,
                    const Tensor& gw_out, const Tensor& gb_out, const Tensor& packed, Tensor (&g)[9]) {
  c10::cuda::CUDAGuard guard(m.dev);
  const size_t wsb = ttt_linear_backward_workspace_bytes(&m.d);
  if (wsb == 0) return TTT_ERR_SHAPE;
  for (int i = 0; i < 3; ++i) g[i] = at::empty({m.B, m.H, m.T, m.F}, m.opt());
  g[3] = at::empty({m.B, m.H, m.F, m.F}, m.opt());
  g[4] = at::empty({m.B, m.H, m.F}, m.opt());
  g[5] = at::empty({m.T}, m.opt());
  g[6] = at::empty({m.B, m.H, m.T}, m.opt());
  g[7] = at::empty({m.H, m.F}, m.opt());
  g[8] = at::empty({m.H, m.F}, m.opt());
  Tensor ws = at::empty({(int64_t)wsb}, m.opt(at::kByte));
  return ttt_internal_linear_backward(
      &m.d, in.p(0), in.p(1), in.p(2), in.p(3), in.p(4), in.p(5), in.p(6), in.p(7), in.p(8), wck.const_data_ptr(),
      bck.const_data_ptr(), go.const_data_ptr(), gw_out.defined() ? gw_out.const_data_ptr() : nullptr,
      gb_out.defined() ? gb_out.const_data_ptr() : nullptr, g[0].data_ptr(), g[1].data_ptr(), g[2].data_ptr(),
      g[3].data_ptr(), g[4].data_ptr(), g[6].data_ptr(), g[5].data_ptr(), g[7].data_ptr(), g[8].data_ptr(), m.d.dtype,
      packed.defined() ? static_cast<float*>(packed.data_ptr()) : nullptr, ws.data_ptr(), wsb, m.status.data_ptr(),
      m.stream());
}

struct LinearFn : torch::autograd::Function<LinearFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& xq, const Tensor& xk, const Tensor& xv, const Tensor& w,
                               const Tensor& b, const Tensor& te, const Tensor& lr, const Tensor& g, const Tensor& be,
                               int64_t mb, int64_t K, int64_t eps_scaled) {
    LinIn in{{xq, xk, xv, w, b, te, lr, g, be}};
    Dims m;
    LinOut o;
    m.set(xq, xq.size(3), mb, K, eps_scaled);
    const int rc = linear_forward(m, in, true, o);
    if (rc != TTT_OK) throw_error(rc);
    // kept as plain references, without version checks, like the Python node keeps its TttSavedStateMulti
    ctx->saved_data["t"] = std::vector<Tensor>{xq, xk, xv, w, b, te, lr, g, be, o.wck, o.bck};
    ctx->saved_data["c"] = std::vector<int64_t>{mb, K, eps_scaled};
    ctx->mark_non_differentiable({o.w, o.b});
    ctx->set_materialize_grads(false);
    return {o.out, o.w, o.b};
  }
  static variable_list backward(AutogradContext* ctx, variable_list go_) {
    const std::vector<Tensor> t = ctx->saved_data["t"].toTensorVector();
    const std::vector<int64_t> c = ctx->saved_data["c"].toIntVector();
    LinIn in;
    for (int i = 0; i < 9; ++i) in.t[i] = t[i];
    Dims m;
    m.set(t[0], t[0].size(3), c[0], c[1], c[2]);
    const Tensor go = go_[0].defined() ? go_[0].contiguous() : at::zeros_like(t[0]);
    Tensor g[9];
    const int rc = linear_backward(m, in, t[9], t[10], go, Tensor(), Tensor(), Tensor(), g);
    if (rc != TTT_OK) throw_error(rc);
    variable_list r(g, g + 9);
    for (int i = 0; i < 3; ++i) r.emplace_back();
    return r;
  }
};

// ---- TTT-MLP -----------------------------------------------------------------------------------------------------
struct MlpIn {  // xq, xk, xv, w1, b1, w2, b2, token_eta, ttt_lr_eta, ln_weight, ln_bias
  Tensor t[11];
  bool plain(const Dims& m) const {
    const int64_t B = m.B, H = m.H, T = m.T, F = m.F, E = 4 * F;
    if (t[7].dim() != 1 || m.dt != at::kBFloat16) return false;
    return is(t[0], m.dt, m.dev, {B, H, T, F}) && is(t[1], m.dt, m.dev, {B, H, T, F}) &&
           is(t[2], m.dt, m.dev, {B, H, T, F}) && is(t[3], m.dt, m.dev, {B, H, F, E}) && is(t[4], m.dt, m.dev, {B, H, E}) &&
           is(t[5], m.dt, m.dev, {B, H, E, F}) && is(t[6], m.dt, m.dev, {B, H, F}) &&
           is(t[7], m.dt, m.dev, {t[7].size(0)}) && is(t[8], m.dt, m.dev, {B, H, T}) && is(t[9], m.dt, m.dev, {H, F}) &&
           is(t[10], m.dt, m.dev, {H, F});
  }
  const void* p(int i) const { return t[i].const_data_ptr(); }
};
int mlp_forward(const Dims& m, const MlpIn& in, const Tensor& ws, Tensor (&o)[5]) {
  c10::cuda::CUDAGuard guard(m.dev);
  o[0] = at::empty({m.B, m.H, m.T, m.F}, m.opt());
  for (int i = 0; i < 4; ++i) o[1 + i] = at::empty(in.t[3 + i].sizes(), m.opt());
  if (!ws.defined()) {
    size_t bytes = ttt_internal_mlp_infer_scratch_bytes(&m.d);
    Tensor scratch;
    if (bytes != 0) {
      try {
        scratch = at::empty({(int64_t)bytes}, m.opt(at::kByte));
      } catch (const c10::OutOfMemoryError&) {  // whole waves need none
        bytes = 0;
      }
    }
    return ttt_internal_mlp_infer(&m.d, in.p(0), in.p(1), in.p(2), in.p(3), in.p(4), in.p(5), in.p(6), in.p(7), in.p(8),
                                  in.p(9), in.p(10), o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(), o[3].data_ptr(),
                                  o[4].data_ptr(), bytes != 0 ? scratch.data_ptr() : nullptr, bytes, m.status.data_ptr(),
                                  m.stream());
  }
  return ttt_mlp_forward(&m.d, in.p(0), in.p(1), in.p(2), in.p(3), in.p(4), in.p(5), in.p(6), in.p(7), in.p(8), in.p(9),
                         in.p(10), o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(), o[3].data_ptr(), o[4].data_ptr(),
                         ws.data_ptr(), (size_t)ws.numel(), m.status.data_ptr(), m.stream());
}
// gradients in the order of the inputs; `from_forward`: ws was filled by the forward on the same inputs
int mlp_backward(const Dims& m, const MlpIn& in, const Tensor& go, const Tensor& ws, bool from_forward, Tensor (&g)[11]) {
  c10::cuda::CUDAGuard guard(m.dev);
  for (int i = 0; i < 11; ++i) g[i] = at::empty(i == 7 ? c10::IntArrayRef({m.T}) : in.t[i].sizes(), m.opt());
  return ttt_internal_mlp_backward(
      &m.d, in.p(0), in.p(1), in.p(2), in.p(3), in.p(4), in.p(5), in.p(6), in.p(7), in.p(8), in.p(9), in.p(10),
      go.const_data_ptr(), g[0].data_ptr(), g[1].data_ptr(), g[2].data_ptr(), g[3].data_ptr(), g[4].data_ptr(),
      g[5].data_ptr(), g[6].data_ptr(), g[8].data_ptr(), g[7].data_ptr(), g[9].data_ptr(), g[10].data_ptr(), m.d.dtype,
      ws.data_ptr(), (size_t)ws.numel(), from_forward ? 1 : 0, m.status.data_ptr(), m.stream());
}

struct MlpFn : torch::autograd::Function<MlpFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& xq, const Tensor& xk, const Tensor& xv,
                               const Tensor& w1, const Tensor& b1, const Tensor& w2, const Tensor& b2, const Tensor& te,
                               const Tensor& lr, const Tensor& g, const Tensor& be, int64_t mb, int64_t K,
                               int64_t eps_scaled) {
    MlpIn in{{xq, xk, xv, w1, b1, w2, b2, te, lr, g, be}};
    Dims m;
    m.set(xq, xq.size(3), mb, K, eps_scaled);
    const size_t wsb = ttt_mlp_backward_workspace_bytes(&m.d);
    if (wsb == 0) throw_error(TTT_ERR_SHAPE);
    // the forward fills the backward's workspace on the way (final state + the operands of every state update)
    Tensor ws = at::empty({(int64_t)wsb}, m.opt(at::kByte)), o[5];
    const int rc = mlp_forward(m, in, ws, o);
    if (rc != TTT_OK) throw_error(rc);
    ctx->save_for_backward({xq, xk, xv, w1, b1, w2, b2, te, lr, g, be});
    ctx->saved_data["c"] = std::vector<int64_t>{mb, K, eps_scaled};
    ctx->saved_data["ws"] = ws;
    ctx->set_materialize_grads(false);
    return {o[0], o[1], o[2], o[3], o[4]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list go_) {
    const variable_list t = ctx->get_saved_variables();
    const std::vector<int64_t> c = ctx->saved_data["c"].toIntVector();
    MlpIn in;
    for (int i = 0; i < 11; ++i) in.t[i] = t[i];
    Dims m;
    m.set(t[0], t[0].size(3), c[0], c[1], c[2]);
    const Tensor go = go_[0].defined() ? go_[0].contiguous() : at::zeros_like(t[0]);
    // the buffer is consumed by the backward: a second backward walks the sequence forward again
    auto it = ctx->saved_data.find("ws");
    const bool filled = it != ctx->saved_data.end();
    Tensor ws = filled ? it->second.toTensor()
                       : at::empty({(int64_t)ttt_mlp_backward_workspace_bytes(&m.d)}, m.opt(at::kByte));
    if (filled) ctx->saved_data.erase(it);
    Tensor g[11];
    const int rc = mlp_backward(m, in, go, ws, filled, g);
    if (rc != TTT_OK) throw_error(rc);
    variable_list r(g, g + 11);
    for (int i = 0; i < 3; ++i) r.emplace_back();
    return r;
  }
};

// ---- Python functions ----------------------------------------------------------------------------------------------
// tensors args[0..n), false when one is not a tensor
template <int N>
bool tensors(PyObject* const* args, Tensor (&t)[N]) {
  for (int i = 0; i < N; ++i) {
    if (!THPVariable_Check(args[i])) return false;
    t[i] = THPVariable_Unpack(args[i]);
  }
  return true;
}
int64_t as_int(PyObject* o) { return PyLong_AsLongLong(o); }
PyObject* wrap(std::initializer_list<Tensor> ts) {
  PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
  Py_ssize_t i = 0;
  for (const Tensor& t : ts) PyTuple_SET_ITEM(r, i++, THPVariable_Wrap(t));
  return r;
}
PyObject* wrap(const variable_list& ts) {
  PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
  for (size_t i = 0; i < ts.size(); ++i) PyTuple_SET_ITEM(r, (Py_ssize_t)i, THPVariable_Wrap(ts[i]));
  return r;
}
#define NONE_IF(cond) \
  if (cond) Py_RETURN_NONE
bool arity(Py_ssize_t n, Py_ssize_t want) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
  return false;
}

// init(TttError)
PyObject* py_init(PyObject*, PyObject* err) {
  Py_XINCREF(err);
  Py_XSETREF(g_error_type, err);
  Py_RETURN_NONE;
}
// set_status(device index, tensor)
PyObject* py_set_status(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 2)) return nullptr;
  const int64_t i = as_int(args[0]);
  if (i >= 0 && i < kMaxDevices && THPVariable_Check(args[1])) g_status[i] = THPVariable_Unpack(args[1]);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
// linear_forward(9 tensors, mini_batch, head_dim, K, eps_scaled, save) -> (out, w, b, w_ckpt | None, b_ckpt | None) | None
PyObject* py_linear_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 14)) return nullptr;
  LinIn in;
  Dims m;
  NONE_IF(!tensors(args, in.t));
  NONE_IF(!m.set(in.t[0], as_int(args[10]), as_int(args[9]), as_int(args[11]), as_int(args[12])));
  NONE_IF(!m.status.defined() || !in.plain(m));
  LinOut o;
  NONE_IF(linear_forward(m, in, args[13] == Py_True, o) != TTT_OK);
  return wrap({o.out, o.w, o.b, o.wck, o.bck});
  END_HANDLE_TH_ERRORS
}
// linear_partial(9 tensors, mini_batch, head_dim, K, eps_scaled, in_place) -> (out, w, b) | None
PyObject* py_linear_partial(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 14)) return nullptr;
  LinIn in;
  Dims m;
  NONE_IF(!tensors(args, in.t));
  NONE_IF(!m.set(in.t[0], as_int(args[10]), as_int(args[9]), as_int(args[11]), as_int(args[12])) || !in.plain(m));
  c10::cuda::CUDAGuard guard(m.dev);
  const bool in_place = args[13] == Py_True;
  Tensor out = at::empty({m.B, m.H, m.T, m.F}, m.opt());
  Tensor w = in_place ? in.t[3] : at::empty({m.B, m.H, m.F, m.F}, m.opt());
  Tensor b = in_place ? in.t[4] : at::empty({m.B, m.H, m.F}, m.opt());
  NONE_IF(ttt_linear_forward_partial(&m.d, in.p(0), in.p(1), in.p(2), in.p(3), in.p(4), in.p(5), in.p(6), in.p(7),
                                     in.p(8), out.data_ptr(), const_cast<void*>(w.const_data_ptr()),
                                     const_cast<void*>(b.const_data_ptr()), m.stream()) != TTT_OK);
  return wrap({out, w, b});
  END_HANDLE_TH_ERRORS
}
// linear_backward(9 tensors, w_ckpt, b_ckpt, grad_out, mini_batch, head_dim, K, eps_scaled, packed | None,
//                 grad_weight_out | None, grad_bias_out | None) -> 9 gradients | None
PyObject* py_linear_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 19)) return nullptr;
  LinIn in;
  Dims m;
  Tensor c[3], opt[3];
  NONE_IF(!tensors(args, in.t) || !tensors(args + 9, c));
  for (int i = 0; i < 3; ++i)
    if (args[16 + i] != Py_None) {
      NONE_IF(!THPVariable_Check(args[16 + i]));
      opt[i] = THPVariable_Unpack(args[16 + i]);
      NONE_IF(!opt[i].is_contiguous());
    }
  NONE_IF(!m.set(in.t[0], as_int(args[13]), as_int(args[12]), as_int(args[14]), as_int(args[15])));
  NONE_IF(!m.status.defined() || !in.plain(m) || !is(c[2], m.dt, m.dev, {m.B, m.H, m.T, m.F}));
  NONE_IF(!c[0].is_contiguous() || !c[1].is_contiguous() || c[0].device() != m.dev || c[1].device() != m.dev);
  NONE_IF((opt[0].defined() && (opt[0].scalar_type() != at::kFloat || opt[0].device() != m.dev)));
  NONE_IF(opt[1].defined() && !is(opt[1], m.dt, m.dev, {m.B, m.H, m.F, m.F}));
  NONE_IF(opt[2].defined() && !is(opt[2], m.dt, m.dev, {m.B, m.H, m.F}));
  Tensor g[9];
  NONE_IF(linear_backward(m, in, c[0], c[1], c[2], opt[1], opt[2], opt[0], g) != TTT_OK);
  return wrap(variable_list(g, g + 9));
  END_HANDLE_TH_ERRORS
}
// linear_apply(9 tensors, mini_batch, head_dim, K, eps_scaled) -> (out, w, b), recorded for autograd | None
PyObject* py_linear_apply(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 13)) return nullptr;
  LinIn in;
  Dims m;
  NONE_IF(!tensors(args, in.t));
  const int64_t mb = as_int(args[9]), K = as_int(args[11]), eps = as_int(args[12]);
  NONE_IF(!m.set(in.t[0], as_int(args[10]), mb, K, eps));
  NONE_IF(!m.status.defined() || !in.plain(m) || ttt_linear_num_checkpoints(&m.d) < 0);
  Tensor* t = in.t;
  return wrap(LinearFn::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], mb, K, eps));
  END_HANDLE_TH_ERRORS
}
// mlp_forward(11 tensors, mini_batch, head_dim, K, eps_scaled, workspace | None) -> (out, w1, b1, w2, b2) | None
PyObject* py_mlp_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 16)) return nullptr;
  MlpIn in;
  Dims m;
  Tensor ws, o[5];
  NONE_IF(!tensors(args, in.t));
  if (args[15] != Py_None) {
    NONE_IF(!THPVariable_Check(args[15]));
    ws = THPVariable_Unpack(args[15]);
    NONE_IF(ws.scalar_type() != at::kByte || !ws.is_contiguous());
  }
  NONE_IF(!m.set(in.t[0], as_int(args[12]), as_int(args[11]), as_int(args[13]), as_int(args[14])));
  NONE_IF(!m.status.defined() || !in.plain(m) || (ws.defined() && ws.device() != m.dev));
  NONE_IF(mlp_forward(m, in, ws, o) != TTT_OK);
  return wrap({o[0], o[1], o[2], o[3], o[4]});
  END_HANDLE_TH_ERRORS
}
// mlp_apply(11 tensors, mini_batch, head_dim, K, eps_scaled) -> (out, w1, b1, w2, b2), recorded for autograd | None
PyObject* py_mlp_apply(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 15)) return nullptr;
  MlpIn in;
  Dims m;
  NONE_IF(!tensors(args, in.t));
  const int64_t mb = as_int(args[11]), K = as_int(args[13]), eps = as_int(args[14]);
  NONE_IF(!m.set(in.t[0], as_int(args[12]), mb, K, eps));
  NONE_IF(!m.status.defined() || !in.plain(m) || ttt_mlp_backward_workspace_bytes(&m.d) == 0);
  Tensor* t = in.t;
  return wrap(MlpFn::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], t[10], mb, K, eps));
  END_HANDLE_TH_ERRORS
}

// ---- the outer layer, inference ------------------------------------------------------------------------------------
// tensors (None entries allowed) -> 16 bytes each that change with its storage, version, dtype or device
void fill_key(PyObject* const* args, Py_ssize_t n, uint64_t* k) {
  for (Py_ssize_t i = 0; i < n; ++i) {
    k[2 * i] = k[2 * i + 1] = 0;
    if (!THPVariable_Check(args[i])) continue;
    const Tensor& t = THPVariable_Unpack(args[i]);
    k[2 * i] = reinterpret_cast<uint64_t>(t.const_data_ptr());
    k[2 * i + 1] = ((uint64_t)t._version() << 16) | ((uint64_t)t.scalar_type() << 8) | (uint64_t)(uint8_t)t.device().index();
  }
}
// param_key(tensors...) -> their key
PyObject* py_param_key(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  PyObject* r = PyBytes_FromStringAndSize(nullptr, n * 16);
  if (r) fill_key(args, n, reinterpret_cast<uint64_t*>(PyBytes_AS_STRING(r)));
  return r;
  END_HANDLE_TH_ERRORS
}
// stream_key(device index, tensors...) -> the current stream of that device, then their key
PyObject* py_stream_key(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 1) return arity(n, 1), nullptr;
  const int64_t dev = as_int(args[0]);
  if (PyErr_Occurred()) return nullptr;
  const uint64_t st = reinterpret_cast<uint64_t>(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
  PyObject* r = PyBytes_FromStringAndSize(nullptr, 8 + (n - 1) * 16);
  if (!r) return nullptr;
  uint64_t* const k = reinterpret_cast<uint64_t*>(PyBytes_AS_STRING(r));
  k[0] = st;
  fill_key(args + 1, n - 1, k + 1);
  return r;
  END_HANDLE_TH_ERRORS
}

// layer_infer(x, stacked weights, token_idx of one mini-batch, lr_bias, conv q weight / bias, conv k weight / bias (or four
//             None), state weight, state bias, ln weight, ln bias, post norm weight, bias, o_proj, gate 0/1, heads,
//             mini_batch, rope_mode, rope_theta, base_lr, lr_col, eps_scaled, allow_partial, in_place, start_idx,
//             learnable_token_idx)
//   -> (y, state weight, state bias) | None
// One call of TTT.forward without gradients, bf16: projections + prologue, inner loop (whole mini-batches, then the
// remainder as a mini-batch of its own), post norm (+ gate), output projection.
// None comes before the first launch only (what a later launch would refuse is looked at up front): the caller then takes
// another way from the same state.  An error after that is raised.
PyObject* py_layer_infer(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 27)) return nullptr;
  Tensor t[15], te_add;
  for (int i = 0; i < 15; ++i) {
    if (args[i] == Py_None && i >= 4 && i < 8) continue;
    NONE_IF(!THPVariable_Check(args[i]));
    t[i] = THPVariable_Unpack(args[i]);
  }
  NONE_IF(!THPVariable_Check(args[26]));
  te_add = THPVariable_Unpack(args[26]);
  const Tensor &x = t[0], &wcat = t[1], &te_idx = t[2], &lr_bias = t[3], &sw = t[8], &sb = t[9];
  const bool use_gate = as_int(args[15]) != 0, conv = t[4].defined();
  const int64_t H = as_int(args[16]), mb = as_int(args[17]), rope = as_int(args[18]), lr_col = as_int(args[21]);
  const float theta = (float)PyFloat_AsDouble(args[19]), base_lr = (float)PyFloat_AsDouble(args[20]);
  const int64_t eps_scaled = as_int(args[22]), start = as_int(args[25]);
  const bool allow_partial = args[23] == Py_True, in_place = args[24] == Py_True;
  if (PyErr_Occurred()) return nullptr;

  NONE_IF(!x.is_cuda() || x.dim() != 3 || x.scalar_type() != at::kBFloat16 || H <= 0 || mb <= 0);
  const c10::Device dev = x.device();
  const at::ScalarType bf = at::kBFloat16;
  const int64_t B = x.size(0), T = x.size(1), C = x.size(2), F = C / H, M = B * T;
  // rows of x: one pitch for all tokens
  NONE_IF(M <= 0 || F * H != C || (F != 64 && F != 32) || C > 2048 || C % 8 != 0 || x.stride(2) != 1);
  const int64_t x_ld = T > 1 ? x.stride(1) : x.stride(0);
  NONE_IF((T > 1 && B > 1 && x.stride(0) != T * x_ld) || x_ld < C || x_ld % 8 != 0);
  const int64_t N = wcat.size(0);
  NONE_IF(!is(wcat, bf, dev, {N, C}) || te_idx.dim() != 1 || te_idx.size(0) < mb ||
          !is(te_idx, bf, dev, {te_idx.size(0)}) || !is(te_add, bf, dev, {te_idx.size(0)}));
  NONE_IF(lr_bias.numel() != H || lr_bias.scalar_type() != bf || !lr_bias.is_contiguous() || lr_bias.device() != dev);
  NONE_IF(!is(sw, bf, dev, {B, H, F, F}) || !is(sb, bf, dev, {B, H, F}) || !is(t[10], bf, dev, {H, F}) ||
          !is(t[11], bf, dev, {H, F}) || !is(t[12], bf, dev, {C}) || !is(t[13], bf, dev, {C}) || !is(t[14], bf, dev, {C, C}));
  int conv_k = 0;
  if (conv) {
    for (int i = 4; i < 8; ++i)
      NONE_IF(!t[i].defined() || t[i].scalar_type() != bf || !t[i].is_contiguous() || t[i].device() != dev || t[i].size(0) != C);
    conv_k = (int)(t[4].numel() / C);
    NONE_IF(t[5].numel() != C || t[7].numel() != C || t[6].numel() != t[4].numel());
  }
  const int64_t L = T / mb * mb, R = T - L;
  NONE_IF(R > 16 || (R != 0 && !allow_partial));
  NONE_IF(L > 0 && ((mb != 16 && mb != 8) || (F == 32 && H % 2 != 0)));
  for (int i : {0, 1, 14}) NONE_IF(!on_16_bytes(t[i]));
  for (int i : {8, 9, 10, 11}) NONE_IF(L > 0 && !on_16_bytes(t[i]));  // (the remainder's kernel takes any alignment)
  Dims m;
  m.dt = bf;
  m.dev = dev;
  m.status = g_status[dev.index()];
  NONE_IF(!m.status.defined() || M > INT32_MAX || H > 64);
  ttt_dims d{(int32_t)B, (int32_t)H, (int32_t)T, (int32_t)F, (int32_t)mb, 1, (float)eps_scaled * 1e-9f, TTT_BF16};

  c10::cuda::CUDAGuard guard(dev);
  void* const st = m.stream();
  void* const status = m.status.data_ptr();
  const bool small = !conv && ttt_internal_layer_small_fits(&d);  // few-token form of the projections,
  const bool small_out = small && ttt_internal_layer_small_out_fits(&d, use_gate);  // of the output side
  NONE_IF(small_out && (!on_16_bytes(t[12]) || !on_16_bytes(t[13])));
  NONE_IF(!small && N % 8 != 0);
  auto must = [](int rc) {
    if (rc != TTT_OK) throw_error(rc);
  };
  const bool fused = !small && !conv && T % 128 == 0 && F == 64 && rope != 2 && mb <= 16 && lr_col % 64 == 0;
  // temporaries from one allocation, each on a 256-byte boundary
  int64_t at_ = 0;
  auto room = [&](int64_t elements) {
    const int64_t o = at_;
    at_ += (elements * 2 + 255) & ~(int64_t)255;
    return o;
  };
  const int64_t lr_pitch = (T + 7) & ~(int64_t)7;
  const int64_t o_q = room(M * C), o_k = room(M * C), o_v = room(M * C), o_lr = room(B * H * lr_pitch), o_in = room(M * C),
                o_te = room(16);
  const int64_t o_proj = small || fused ? 0 : room(M * N);
  const int64_t o_gate = use_gate && (small || fused) ? room(M * C) : 0;
  const int64_t o_y = small_out ? 0 : room(M * C);
  Tensor tmp = at::empty({at_}, m.opt(at::kByte));
  uint8_t* const base = static_cast<uint8_t*>(tmp.data_ptr());
  Tensor y = at::empty({B, T, C}, m.opt());
  const void* const idx = te_idx.const_data_ptr();
  const void* const learnable = te_add.const_data_ptr();
  void* const te = base + o_te;
  const uint8_t* gate = nullptr;
  int64_t gate_ld = C;
  const int64_t g_col = lr_col - C;
  // ---- projections, head split, rotary embedding, learning rates, token_eta
  if (small) {
    NONE_IF(ttt_internal_layer_small_proj(&d, x.const_data_ptr(), x_ld, wcat.const_data_ptr(), C, (int)N, (int)lr_col,
                                          lr_bias.const_data_ptr(), (int)start, (int)rope, theta, base_lr, idx, learnable, te,
                                          base + o_q, base + o_k, base + o_v, use_gate ? base + o_gate : nullptr, base + o_lr,
                                          (int)lr_pitch, st) != TTT_OK);
    if (use_gate) gate = base + o_gate;
  } else if (fused) {
    NONE_IF(ttt_internal_layer_projections(&d, x.const_data_ptr(), x_ld, C, wcat.const_data_ptr(), C, N, 0, C, 2 * C,
                                           use_gate ? g_col : -1, lr_col, lr_bias.const_data_ptr(), (int)start,
                                           (int)rope, theta, base_lr, 0, idx, learnable, te, base + o_q, base + o_k,
                                           base + o_v, use_gate ? base + o_gate : nullptr, base + o_lr, status,
                                           st) != TTT_OK);
    if (use_gate) gate = base + o_gate;
  } else {
    uint8_t* const proj = base + o_proj;
    NONE_IF(ttt_gemm_bf16_tn(M, N, C, x.const_data_ptr(), x_ld, wcat.const_data_ptr(), C, proj, N, status, st) != TTT_OK);
    const int64_t k_col = conv ? 0 : C, v_col = conv ? C : 2 * C;
    must(ttt_internal_layer_prologue(&d, proj, proj + 2 * k_col, proj + 2 * v_col, N, proj + 2 * lr_col, N,
                                     lr_bias.const_data_ptr(), conv ? t[4].const_data_ptr() : nullptr,
                                     conv ? t[5].const_data_ptr() : nullptr, conv ? t[6].const_data_ptr() : nullptr,
                                     conv ? t[7].const_data_ptr() : nullptr, conv_k, (int)start, (int)rope, theta,
                                     base_lr, idx, learnable, te, base + o_q, base + o_k, base + o_v, base + o_lr,
                                     (int)lr_pitch, st));
    if (use_gate) gate = proj + 2 * g_col, gate_ld = N;
  }
  // ---- inner loop
  Tensor w = sw, b = sb;
  if (L > 0) {
    w = at::empty({B, H, F, F}, m.opt());
    b = at::empty({B, H, F}, m.opt());
    ttt_dims di = d;
    di.seq_len = (int32_t)L;
    must(ttt_internal_linear_infer(&di, (int)T, (int)lr_pitch, base + o_q, base + o_k, base + o_v,
                                   sw.const_data_ptr(), sb.const_data_ptr(), te, base + o_lr,
                                   t[10].const_data_ptr(), t[11].const_data_ptr(), base + o_in, w.data_ptr(),
                                   b.data_ptr(), status, st));
  }
  if (R > 0) {
    const Tensor w_in = w, b_in = b;
    if (L == 0 && !in_place) {
      w = at::empty({B, H, F, F}, m.opt());
      b = at::empty({B, H, F}, m.opt());
    }
    ttt_dims dt = d;
    dt.seq_len = (int32_t)R;
    must(ttt_internal_linear_tail(&dt, (int)T, (int)L, (int)lr_pitch, small && L == 0, base + o_q, base + o_k, base + o_v,
                                  w_in.const_data_ptr(), b_in.const_data_ptr(), te, base + o_lr,
                                  t[10].const_data_ptr(), t[11].const_data_ptr(), base + o_in,
                                  const_cast<void*>(w.const_data_ptr()), const_cast<void*>(b.const_data_ptr()),
                                  st));
  }
  // ---- post norm, gate, output projection
  if (small_out) {
    must(ttt_internal_layer_small_out(&d, base + o_in, gate, (int)gate_ld, t[12].const_data_ptr(),
                                      t[13].const_data_ptr(), 1e-6f, t[14].const_data_ptr(), C, y.data_ptr(), st));
  } else {
    must(ttt_layer_epilogue(&d, base + o_in, gate, gate != nullptr ? gate_ld : 0, t[12].const_data_ptr(),
                            t[13].const_data_ptr(), 1e-6f, base + o_y, st));
    must(ttt_gemm_bf16_tn(M, C, C, base + o_y, C, t[14].const_data_ptr(), C, y.data_ptr(), C, status, st));
  }
  return wrap({y, w, b});
  END_HANDLE_TH_ERRORS
}

// ---- the outer layer, training -----------------------------------------------------------------------------------------
// The whole layer as one node of the graph, for the lengths whose projections are a product of their own: the steps of the
// Python composition (a node per step: its interpreter time is most of a training step of a few thousand tokens) with the
// same kernels and roundings, forward and backward.  The projections' gradients, the gate's among them, are the columns of one
// buffer, so the weights' and the input's are one product each.  5 x 192 tokens of 768 features, forward + backward: 1148 us
// through the composition, 528 here.
struct LayerDims {
  ttt_dims d;
  int64_t B, T, C, H, F, mb, M;
  int64_t v, lr, N0, g, N;  // columns q | k | v | lr (and padding) up to N0 | gate from g (-1: none) up to N
  int64_t taps;             // shared q / k projection (v = C then): taps of its two convolutions; 0: projections of their own
  int64_t K, rope, start, eps_scaled;
  float theta, base_lr;
};
struct LayerFn : torch::autograd::Function<LayerFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& q, const Tensor& k, const Tensor& v,
                               const Tensor& g, const Tensor& lrw, const Tensor& lrb, const Tensor& learnable,
                               const Tensor& post_w, const Tensor& post_b, const Tensor& o, const Tensor& w0,
                               const Tensor& b0, const Tensor& ln_w, const Tensor& ln_b, const Tensor& cqw, const Tensor& cqb,
                               const Tensor& ckw, const Tensor& ckb, const Tensor& idx, const LayerDims& l) {
    Dims m;
    m.d = l.d;
    m.B = l.B, m.H = l.H, m.T = l.T, m.F = l.F;
    m.dt = x.scalar_type();
    m.dev = x.device();
    m.status = g_status[m.dev.index()];
    c10::cuda::CUDAGuard guard(m.dev);
    void* const st = m.stream();
    auto must = [](int rc) {
      if (rc != TTT_OK) throw_error(rc);
    };
    const bool gated = l.g >= 0, bf = m.dt == at::kBFloat16;
    const Tensor x2 = x.reshape({l.M, l.C}).contiguous();
    const Tensor lr2 = lrw.reshape({l.H, l.C});  // weights stacked in the order of the columns
    std::vector<Tensor> rows{q};
    if (!l.taps) rows.push_back(k);
    rows.push_back(v);
    rows.push_back(lr2);
    if (l.N0 > l.lr + l.H) rows.push_back(at::zeros({l.N0 - l.lr - l.H, l.C}, m.opt()));
    if (gated) rows.push_back(g);
    const Tensor wcat = at::cat(rows, 0);
    const Tensor te = at::add(idx, learnable);
    // token_eta of one mini-batch, which is all that is read of it: by the projections' kernel, or here in float32
    Tensor te16 = bf ? at::empty({16}, m.opt()) : at::clamp_min(te, 0.0);
    Tensor s[4];
    for (int i = 0; i < 3; ++i) s[i] = at::empty({l.B, l.H, l.T, l.F}, m.opt());
    s[3] = at::empty({l.B, l.H, l.T}, m.opt());
    const void* const ip = bf ? idx.const_data_ptr() : nullptr;
    const void* const lp = bf ? learnable.const_data_ptr() : nullptr;
    Tensor gate, proj = at::mm(x2, wcat.narrow(0, 0, l.N0).t());
    {
      const uint8_t* const p = static_cast<const uint8_t*>(proj.const_data_ptr());
      const int64_t e = proj.element_size();
      const bool cv = l.taps != 0;
      must(ttt_internal_layer_prologue(&l.d, p, p + (cv ? 0 : e * l.C), p + e * l.v, l.N0, p + e * l.lr, l.N0, lrb.const_data_ptr(),
                                       cv ? cqw.const_data_ptr() : nullptr, cv ? cqb.const_data_ptr() : nullptr,
                                       cv ? ckw.const_data_ptr() : nullptr, cv ? ckb.const_data_ptr() : nullptr, (int)l.taps,
                                       (int)l.start, (int)l.rope, l.theta, l.base_lr, ip, lp, bf ? te16.data_ptr() : nullptr,
                                       s[0].data_ptr(), s[1].data_ptr(), s[2].data_ptr(), s[3].data_ptr(), (int)l.T, st));
    }
    if (!l.taps) proj = Tensor();  // (the convolutions' gradient reads it)
    if (gated) gate = at::mm(x2, wcat.narrow(0, l.g, l.C).t());
    LinIn in{{s[0], s[1], s[2], w0, b0, te16, s[3], ln_w, ln_b}};
    LinOut lo;
    must(linear_forward(m, in, true, lo));
    const Tensor y = at::empty({l.M, l.C}, m.opt());
    must(ttt_layer_epilogue(&l.d, lo.out.const_data_ptr(), gated ? gate.const_data_ptr() : nullptr, gated ? l.C : 0,
                            post_w.const_data_ptr(), post_b.const_data_ptr(), 1e-6f, y.data_ptr(), st));
    const Tensor out = at::mm(y, o.t()).view({l.B, l.T, l.C});
    ctx->save_for_backward({x, wcat, te, lo.out, gate, post_w, post_b, y, o, proj, cqw, ckw});
    // kept as plain references, as the inner loop's own node keeps what it saves
    ctx->saved_data["t"] = std::vector<Tensor>{s[0], s[1], s[2], w0, b0, te16, s[3], ln_w, ln_b, lo.wck, lo.bck};
    ctx->saved_data["l"] = c10::IValue(std::string(reinterpret_cast<const char*>(&l), sizeof(l)));
    ctx->saved_data["s"] = std::vector<std::vector<int64_t>>{lrw.sizes().vec(), lrb.sizes().vec()};
    ctx->mark_non_differentiable({lo.w, lo.b});
    ctx->set_materialize_grads(false);
    return {out, lo.w, lo.b};
  }
  static variable_list backward(AutogradContext* ctx, variable_list go_) {
    const variable_list sv = ctx->get_saved_variables();
    const Tensor &x = sv[0], &wcat = sv[1], &te = sv[2], &inner_out = sv[3], &gate = sv[4], &post_w = sv[5], &post_b = sv[6],
                 &y = sv[7], &o = sv[8];
    const std::vector<Tensor> t = ctx->saved_data["t"].toTensorVector();
    LayerDims l;
    memcpy(&l, ctx->saved_data["l"].toStringRef().data(), sizeof(l));
    const auto shapes = ctx->saved_data["s"].toList();
    Dims m;
    m.d = l.d;
    m.B = l.B, m.H = l.H, m.T = l.T, m.F = l.F;
    m.dt = x.scalar_type();
    m.dev = x.device();
    m.status = g_status[m.dev.index()];
    c10::cuda::CUDAGuard guard(m.dev);
    void* const st = m.stream();
    auto must = [](int rc) {
      if (rc != TTT_OK) throw_error(rc);
    };
    const Tensor go = (go_[0].defined() ? go_[0] : at::zeros_like(x)).reshape({l.M, l.C}).contiguous();
    variable_list r(21);  // x q k v g lrw lrb learnable post_w post_b o w0 b0 ln_w ln_b, four of the convolutions, idx dims
    if (ctx->needs_input_grad(10)) r[10] = at::mm(go.t(), y);
    const Tensor dy = at::mm(go, o);
    // post norm and gate: the gate's gradient goes to its columns of the projections' gradient
    const Tensor dproj = at::empty({l.M, l.N}, m.opt());
    uint8_t* const dp = static_cast<uint8_t*>(dproj.data_ptr());
    const int64_t e = dproj.element_size();
    const bool gated = gate.defined();
    const Tensor d_inner = at::empty({l.B, l.H, l.T, l.F}, m.opt()), dn = at::empty({2, l.C}, m.opt(at::kFloat));
    {
      const size_t wsb = ttt_layer_epilogue_backward_workspace_bytes(&l.d);
      const Tensor ws = at::empty({(int64_t)wsb}, m.opt(at::kByte));
      must(ttt_layer_epilogue_backward(&l.d, dy.const_data_ptr(), inner_out.const_data_ptr(), gated ? gate.const_data_ptr() : nullptr,
                                       gated ? l.C : 0, post_w.const_data_ptr(), post_b.const_data_ptr(), 1e-6f, d_inner.data_ptr(),
                                       gated ? dp + e * l.g : nullptr, gated ? l.N : 0, static_cast<float*>(dn.data_ptr()),
                                       static_cast<float*>(dn.data_ptr()) + l.C, ws.data_ptr(), wsb, st));
    }
    const Tensor dnt = m.dt == at::kFloat ? dn : dn.to(m.dt);
    r[8] = dnt.select(0, 0);
    r[9] = dnt.select(0, 1);
    LinIn in;
    for (int i = 0; i < 9; ++i) in.t[i] = t[i];
    Tensor gr[9];
    must(linear_backward(m, in, t[9], t[10], d_inner, Tensor(), Tensor(), Tensor(), gr));
    r[11] = gr[3];
    r[12] = gr[4];
    r[13] = gr[7];
    r[14] = gr[8];
    auto prologue_backward = [&](void* dq, void* dk, void* dv, int64_t ld) {
      must(ttt_layer_prologue_backward(&l.d, gr[0].const_data_ptr(), gr[1].const_data_ptr(), gr[2].const_data_ptr(),
                                       gr[6].const_data_ptr(), t[6].const_data_ptr(), (int)l.start, (int)l.rope, l.theta, l.base_lr,
                                       dq, dk, dv, ld, dp + e * l.lr, l.N, (int)(l.N0 - l.lr), st));
    };
    if (!l.taps) {
      prologue_backward(dp, dp + e * l.C, dp + e * l.v, l.N);
    } else {
      // through the two convolutions to their shared projection
      const Tensor &proj = sv[9], d4 = at::empty({4, l.M, l.C}, m.opt());  // of q, k, v, and of the shared projection
      uint8_t* const d0 = static_cast<uint8_t*>(d4.data_ptr());
      const int64_t one = e * l.M * l.C;
      prologue_backward(d0, d0 + one, d0 + 2 * one, l.C);
      const Tensor gp = at::empty({2, 5, l.C}, m.opt(at::kFloat));  // four taps and the bias, of each
      auto taps4 = [&](const Tensor& w) {  // [C][4], aligned to the end
        const Tensor w2 = w.reshape({l.C, l.taps});
        if (l.taps == 4) return w2;
        Tensor w4 = at::zeros({l.C, 4}, w2.options());
        w4.narrow(1, 4 - l.taps, l.taps).copy_(w2);
        return w4;
      };
      const Tensor wq4 = taps4(sv[10]), wk4 = taps4(sv[11]);
      const size_t wsb = ttt_layer_qk_conv_backward_workspace_bytes(&l.d);
      const Tensor ws = at::empty({(int64_t)wsb}, m.opt(at::kByte));
      must(ttt_layer_qk_conv_backward(&l.d, d0, d0 + one, proj.const_data_ptr(), l.N0, wq4.const_data_ptr(), wk4.const_data_ptr(),
                                      d0 + 3 * one, static_cast<float*>(gp.data_ptr()), static_cast<float*>(gp.data_ptr()) + 5 * l.C,
                                      ws.data_ptr(), wsb, st));
      dproj.narrow(1, 0, l.C).copy_(d4.select(0, 3));
      dproj.narrow(1, l.v, l.C).copy_(d4.select(0, 2));
      const Tensor gpt = gp.to(m.dt);
      for (int i = 0; i < 2; ++i) {
        r[15 + 2 * i] = gpt.select(0, i).narrow(0, 4 - l.taps, l.taps).t().reshape(sv[10 + i].sizes());
        r[16 + 2 * i] = gpt.select(0, i).select(0, 4);
      }
    }
    if (ctx->needs_input_grad(0)) r[0] = at::mm(dproj, wcat).view(x.sizes());
    bool weights = false;
    for (int i = 1; i <= 5; ++i) weights = weights || ctx->needs_input_grad(i);
    if (weights) {
      const Tensor dw = at::mm(dproj.t(), x.reshape({l.M, l.C}));
      r[1] = dw.narrow(0, 0, l.C);
      if (!l.taps) r[2] = dw.narrow(0, l.C, l.C);
      r[3] = dw.narrow(0, l.v, l.C);
      if (gated) r[4] = dw.narrow(0, l.g, l.C);
      r[5] = dw.narrow(0, l.lr, l.H).view(shapes.get(0).toIntVector());
    }
    if (ctx->needs_input_grad(6))
      r[6] = at::sum(dproj.narrow(1, l.lr, l.H), {0}, false, at::kFloat).to(m.dt).view(shapes.get(1).toIntVector());
    if (ctx->needs_input_grad(7)) {
      const Tensor sum = at::sum(gr[5].view({l.T / l.mb, l.mb}), {0}, false, m.dt);
      r[7] = at::where(at::ge(te, 0), sum, at::zeros({}, sum.options()));
    }
    return r;
  }
};
// layer_train(x, q_proj, k_proj | None, v_proj, g_proj | None, lr weight, lr bias, learnable_token_idx, post norm weight, bias,
//             o_proj, state weight, state bias, ln weight, ln bias, conv q weight, bias, conv k weight, bias (with k_proj: four
//             None), token_idx, heads, mini_batch, rope_mode, rope_theta, base_lr,
//             checkpoint interval, eps_scaled, start_idx) -> (y, state weight, state bias), recorded for autograd | None
PyObject* py_layer_train(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 28)) return nullptr;
  Tensor t[20];
  const bool shared = args[2] == Py_None;
  for (int i = 0; i < 20; ++i) {
    if (args[i] == Py_None && (i == 4 || (shared ? i == 2 : i >= 15 && i < 19))) continue;
    NONE_IF(!THPVariable_Check(args[i]));
    t[i] = THPVariable_Unpack(args[i]);
    NONE_IF(t[i].unsafeGetTensorImpl()->is_python_dispatch());
  }
  LayerDims l;
  l.H = as_int(args[20]), l.mb = as_int(args[21]), l.rope = as_int(args[22]);
  l.theta = (float)PyFloat_AsDouble(args[23]), l.base_lr = (float)PyFloat_AsDouble(args[24]);
  l.K = as_int(args[25]), l.eps_scaled = as_int(args[26]), l.start = as_int(args[27]);
  if (PyErr_Occurred()) return nullptr;
  const Tensor& x = t[0];
  NONE_IF(at::autocast::is_autocast_enabled(at::kCUDA));
  NONE_IF(!x.is_cuda() || x.layout() != c10::kStrided || x.dim() != 3 || l.H <= 0 || l.mb <= 0);
  const c10::Device dev = x.device();
  const at::ScalarType dt = x.scalar_type();
  NONE_IF((dt != at::kBFloat16 && dt != at::kFloat) || dev.index() >= kMaxDevices || !g_status[dev.index()].defined());
  l.B = x.size(0), l.T = x.size(1), l.C = x.size(2), l.F = l.C / l.H, l.M = l.B * l.T;
  NONE_IF(l.M <= 0 || l.M > INT32_MAX || l.F * l.H != l.C || (l.F != 64 && l.F != 32) || l.C > 2048 || l.H > 64 || l.C % 8 != 0);
  NONE_IF((l.mb != 16 && l.mb != 8) || l.T % l.mb != 0 || (l.F == 32 && l.H % 2 != 0));
  for (int i : {1, 2, 3, 10}) NONE_IF(t[i].defined() && !is(t[i], dt, dev, {l.C, l.C}));
  const bool gated = t[4].defined();
  NONE_IF(gated && !is(t[4], dt, dev, {l.C, l.C}));
  NONE_IF(t[5].numel() != l.H * l.C || t[5].size(0) != l.H || t[5].scalar_type() != dt || t[5].device() != dev || !t[5].is_contiguous());
  NONE_IF(t[6].numel() != l.H || t[6].scalar_type() != dt || t[6].device() != dev || !t[6].is_contiguous());
  for (int i : {7, 19}) NONE_IF(!is(t[i], dt, dev, {l.mb}));
  for (int i : {8, 9}) NONE_IF(!is(t[i], dt, dev, {l.C}));
  NONE_IF(!is(t[11], dt, dev, {l.B, l.H, l.F, l.F}) || !is(t[12], dt, dev, {l.B, l.H, l.F}));
  for (int i : {13, 14}) NONE_IF(!is(t[i], dt, dev, {l.H, l.F}));
  l.taps = 0;
  if (shared) {
    for (int i = 15; i < 19; ++i)
      NONE_IF(t[i].dim() < 1 || t[i].size(0) != l.C || t[i].scalar_type() != dt || t[i].device() != dev || !t[i].is_contiguous());
    l.taps = t[15].numel() / l.C;
    NONE_IF(l.taps < 1 || l.taps > 4 || t[17].numel() != t[15].numel() || t[16].numel() != l.C || t[18].numel() != l.C);
  }
  for (int i = 0; i < 20; ++i) NONE_IF(t[i].defined() && !on_16_bytes(t[i]));
  // (those run projections and prologue in one launch: the composition)
  NONE_IF(!shared && dt == at::kBFloat16 && l.T % 128 == 0 && l.F == 64 && l.rope != 2);
  l.v = shared ? l.C : 2 * l.C;
  l.lr = l.v + l.C;
  l.N0 = (l.lr + l.H + 7) & ~(int64_t)7;
  l.g = gated ? l.N0 : -1;
  l.N = l.N0 + (gated ? l.C : 0);
  l.d = ttt_dims{(int32_t)l.B, (int32_t)l.H, (int32_t)l.T, (int32_t)l.F, (int32_t)l.mb, (int32_t)l.K, (float)l.eps_scaled * 1e-9f,
                 dt == at::kBFloat16 ? TTT_BF16 : TTT_F32};
  NONE_IF(ttt_linear_num_checkpoints(&l.d) < 0);
  for (Tensor& u : t)
    if (!u.defined()) u = at::empty({0});  // (a node's arguments are defined tensors)
  return wrap(LayerFn::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], t[10], t[11], t[12], t[13], t[14], t[15],
                             t[16], t[17], t[18], t[19], l));
  END_HANDLE_TH_ERRORS
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"init", py_init, METH_O, nullptr},
                         FAST(set_status),
                         FAST(linear_forward),
                         FAST(linear_partial),
                         FAST(linear_backward),
                         FAST(linear_apply),
                         FAST(mlp_forward),
                         FAST(mlp_apply),
                         FAST(param_key),
                         FAST(stream_key),
                         FAST(layer_infer),
                         FAST(layer_train),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
