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
  return ttt_mlp_forward(&m.d, in.p(0), in.p(1), in.p(2), in.p(3), in.p(4), in.p(5), in.p(6), in.p(7), in.p(8), in.p(9),
                         in.p(10), o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(), o[3].data_ptr(), o[4].data_ptr(),
                         ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? (size_t)ws.numel() : 0,
                         m.status.data_ptr(), m.stream());
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
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
