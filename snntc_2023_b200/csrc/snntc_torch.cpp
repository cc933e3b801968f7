// Host path of the Python operators as a CPython extension (module snntc_2023_b200._native): argument checks, output
// and workspace tensors, the autograd nodes and the C-ABI call of every operator in one native call.
//
// What bounds it: a call on a small problem is a few kernels of some microseconds each, and the same steps written in
// Python (tensor checks, numpy parameter vectors, a device context manager, torch.empty, a ctypes call with fifteen
// arguments, a Python autograd.Function) cost 35 to 50 us per operator and direction -- more than its kernels. Nothing
// is computed here and nothing is kept between calls; the kernels are reached through the C ABI of libsnntc_b200.so.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/engine.h>
#include <torch/csrc/autograd/functions/accumulate_grad.h>
#include <torch/csrc/autograd/graph_task.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "../../include/snntc_b200.h"

namespace py = pybind11;

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

py::handle g_error_class;    // snntc_2023_b200._lib.SnntcError, set once at import and kept alive by its module
py::handle g_params_fn;      // snntc_2023_b200.ops._params: parameter vectors that are no plain float32 array

struct SnntcFailure : std::runtime_error {
  using std::runtime_error::runtime_error;
};

void check(int rc, const char* what) {
  if (rc == SNNTC_OK) return;
  std::string msg = std::string(what) + ": " + snntc_status_string(rc);
  if (rc == SNNTC_E_CUDA) throw SnntcFailure(msg + " (" + snntc_last_cuda_error() + ")");
  TORCH_CHECK_VALUE(!(rc == SNNTC_E_NULL || rc == SNNTC_E_SHAPE || rc == SNNTC_E_WEIGHT_ROWS ||
                      rc == SNNTC_E_TOO_LARGE || rc == SNNTC_E_PARAMS), msg);
  throw SnntcFailure(msg);
}

Tensor as_cuda_f32(const Tensor& t, const char* name) {
  if (!t.is_cuda())
    throw SnntcFailure(std::string(name) + " is not on a CUDA device: the SNN-TC operators have no CPU implementation");
  TORCH_CHECK_VALUE(t.scalar_type() == at::kFloat, name, " must be float32 (the operators are fp32 only), got ",
                    t.scalar_type());
  return t.contiguous();
}

void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

Tensor empty_like_dev(at::IntArrayRef shape, const Tensor& t) { return at::empty(shape, t.options().requires_grad(false)); }

Tensor workspace(size_t bytes, const Tensor& t) {
  return at::empty({(int64_t)bytes}, t.options().dtype(at::kByte).requires_grad(false));
}

float* ptr(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }

int to_int(int64_t v, const char* what) {
  TORCH_CHECK_VALUE(v >= 0 && v <= INT_MAX, what, ": too many elements in a tensor (limit 2^31-1)");
  return (int)v;
}

// The params vector of an operator (6 or 12 floats on the host). The usual one is the layer's float32 numpy array.
struct Params {
  float v[12];
  int n;
};
Params read_params(py::handle obj, int n) {
  Params p;
  p.n = n;
  Py_buffer b;
  if (PyObject_CheckBuffer(obj.ptr()) && PyObject_GetBuffer(obj.ptr(), &b, PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) == 0) {
    const bool plain = b.itemsize == 4 && b.format && b.format[0] == 'f' && b.format[1] == 0 && b.len == 4 * n;
    if (plain) std::memcpy(p.v, b.buf, 4 * n);
    PyBuffer_Release(&b);
    if (plain) return p;
  }
  PyErr_Clear();
  const py::object arr = g_params_fn(obj, n);   // raises ValueError where the length is wrong
  const py::buffer_info info = py::reinterpret_borrow<py::buffer>(arr).request();
  std::memcpy(p.v, info.ptr, 4 * n);
  return p;
}

// ------------------------------------------------------------------------------------------------ dense
Tensor fc_forward_call(const Tensor& X, const Tensor& W, const Params& p, bool infer) {
  const Tensor x = as_cuda_f32(X, "in"), w = as_cuda_f32(W, "weight");
  TORCH_CHECK_VALUE(x.dim() == 2 && w.dim() == 2, "snn_fc expects in[B,I] and weight[rows,J]");
  const int B = to_int(x.size(0), "SnnFc"), I = to_int(x.size(1), "SnnFc");
  const int rows = to_int(w.size(0), "SnnFc"), J = to_int(w.size(1), "SnnFc");
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor out = empty_like_dev({infer ? (int64_t)B : 2 * (int64_t)B, (int64_t)J}, x);
  const size_t bytes = snntc_fc_forward_workspace_bytes(B, I, J);
  const Tensor ws = workspace(bytes, x);
  const int rc = infer ? snntc_fc_infer(ptr(x), ptr(w), p.v, ptr(out), nullptr, B, I, rows, J, ws.data_ptr(), bytes, stream_of(x))
                       : snntc_fc_forward(ptr(x), ptr(w), p.v, ptr(out), B, I, rows, J, ws.data_ptr(), bytes, stream_of(x));
  check(rc, infer ? "SnnFc (inference)" : "SnnFc");
  return out;
}

// dx (undefined when not wanted) and dw; `sink`, where defined, receives dw
std::pair<Tensor, Tensor> fc_grad_call(const Tensor& G, const Tensor& X, const Tensor& W, const Params& p, const Tensor& out,
                                       bool need_dx, const Tensor& sink, const Tensor& dparams) {
  const Tensor g = as_cuda_f32(G, "grad"), x = as_cuda_f32(X, "in"), w = as_cuda_f32(W, "weight"), y = as_cuda_f32(out, "oldout");
  TORCH_CHECK_VALUE(x.dim() == 2 && w.dim() == 2, "snn_fc_grad expects in[B,I] and weight[rows,J]");
  const int B = to_int(x.size(0), "SnnFcGrad"), I = to_int(x.size(1), "SnnFcGrad");
  const int rows = to_int(w.size(0), "SnnFcGrad"), J = to_int(w.size(1), "SnnFcGrad");
  TORCH_CHECK_VALUE(y.dim() == 2 && y.size(0) == 2 * (int64_t)B && y.size(1) == J, "snn_fc_grad: oldout must be [2B,J]");
  TORCH_CHECK_VALUE(g.dim() == 2 && (g.size(0) == B || g.size(0) == 2 * (int64_t)B) && g.size(1) == J,
                    "snn_fc_grad: Grad/Oldout batch should be 2 * batch");
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor dx = need_dx ? at::empty_like(x) : Tensor();
  const Tensor dw = sink.defined() ? sink : at::empty_like(w);
  const size_t bytes = snntc_fc_backward_workspace_bytes(B, I, rows, J);
  const Tensor ws = workspace(bytes, x);
  check(snntc_fc_backward(ptr(g), ptr(x), ptr(w), p.v, ptr(y), ptr(dx), ptr(dw), ptr(dparams), B, I, rows, J, ws.data_ptr(),
                          bytes, stream_of(x)), "SnnFcGrad");
  return {dx, dw};
}

// ------------------------------------------------------------------------------------------------ convolution
struct ConvGeom {
  int pt, pl;
  int64_t Nh, Nw;   // Nh < 0: the reference's convention, a pre-padded input and its output size from the params vector
};

Tensor cv_forward_call(const Tensor& X, const Tensor& W, const Params& p, ConvGeom q, bool infer) {
  const Tensor x = as_cuda_f32(X, "in"), w = as_cuda_f32(W, "weight");
  TORCH_CHECK_VALUE(x.dim() == 4 && w.dim() == 2, "snn_cv expects in[B,H,W,C] (NHWC) and weight[rows,Kc]");
  const int B = to_int(x.size(0), "SnnCv"), H = to_int(x.size(1), "SnnCv"), Wd = to_int(x.size(2), "SnnCv"), C = to_int(x.size(3), "SnnCv");
  const int rows = to_int(w.size(0), "SnnCv"), J = to_int(w.size(1), "SnnCv");
  const int Kh = (int)p.v[6], Kw = (int)p.v[7], Sh = (int)p.v[8], Sw = (int)p.v[9];
  if (q.Nh < 0) {
    TORCH_CHECK_VALUE(Kh > 0 && Kw > 0 && Sh > 0 && Sw > 0, "snn_cv: invalid params vector");
    q.Nh = H >= Kh ? (H - Kh) / Sh + 1 : 0;
    q.Nw = Wd >= Kw ? (Wd - Kw) / Sw + 1 : 0;
  }
  TORCH_CHECK_VALUE(q.Nh > 0 && q.Nw > 0, "snn_cv: kernel larger than the (padded) input");
  const int Nh = to_int(q.Nh, "SnnCv"), Nw = to_int(q.Nw, "SnnCv");
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor out = empty_like_dev({infer ? (int64_t)B : 2 * (int64_t)B, q.Nh, q.Nw, (int64_t)J}, x);
  const size_t bytes = snntc_cv_forward_workspace_bytes(B, H, Wd, C, J, Kh, Kw, Nh, Nw);
  const Tensor ws = workspace(bytes, x);
  const int rc = infer ? snntc_cv_infer(ptr(x), ptr(w), p.v, ptr(out), nullptr, B, H, Wd, C, rows, J, q.pt, q.pl, Nh, Nw,
                                        ws.data_ptr(), bytes, stream_of(x))
                       : snntc_cv_forward(ptr(x), ptr(w), p.v, ptr(out), B, H, Wd, C, rows, J, q.pt, q.pl, Nh, Nw,
                                          ws.data_ptr(), bytes, stream_of(x));
  check(rc, infer ? "SnnCv (inference)" : "SnnCv");
  return out;
}

std::pair<Tensor, Tensor> cv_grad_call(const Tensor& G, const Tensor& X, const Tensor& W, const Params& p, const Tensor& out,
                                       int pt, int pl, bool need_dx, const Tensor& sink, const Tensor& dparams) {
  const Tensor g = as_cuda_f32(G, "grad"), x = as_cuda_f32(X, "in"), w = as_cuda_f32(W, "weight"), y = as_cuda_f32(out, "oldout");
  TORCH_CHECK_VALUE(y.dim() == 4, "snn_cv_grad: oldout must be [2B,Nh,Nw,Kc]");
  TORCH_CHECK_VALUE(x.dim() == 4 && w.dim() == 2, "snn_cv expects in[B,H,W,C] (NHWC) and weight[rows,Kc]");
  const int B = to_int(x.size(0), "SnnCvGrad"), H = to_int(x.size(1), "SnnCvGrad"), Wd = to_int(x.size(2), "SnnCvGrad"), C = to_int(x.size(3), "SnnCvGrad");
  const int rows = to_int(w.size(0), "SnnCvGrad"), J = to_int(w.size(1), "SnnCvGrad");
  const int Nh = to_int(y.size(1), "SnnCvGrad"), Nw = to_int(y.size(2), "SnnCvGrad");
  TORCH_CHECK_VALUE(y.size(0) == 2 * (int64_t)B && y.size(3) == J, "snn_cv_grad: oldout must be [2B,Nh,Nw,Kc]");
  TORCH_CHECK_VALUE(g.dim() == 4 && (g.size(0) == B || g.size(0) == 2 * (int64_t)B) && g.size(1) == Nh && g.size(2) == Nw &&
                    g.size(3) == J, "snn_cv_grad: Grad/Oldout batch should be 2 * batch");
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor dx = need_dx ? at::empty_like(x) : Tensor();
  const Tensor dw = sink.defined() ? sink : at::empty_like(w);
  const size_t bytes = snntc_cv_backward_workspace_bytes(B, H, Wd, C, rows, J, Nh, Nw);
  const Tensor ws = workspace(bytes, x);
  check(snntc_cv_backward(ptr(g), ptr(x), ptr(w), p.v, ptr(y), ptr(dx), ptr(dw), ptr(dparams), B, H, Wd, C, rows, J, pt, pl,
                          Nh, Nw, ws.data_ptr(), bytes, stream_of(x)), "SnnCvGrad");
  return {dx, dw};
}

// ------------------------------------------------------------------------------------------------ autograd
// What the backward of one operator call needs besides the saved tensors.
struct CallState : torch::CustomClassHolder {
  Params p;
  ConvGeom q{0, 0, -1, -1};
  Tensor sink;      // where dW goes instead of into autograd: a slice of the flat gradient bucket
};

void keep(AutogradContext* ctx, const c10::intrusive_ptr<CallState>& s) {
  ctx->saved_data["call"] = c10::IValue::make_capsule(s);
}
c10::intrusive_ptr<CallState> kept(AutogradContext* ctx) {
  return c10::static_intrusive_pointer_cast<CallState>(ctx->saved_data["call"].toCapsule());
}

// `layer`: only the spike values are returned (the packed second half never goes through autograd)
struct FcFunction : torch::autograd::Function<FcFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& X, const Tensor& W, c10::intrusive_ptr<CallState> s, bool layer) {
    const Tensor out = fc_forward_call(X, W, s->p, false);
    keep(ctx, s);
    ctx->save_for_backward({X, W, out});
    return layer ? out.narrow(0, 0, X.size(0)) : out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const auto s = kept(ctx);
    auto r = fc_grad_call(grads[0], saved[0], saved[1], s->p, saved[2], ctx->needs_input_grad(0), s->sink, Tensor());
    return {r.first, s->sink.defined() ? Tensor() : r.second, Tensor(), Tensor()};
  }
};

struct CvFunction : torch::autograd::Function<CvFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& X, const Tensor& W, c10::intrusive_ptr<CallState> s, bool layer) {
    const Tensor out = cv_forward_call(X, W, s->p, s->q, false);
    keep(ctx, s);
    ctx->save_for_backward({X, W, out});
    return layer ? out.narrow(0, 0, X.size(0)) : out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const auto s = kept(ctx);
    auto r = cv_grad_call(grads[0], saved[0], saved[1], s->p, saved[2], s->q.pt, s->q.pl, ctx->needs_input_grad(0), s->sink, Tensor());
    return {r.first, s->sink.defined() ? Tensor() : r.second, Tensor(), Tensor()};
  }
};

bool wants_grad(const Tensor& X, const Tensor& W) {
  return at::GradMode::is_enabled() && (X.requires_grad() || W.requires_grad());
}

c10::intrusive_ptr<CallState> call_state(py::handle params, int n, const std::optional<Tensor>& sink) {
  auto s = c10::make_intrusive<CallState>();
  s->p = read_params(params, n);
  if (sink.has_value()) s->sink = *sink;
  return s;
}

Tensor fc_layer(const Tensor& X, const Tensor& W, py::handle params, const std::optional<Tensor>& sink) {
  auto s = call_state(params, 6, sink);
  const py::gil_scoped_release nogil;
  if (!wants_grad(X, W)) return fc_forward_call(X, W, s->p, true);   // nothing will read 1/(sum w - theta)
  return FcFunction::apply(X, W, s, true);
}

Tensor cv_layer(const Tensor& X, const Tensor& W, py::handle params, int pt, int pl, int64_t Nh, int64_t Nw,
                const std::optional<Tensor>& sink) {
  auto s = call_state(params, 12, sink);
  s->q = {pt, pl, Nh, Nw};
  const py::gil_scoped_release nogil;
  if (!wants_grad(X, W)) return cv_forward_call(X, W, s->p, s->q, true);
  return CvFunction::apply(X, W, s, true);
}

Tensor fc_op(const Tensor& X, const Tensor& W, py::handle params) {
  auto s = call_state(params, 6, std::nullopt);
  const py::gil_scoped_release nogil;
  return FcFunction::apply(X, W, s, false);
}
Tensor cv_op(const Tensor& X, const Tensor& W, py::handle params) {
  auto s = call_state(params, 12, std::nullopt);
  const py::gil_scoped_release nogil;
  return CvFunction::apply(X, W, s, false);
}

Tensor fc_forward(const Tensor& X, const Tensor& W, py::handle params, bool infer) {
  const Params p = read_params(params, 6);
  const py::gil_scoped_release nogil;
  return fc_forward_call(X, W, p, infer);
}
Tensor cv_forward(const Tensor& X, const Tensor& W, py::handle params, int pt, int pl, int64_t Nh, int64_t Nw, bool infer) {
  const Params p = read_params(params, 12);
  const py::gil_scoped_release nogil;
  return cv_forward_call(X, W, p, {pt, pl, Nh, Nw}, infer);
}
py::tuple fc_grad(const Tensor& G, const Tensor& X, const Tensor& W, py::handle params, const Tensor& out, bool need_dx,
                  const std::optional<Tensor>& dw_out) {
  const Tensor dp = X.is_cuda() ? empty_like_dev({6}, X) : Tensor();
  const Params p = read_params(params, 6);
  std::pair<Tensor, Tensor> r;
  {
    const py::gil_scoped_release nogil;
    r = fc_grad_call(G, X, W, p, out, need_dx, dw_out.value_or(Tensor()), dp);
  }
  return py::make_tuple(need_dx ? py::cast(r.first) : py::none(), r.second, dp);
}
py::tuple cv_grad(const Tensor& G, const Tensor& X, const Tensor& W, py::handle params, const Tensor& out, int pt, int pl,
                  bool need_dx, const std::optional<Tensor>& dw_out) {
  const Tensor dp = X.is_cuda() ? empty_like_dev({12}, X) : Tensor();
  const Params p = read_params(params, 12);
  std::pair<Tensor, Tensor> r;
  {
    const py::gil_scoped_release nogil;
    r = cv_grad_call(G, X, W, p, out, pt, pl, need_dx, dw_out.value_or(Tensor()), dp);
  }
  return py::make_tuple(need_dx ? py::cast(r.first) : py::none(), r.second, dp);
}

// ------------------------------------------------------------------------------------------------ pooling
struct PoolGeom { int Kh, Kw, Sh, Sw, pt, pl, Nh, Nw; };

std::pair<Tensor, Tensor> minpool_call(const Tensor& X, const PoolGeom& q, float padvalue, bool want_arg) {
  const Tensor x = as_cuda_f32(X, "input");
  TORCH_CHECK_VALUE(x.dim() == 4, "snn_minpool expects an NHWC input");
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor y = empty_like_dev({x.size(0), q.Nh, q.Nw, x.size(3)}, x);
  const Tensor arg = want_arg ? at::empty({x.size(0), q.Nh, q.Nw, x.size(3)}, x.options().dtype(at::kInt).requires_grad(false)) : Tensor();
  check(snntc_minpool_forward(ptr(x), ptr(y), want_arg ? arg.data_ptr<int>() : nullptr, (int)x.size(0), (int)x.size(1),
                              (int)x.size(2), (int)x.size(3), q.Kh, q.Kw, q.Sh, q.Sw, q.pt, q.pl, q.Nh, q.Nw, padvalue,
                              stream_of(x)), "minpool forward");
  return {y, arg};
}

struct PoolState : torch::CustomClassHolder {
  PoolGeom q;
  std::vector<int64_t> shape;
};

struct PoolFunction : torch::autograd::Function<PoolFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& X, c10::intrusive_ptr<PoolState> s, double padvalue) {
    auto r = minpool_call(X, s->q, (float)padvalue, true);
    s->shape = X.sizes().vec();
    ctx->save_for_backward({r.second});
    ctx->saved_data["call"] = c10::IValue::make_capsule(s);
    return r.first;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = c10::static_intrusive_pointer_cast<PoolState>(ctx->saved_data["call"].toCapsule());
    const Tensor arg = ctx->get_saved_variables()[0];
    const Tensor gy = as_cuda_f32(grads[0], "grad");
    const c10::cuda::CUDAGuard guard(gy.device());
    const Tensor dx = empty_like_dev(s->shape, gy);
    const PoolGeom& q = s->q;
    check(snntc_minpool_backward(ptr(gy), arg.data_ptr<int>(), ptr(dx), (int)s->shape[0], (int)s->shape[1], (int)s->shape[2],
                                 (int)s->shape[3], q.Kh, q.Kw, q.Sh, q.Sw, q.pt, q.pl, q.Nh, q.Nw, stream_of(gy)),
          "minpool backward");
    return {dx, Tensor(), Tensor()};
  }
};

Tensor minpool(const Tensor& X, int Kh, int Kw, int Sh, int Sw, int pt, int pl, int Nh, int Nw, double padvalue) {
  const PoolGeom q{Kh, Kw, Sh, Sw, pt, pl, Nh, Nw};
  if (!(at::GradMode::is_enabled() && X.requires_grad())) return minpool_call(X, q, (float)padvalue, false).first;
  auto s = c10::make_intrusive<PoolState>();
  s->q = q;
  return PoolFunction::apply(X, s, padvalue);
}

// ------------------------------------------------------------------------------------------------ rest of a step
Tensor encode(const Tensor& P, double scale, bool one_minus) {
  const Tensor p = as_cuda_f32(P, "p");
  const c10::cuda::CUDAGuard guard(p.device());
  const Tensor x = at::empty_like(p);
  check(snntc_encode(ptr(p), ptr(x), (size_t)p.numel(), (float)scale, one_minus ? 1 : 0, stream_of(p)), "encode");
  return x;
}

// Mean cross-entropy on the negated spike times and the number of arg-min hits; the gradient is formed in the backward
// (one kernel that reads the incoming scalar), not in the forward.
struct LossFunction : torch::autograd::Function<LossFunction> {
  static variable_list forward(AutogradContext* ctx, const Tensor& logit, const Tensor& label) {
    const Tensor y = as_cuda_f32(logit, "logit");
    const int B = to_int(y.size(0), "loss_func"), J = to_int(y.size(1), "loss_func");
    const c10::cuda::CUDAGuard guard(y.device());
    const Tensor loss = empty_like_dev({}, y), hits = empty_like_dev({}, y);
    const size_t bytes = snntc_loss_forward_workspace_bytes(B, J);
    const Tensor ws = bytes ? workspace(bytes, y) : Tensor();
    check(snntc_loss_forward_ws(ptr(y), (const long long*)label.data_ptr<int64_t>(), ptr(loss), ptr(hits), B, J, 1.0f / B,
                                bytes ? ws.data_ptr() : nullptr, bytes, stream_of(y)), "loss_func");
    ctx->save_for_backward({y, label});
    ctx->mark_non_differentiable({hits});
    return {loss, hits};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor& y = saved[0];
    const Tensor g = as_cuda_f32(grads[0], "gradient of the loss");
    const c10::cuda::CUDAGuard guard(y.device());
    const Tensor grad = at::empty_like(y);
    check(snntc_loss_backward(ptr(y), (const long long*)saved[1].data_ptr<int64_t>(), ptr(g), ptr(grad), (int)y.size(0),
                              (int)y.size(1), 1.0f / y.size(0), stream_of(y)), "loss_func");
    return {grad, Tensor()};
  }
};

std::pair<Tensor, Tensor> loss(const Tensor& logit, const Tensor& label) {
  TORCH_CHECK_VALUE(logit.dim() == 2, "loss_func expects logit[B,classes]");
  if (!logit.is_cuda()) (void)as_cuda_f32(logit, "logit");
  Tensor lab = label.dim() == 2 ? label.argmax(1) : label;   // one-hot, as the reference passes it
  lab = lab.to(logit.device(), at::kLong).contiguous();
  TORCH_CHECK_VALUE(lab.numel() == logit.size(0), "loss_func expects one label per row of logit");
  auto r = LossFunction::apply(logit, lab);
  return {r[0], r[1]};
}

// The constraint cost of all weight tensors of a network in two launches, its gradient in one.
struct CostState : torch::CustomClassHolder {
  float K, K2;
  Tensor colsum;
};

struct WeightList {
  std::vector<const float*> w;
  std::vector<int> rows, cols;
  int64_t columns = 0;
  void add(const Tensor& t) {
    TORCH_CHECK_VALUE(t.dim() == 2, "constraint_cost expects [fan_in, fan_out] weights");
    w.push_back(t.data_ptr<float>());
    rows.push_back(to_int(t.size(0), "constraint_cost"));
    cols.push_back(to_int(t.size(1), "constraint_cost"));
    columns += t.size(1);
  }
};

void cost_grads(const variable_list& ws, const variable_list& gw, const CostState& s, const Tensor& g, bool add) {
  const c10::cuda::CUDAGuard guard(g.device());
  WeightList l;
  std::vector<float*> to;
  for (const Tensor& t : ws) l.add(t);
  for (const Tensor& t : gw) to.push_back(ptr(t));
  check(snntc_weight_cost_grads((int)ws.size(), l.w.data(), to.data(), l.rows.data(), l.cols.data(), s.K, s.K2, ptr(s.colsum),
                                ptr(g), add ? 1 : 0, stream_of(g)), "constraint_cost");
}

// A backward pass in which the gradient of a network's constraint cost is added straight to the flat gradient bucket that the
// layers' dW kernels write (SnnNet.backward), instead of going through one gradient tensor per weight, an accumulation each
// and an addition: the cost's node leaves what it would have computed here, and it is computed once autograd is through --
// the dW kernels write their slices, in whatever order autograd visits the nodes.
struct Fold {
  struct Pending { variable_list weights; c10::intrusive_ptr<CostState> state; Tensor grad; };
  int graph_task = -1;             // of the pass: a cost's node that runs in any other pass is none of this one's
  c10::cuda::CUDAStream stream;    // the caller's, on which the gradients are formed in the end
  std::vector<const void*> weights;
  variable_list sinks;
  std::vector<Pending> pending;
  const Tensor* sink_of(const Tensor& w) const {
    for (size_t k = 0; k < weights.size(); ++k)
      if (weights[k] == w.data_ptr()) return &sinks[k];
    return nullptr;
  }
};
std::mutex g_fold_mutex;
std::vector<Fold*> g_folds;        // the backward passes of this kind under way

// The first node of such a pass (autograd runs it on a thread of its own choice): hands the gradient on, and the pass is known.
struct FoldRoot : torch::autograd::Node {
  Fold* fold = nullptr;
  variable_list apply(variable_list&& grads) override {
    const std::lock_guard<std::mutex> lock(g_fold_mutex);
    fold->graph_task = torch::autograd::get_current_graph_task_id();
    g_folds.push_back(fold);
    return std::move(grads);
  }
};

// Whether autograd would do no more with the calling node's k-th gradient than add it to a leaf's .grad. Not so for a weight that
// requires no gradient, which gets none, nor where a hook of any kind is to see the gradient.
bool only_accumulated(size_t k) {
  const torch::autograd::Edge& edge = torch::autograd::get_current_node()->next_edge(k);
  auto* leaf = dynamic_cast<torch::autograd::AccumulateGrad*>(edge.function.get());
  return leaf != nullptr && leaf->tensor_pre_hooks().empty() && leaf->tensor_post_acc_grad_hooks() == nullptr &&
         leaf->retains_grad_hooks().empty() && leaf->pre_hooks().empty() && leaf->post_hooks().empty();
}

// true: the pass that the calling node runs in takes the cost's gradient itself (it knows every weight, nothing else is to happen
// to their gradients, and the node runs on the caller's stream, so that nothing has to be waited for)
bool fold_cost(const variable_list& ws, const c10::intrusive_ptr<CostState>& s, const Tensor& g) {
  const std::lock_guard<std::mutex> lock(g_fold_mutex);
  const int task = torch::autograd::get_current_graph_task_id();
  for (Fold* f : g_folds) {
    if (f->graph_task != task) continue;
    if (at::cuda::getCurrentCUDAStream(g.get_device()) != f->stream) return false;
    for (size_t k = 0; k < ws.size(); ++k)
      if (f->sink_of(ws[k]) == nullptr || !only_accumulated(k)) return false;
    f->pending.push_back({ws, s, g});
    return true;
  }
  return false;
}

struct CostFunction : torch::autograd::Function<CostFunction> {
  static Tensor forward(AutogradContext* ctx, at::TensorList weights, c10::intrusive_ptr<CostState> s) {
    variable_list ws;
    WeightList l;
    for (const Tensor& t : weights) ws.push_back(as_cuda_f32(t, "weight"));
    for (const Tensor& t : ws) l.add(t);
    const c10::cuda::CUDAGuard guard(ws[0].device());
    const Tensor cost = empty_like_dev({}, ws[0]);
    s->colsum = empty_like_dev({l.columns}, ws[0]);
    const size_t bytes = snntc_weight_costs_workspace_bytes((int)ws.size(), l.rows.data(), l.cols.data());
    const Tensor tmp = workspace(bytes, ws[0]);
    check(snntc_weight_costs((int)ws.size(), l.w.data(), l.rows.data(), l.cols.data(), s->K, s->K2, ptr(s->colsum), ptr(cost),
                             tmp.data_ptr(), bytes, stream_of(ws[0])), "constraint_cost");
    ctx->saved_data["call"] = c10::IValue::make_capsule(s);
    ctx->save_for_backward(ws);
    return cost;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto ws = ctx->get_saved_variables();
    const auto s = c10::static_intrusive_pointer_cast<CostState>(ctx->saved_data["call"].toCapsule());
    const Tensor g = as_cuda_f32(grads[0], "gradient of the cost");
    if (fold_cost(ws, s, g)) return variable_list(ws.size() + 1);
    variable_list out;
    for (const Tensor& t : ws) out.push_back(at::empty_like(t));
    cost_grads(ws, out, *s, g, false);
    out.push_back(Tensor());
    return out;
  }
};

// objective.backward() with the upstream gradient `one`; constraint costs of `weights` go into `sinks` (see Fold)
void backward(const Tensor& objective, const Tensor& one, const std::vector<Tensor>& weights, const std::vector<Tensor>& sinks) {
  Fold f{.stream = at::cuda::getCurrentCUDAStream(objective.get_device())};
  for (const Tensor& w : weights) f.weights.push_back(w.data_ptr());
  f.sinks = sinks;
  struct Leave {
    Fold* f;
    ~Leave() {
      const std::lock_guard<std::mutex> lock(g_fold_mutex);
      g_folds.erase(std::remove(g_folds.begin(), g_folds.end(), f), g_folds.end());
    }
  };
  {
    const Leave leave{&f};
    if (objective.requires_grad()) {
      auto node = std::make_shared<FoldRoot>();
      node->fold = &f;
      node->add_input_metadata(objective);
      node->add_next_edge(torch::autograd::impl::gradient_edge(objective));
      torch::autograd::Engine::get_default_engine().execute({torch::autograd::Edge(std::move(node), 0)}, {one}, false, false, true);
    } else {
      torch::autograd::backward({objective}, {one});     // raises
    }
  }
  for (const Fold::Pending& p : f.pending) {
    variable_list to;
    for (const Tensor& w : p.weights) to.push_back(*f.sink_of(w));
    cost_grads(p.weights, to, *p.state, p.grad, true);
  }
}

Tensor constraint_cost(const std::vector<Tensor>& weights, double K, double K2) {
  TORCH_CHECK_VALUE(!weights.empty(), "constraint_cost needs at least one weight");
  auto s = c10::make_intrusive<CostState>();
  s->K = (float)K;
  s->K2 = (float)K2;
  return CostFunction::apply(at::TensorList(weights), s);
}

void adam_step(const Tensor& w, const Tensor& g, const Tensor& m, const Tensor& v, double lr, double b1, double b2, double eps,
               double scale, const Tensor& steps) {
  const c10::cuda::CUDAGuard guard(w.device());
  check(snntc_adam_step(ptr(w), ptr(g), ptr(m), ptr(v), (size_t)w.numel(), (float)lr, (float)b1, (float)b2, (float)eps,
                        (float)scale, steps.data_ptr<int>(), stream_of(w)), "Adam.step");
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  m.doc() = "native host path of the SNN-TC operators (see ops.py and train.py)";
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const SnntcFailure& e) {
      PyErr_SetString(g_error_class.ptr() ? g_error_class.ptr() : PyExc_RuntimeError, e.what());
    }
  });
  m.def("init", [](py::object error_class, py::object params_fn) {
    g_error_class = error_class.release();
    g_params_fn = params_fn.release();
  });
  m.def("fc_forward", &fc_forward);
  m.def("cv_forward", &cv_forward);
  m.def("fc_grad", &fc_grad);
  m.def("cv_grad", &cv_grad);
  m.def("fc_layer", &fc_layer);
  m.def("cv_layer", &cv_layer);
  m.def("fc_op", &fc_op);
  m.def("cv_op", &cv_op);
  m.def("minpool", &minpool, py::call_guard<py::gil_scoped_release>());
  m.def("encode", &encode, py::call_guard<py::gil_scoped_release>());
  m.def("loss", &loss, py::call_guard<py::gil_scoped_release>());
  m.def("constraint_cost", &constraint_cost, py::call_guard<py::gil_scoped_release>());
  m.def("backward", &backward, py::call_guard<py::gil_scoped_release>());
  m.def("adam_step", &adam_step, py::call_guard<py::gil_scoped_release>());
}
