// Host side of the operator layer: allocates a call's outputs and workspace with torch's caching allocator and
// enters the C ABI.  The checks on arguments and dtypes, and all choices, stay in core/ops.py; what is here,
// beside the checks that operands fit each other (5 us a layer in Python, under 1 here), is what every call pays
// for -- device guard, current stream, two to five allocations, argument marshalling -- which through ctypes and
// torch's Python functions took 20 us an operator, more than the kernels of a small layer.  Every function
// returns (status, outputs...).
#include <stdexcept>
#include <string>

#include <torch/extension.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include "../../include/fdp_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

// Entry points of the library that _lib.py has loaded (it may be another build than the one beside this file).
struct Abi {
  decltype(&fdp_linear_wgrad_workspace_bytes) linear_wgrad_workspace_bytes;
  decltype(&fdp_linear_wgrad) linear_wgrad;
  decltype(&fdp_bias_grad_workspace_bytes) bias_grad_workspace_bytes;
  decltype(&fdp_bias_grad) bias_grad;
  decltype(&fdp_linear_dgrad_workspace_bytes) linear_dgrad_workspace_bytes;
  decltype(&fdp_linear_dgrad) linear_dgrad;
  decltype(&fdp_linear_bwd_workspace_bytes) linear_bwd_workspace_bytes;
  decltype(&fdp_linear_bwd) linear_bwd;
  decltype(&fdp_linear_fwd) linear_fwd;
  decltype(&fdp_layernorm_fwd) layernorm_fwd;
  decltype(&fdp_layernorm_bwd_workspace_bytes) layernorm_bwd_workspace_bytes;
  decltype(&fdp_layernorm_bwd) layernorm_bwd;
} abi;

void bind(const std::map<std::string, uint64_t>& fns) {
#define FDP_BIND(NAME) abi.NAME = reinterpret_cast<decltype(abi.NAME)>(fns.at("fdp_" #NAME))
  FDP_BIND(linear_wgrad_workspace_bytes); FDP_BIND(linear_wgrad);
  FDP_BIND(bias_grad_workspace_bytes); FDP_BIND(bias_grad);
  FDP_BIND(linear_bwd_workspace_bytes); FDP_BIND(linear_bwd);
  FDP_BIND(linear_dgrad_workspace_bytes); FDP_BIND(linear_dgrad); FDP_BIND(linear_fwd);
  FDP_BIND(layernorm_fwd); FDP_BIND(layernorm_bwd_workspace_bytes); FDP_BIND(layernorm_bwd);
#undef FDP_BIND
}

at::ScalarType scalar_type(int dt) {
  return dt == FDP_F32 ? at::kFloat : dt == FDP_BF16 ? at::kBFloat16 : at::kHalf;
}
Tensor new_tensor(const Tensor& like, at::IntArrayRef sizes, at::ScalarType t) {
  return at::empty(sizes, like.options().dtype(t).memory_format(std::nullopt));
}
Tensor workspace(const Tensor& like, size_t bytes) {
  return new_tensor(like, {static_cast<int64_t>(bytes < 256 ? 256 : bytes)}, at::kByte);
}
// The workspace that `query` asks for under the flags of `code`.  Where it does not fit the card, what asks for most is given
// up first: the per-sample products (up to 512 MiB) and the parts of a K split (38.8 MB); then the split copies of fp32
// operands in six products (1.5 times the operands, and 38.8 MB for a weight gradient) and the padded ones of 16-bit
// operands, whose shapes then stay on the FMA kernels, which need next to nothing.
template <typename Query>
Tensor workspace_or_less(const Tensor& like, int& code, Query query) {
  constexpr int SPEED = FDP_KEEP_PRODUCTS | FDP_GEMM_SPLIT_K, COPIES = FDP_FP32_WIDE | FDP_FP32_WIDE_GEMM | FDP_PAD_16BIT;
  for (const int flags : {SPEED, COPIES}) {
    try {
      return workspace(like, query(code));
    } catch (const c10::OutOfMemoryError&) {
      if ((code & (SPEED | COPIES)) == 0) throw;
      code &= ~flags;
    }
  }
  return workspace(like, query(code));
}
// The kernels take bare pointers and their sizes from one operand each: what does not fit would be misread, or read past
// its end.  Raised as RuntimeError before anything is allocated or launched.
void refuse(const char* what, const Tensor& t) {
  // (no stream: the module may carry a C++ library of its own beside torch's, whose locales do not mix)
  std::string s(what);
  s += ": got (";
  for (int64_t d = 0; d < t.dim(); ++d) s += (d ? ", " : "") + std::to_string(t.size(d));
  s += ") on " + std::string(c10::DeviceTypeName(t.device().type(), true)) + (t.device().has_index() ? ":" + std::to_string(t.device().index()) : "");
  throw std::runtime_error(s);
}
// weight of a product that contracts `k` columns: [n, k] or, with k_rows, [k, n] (n < 0: any)
void check_weight(const Tensor& W, int64_t k, int64_t n, bool k_rows, const Tensor& like) {
  if (W.dim() != 2 || W.size(k_rows ? 0 : 1) != k || (n >= 0 && W.size(k_rows ? 1 : 0) != n)) refuse("weight does not fit the other operands", W);
  if (W.device() != like.device()) refuse("weight is on another device", W);
}

// parameters and statistics of a layer norm over the last dimension of `x`, and what has its shape (dy)
void check_layernorm(const Tensor& x, const Tensor& w, const OptTensor& b, const OptTensor& mean, const OptTensor& rstd, const OptTensor& dy) {
  if (x.dim() < 1) refuse("input has no last dimension", x);
  const int64_t d = x.size(-1), rows = d > 0 ? x.numel() / d : 0;
  if (w.device() != x.device() || (b.has_value() && b->device() != x.device())) refuse("layer norm: input and parameters are not on one device", w);
  if (w.numel() != d || (b.has_value() && b->numel() != d)) refuse("layer norm: parameters do not fit the input's last dimension", w);
  for (const OptTensor& t : {mean, rstd})
    if (t.has_value() && (t->device() != x.device() || t->numel() != rows || t->scalar_type() != at::kFloat)) refuse("layer norm: statistics do not fit the input", *t);
  if (dy.has_value() && (dy->device() != x.device() || dy->numel() != x.numel())) refuse("layer norm: grad_output does not fit the input", *dy);
}

void* ptr(const Tensor& t) { return t.data_ptr(); }
void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }
fdp_stream_t stream(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// (C, clamp_value, noise std, batch divisor, seed, param_id, param_id2, step, rank, world, step counter or None)
fdp_dp_params params(const py::tuple& p) {
  fdp_dp_params q{};
  q.C = p[0].cast<float>(); q.clamp_value = p[1].cast<float>(); q.noise_std = p[2].cast<float>();
  q.batch_divisor = p[3].cast<int32_t>(); q.seed = p[4].cast<uint64_t>();
  q.param_id = p[5].cast<uint32_t>(); q.param_id2 = p[6].cast<uint32_t>(); q.step = p[7].cast<uint32_t>();
  q.noise_rank = p[8].cast<int32_t>(); q.noise_world = p[9].cast<int32_t>();
  q.step_device = p[10].is_none() ? nullptr : reinterpret_cast<decltype(q.step_device)>(p[10].cast<uint64_t>());
  return q;
}

py::tuple linear_wgrad(const Tensor& G, const Tensor& X, const OptTensor& out, int in_dt, int out_dt, int layout, int algo,
                       const py::tuple& p, bool want_norms) {
  const fdp_dp_params q = params(p);
  const c10::cuda::CUDAGuard guard(G.device());
  const int B = static_cast<int>(X.size(0)), T = static_cast<int>(X.size(1));
  const int n_in = static_cast<int>(X.size(2)), n_out = static_cast<int>(G.size(2));
  Tensor dW = out.has_value() ? *out
              : layout == FDP_OUT_IN ? new_tensor(G, {n_out, n_in}, scalar_type(out_dt)) : new_tensor(G, {n_in, n_out}, scalar_type(out_dt));
  OptTensor norms, factors;
  if (want_norms) { norms = new_tensor(G, {B}, at::kFloat); factors = new_tensor(G, {B}, at::kFloat); }
  const Tensor ws = workspace_or_less(G, algo, [&](int a) { return abi.linear_wgrad_workspace_bytes(B, T, n_in, n_out, in_dt, a); });
  int st;
  {
    py::gil_scoped_release nogil;
    st = abi.linear_wgrad(ptr(G), ptr(X), ptr(dW), static_cast<float*>(ptr(norms)), static_cast<float*>(ptr(factors)), B, T, n_in,
                          n_out, in_dt, out_dt, layout, algo, &q, ptr(ws), ws.numel(), stream(G));
  }
  return py::make_tuple(st, dW, norms, factors);
}

py::tuple bias_grad(const Tensor& G, int B, int T, int in_dt, int out_dt, const py::tuple& p, bool want_norms) {
  const fdp_dp_params q = params(p);
  const c10::cuda::CUDAGuard guard(G.device());
  const int n_out = static_cast<int>(G.size(-1));
  const Tensor db = new_tensor(G, {n_out}, scalar_type(out_dt));
  OptTensor norms, factors;
  if (want_norms) { norms = new_tensor(G, {B}, at::kFloat); factors = new_tensor(G, {B}, at::kFloat); }
  const Tensor ws = workspace(G, abi.bias_grad_workspace_bytes(B, T, n_out, in_dt));
  int st;
  {
    py::gil_scoped_release nogil;
    st = abi.bias_grad(ptr(G), ptr(db), static_cast<float*>(ptr(norms)), static_cast<float*>(ptr(factors)), B, T, n_out, in_dt, out_dt,
                       &q, ptr(ws), ws.numel(), stream(G));
  }
  return py::make_tuple(st, db, norms, factors);
}

// the leading sizes of `a` with `cols` columns
Tensor with_columns(const Tensor& a, int64_t cols, int dt) {
  c10::SmallVector<int64_t, 6> sizes(a.sizes().begin(), a.sizes().end());
  sizes.back() = cols;
  return new_tensor(a, sizes, scalar_type(dt));
}

py::tuple linear_dgrad(const Tensor& G, const Tensor& W, int rows, int code, int out_dt, int w_layout) {
  check_weight(W, G.size(-1), -1, w_layout == FDP_OUT_IN, G);
  const c10::cuda::CUDAGuard guard(G.device());
  const int n_out = static_cast<int>(G.size(-1)), n_in = static_cast<int>(W.size(w_layout == FDP_OUT_IN ? 1 : 0));
  const Tensor dX = with_columns(G, n_in, out_dt);
  const Tensor ws = workspace_or_less(G, code, [&](int c) { return abi.linear_dgrad_workspace_bytes(rows, n_in, n_out, c); });
  int st;
  {
    py::gil_scoped_release nogil;
    st = abi.linear_dgrad(ptr(G), ptr(W), ptr(dX), rows, n_in, n_out, code, out_dt, w_layout, ptr(ws), ws.numel(), stream(G));
  }
  return py::make_tuple(st, dX);
}

struct Bwd { int st; OptTensor dX, dW, db; };
// G, X as (B, T, .); X only where dW is wanted, W only where dX is
Bwd linear_bwd_call(const Tensor& G, const OptTensor& X, const OptTensor& W, const OptTensor& out, int n_in, int in_dt, int dx_dt, int dw_dt, int db_dt,
                     int layout, int algo, const fdp_dp_params& q, const fdp_dp_params& qb, bool need_dx, bool need_dw, bool need_db) {
  if (need_dx) check_weight(W.value(), G.size(2), n_in, layout == FDP_OUT_IN, G);
  if (X.has_value() && X->device() != G.device()) refuse("input is on another device than grad_output", *X);
  const c10::cuda::CUDAGuard guard(G.device());
  const int B = static_cast<int>(G.size(0)), T = static_cast<int>(G.size(1)), n_out = static_cast<int>(G.size(2));
  OptTensor dX, dW, db;
  const auto allocate = [&](int outputs) {
    if (outputs & FDP_BWD_DX) dX = with_columns(G, n_in, dx_dt);
    if (outputs & FDP_BWD_DW) dW = out.has_value() ? *out
                                   : layout == FDP_OUT_IN ? new_tensor(G, {n_out, n_in}, scalar_type(dw_dt)) : new_tensor(G, {n_in, n_out}, scalar_type(dw_dt));
    if (outputs & FDP_BWD_DB) db = new_tensor(G, {n_out}, scalar_type(db_dt));
  };
  // one call for the outputs that are named, in the workspace `ws`
  const auto call = [&](int outputs, int a, const Tensor& ws) {
    return abi.linear_bwd(ptr(G), ptr(X), ptr(W), (outputs & FDP_BWD_DX) ? ptr(dX) : nullptr, (outputs & FDP_BWD_DW) ? ptr(dW) : nullptr,
                          (outputs & FDP_BWD_DB) ? ptr(db) : nullptr, B, T, n_in, n_out, in_dt, dx_dt, dw_dt, db_dt, layout, a,
                          &q, &qb, ptr(ws), ws.numel(), stream(G));
  };
  const auto bytes = [&](int outputs, int a) { return abi.linear_bwd_workspace_bytes(B, T, n_in, n_out, in_dt, a, outputs); };
  const int outputs = (need_dx ? FDP_BWD_DX : 0) | (need_dw ? FDP_BWD_DW : 0) | (need_db ? FDP_BWD_DB : 0);
  int st = FDP_OK;
  OptTensor ws;
  const auto take = [&] {
    try {
      allocate(outputs);
      ws = workspace(G, bytes(outputs, algo));
    } catch (const c10::OutOfMemoryError&) {
      dX.reset(); dW.reset(); db.reset();
    }
    return ws.has_value();
  };
  constexpr int SPEED = FDP_KEEP_PRODUCTS | FDP_GEMM_SPLIT_K;
  if (!take() && bytes(outputs, algo & ~SPEED) < bytes(outputs, algo)) {
    algo &= ~SPEED;
    take();
  }
  if (ws.has_value()) {
    st = call(outputs, algo, *ws);
  } else {
    // One output at a time: the same results from less memory.  The workspaces follow one another, and no parts of W
    // and no statistics lie beside the parts of G and X.
    for (const int one : {FDP_BWD_DX, FDP_BWD_DW, FDP_BWD_DB}) {
      if ((outputs & one) == 0 || st != FDP_OK) continue;
      allocate(one);
      int a = algo;
      const Tensor own = workspace_or_less(G, a, [&](int b) { return bytes(one, b); });
      st = call(one, a, own);
    }
  }
  return {st, dX, dW, db};
}
py::tuple linear_bwd(const Tensor& G, const OptTensor& X, const OptTensor& W, const OptTensor& out, int n_in, int in_dt, int dx_dt, int dw_dt, int db_dt,
                     int layout, int algo, const py::tuple& p, const py::tuple& p_bias, bool need_dx, bool need_dw, bool need_db) {
  const fdp_dp_params q = params(p), qb = params(p_bias);
  Bwd r;
  {
    py::gil_scoped_release nogil;
    r = linear_bwd_call(G, X, W, out, n_in, in_dt, dx_dt, dw_dt, db_dt, layout, algo, q, qb, need_dx, need_dw, need_db);
  }
  return py::make_tuple(r.st, r.dX, r.dW, r.db);
}

std::pair<int, Tensor> linear_fwd_call(const Tensor& X, const Tensor& W, const OptTensor& bias, int rows, int code, int out_dt, int w_layout) {
  check_weight(W, X.size(-1), -1, w_layout != FDP_OUT_IN, X);
  if (bias.has_value() && (bias->numel() != W.size(w_layout == FDP_OUT_IN ? 0 : 1) || bias->device() != X.device()))
    refuse("bias does not fit the output's columns", *bias);
  const c10::cuda::CUDAGuard guard(X.device());
  const int n_in = static_cast<int>(X.size(-1)), n_out = static_cast<int>(W.size(w_layout == FDP_OUT_IN ? 0 : 1));
  const Tensor Y = with_columns(X, n_out, out_dt);
  const Tensor ws = workspace_or_less(X, code, [&](int c) { return abi.linear_dgrad_workspace_bytes(rows, n_out, n_in, c); });
  const int st = abi.linear_fwd(ptr(X), ptr(W), ptr(bias), ptr(Y), rows, n_in, n_out, code, out_dt, w_layout, ptr(ws), ws.numel(), stream(X));
  return {st, Y};
}
py::tuple linear_fwd(const Tensor& X, const Tensor& W, const OptTensor& bias, int rows, int code, int out_dt, int w_layout) {
  std::pair<int, Tensor> r;
  {
    py::gil_scoped_release nogil;
    r = linear_fwd_call(X, W, bias, rows, code, out_dt, w_layout);
  }
  return py::make_tuple(r.first, r.second);
}


struct LnFwd { int st; Tensor y, mean, rstd; };
LnFwd layernorm_fwd_call(const Tensor& x, const Tensor& w, const Tensor& b, double eps, int rows, int dt, int pdt) {
  check_layernorm(x, w, b, {}, {}, {});
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor y = new_tensor(x, x.sizes(), x.scalar_type());
  const Tensor mean = new_tensor(x, {rows}, at::kFloat), rstd = new_tensor(x, {rows}, at::kFloat);
  const int st = abi.layernorm_fwd(ptr(x), ptr(w), ptr(b), ptr(y), static_cast<float*>(ptr(mean)), static_cast<float*>(ptr(rstd)), rows,
                                   static_cast<int>(x.size(-1)), static_cast<float>(eps), dt, pdt, stream(x));
  return {st, y, mean, rstd};
}
py::tuple layernorm_fwd(const Tensor& x, const Tensor& w, const Tensor& b, double eps, int rows, int dt, int pdt) {
  LnFwd r;
  {
    py::gil_scoped_release nogil;
    r = layernorm_fwd_call(x, w, b, eps, rows, dt, pdt);
  }
  return py::make_tuple(r.st, r.y, r.mean, r.rstd);
}

struct LnBwd { int st; OptTensor dx; Tensor dgamma; OptTensor dbeta, ng, nb; };
LnBwd layernorm_bwd_call(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& mean, const Tensor& rstd, int B, int T,
                         int dt, int pdt, const fdp_dp_params& q, bool need_dx, bool need_dbeta, bool want_norms) {
  check_layernorm(x, w, {}, mean, rstd, dy);
  const c10::cuda::CUDAGuard guard(x.device());
  const int d = static_cast<int>(x.size(-1));
  OptTensor dx, dbeta, ng, nb;
  if (need_dx) dx = new_tensor(x, x.sizes(), x.scalar_type());
  const Tensor dgamma = new_tensor(x, {d}, w.scalar_type());
  if (need_dbeta) dbeta = new_tensor(x, {d}, w.scalar_type());
  if (want_norms) ng = new_tensor(x, {B}, at::kFloat);
  if (want_norms && need_dbeta) nb = new_tensor(x, {B}, at::kFloat);
  const Tensor ws = workspace(x, abi.layernorm_bwd_workspace_bytes(B, T, d));
  const int st = abi.layernorm_bwd(ptr(dy), ptr(x), ptr(w), static_cast<const float*>(ptr(mean)), static_cast<const float*>(ptr(rstd)), ptr(dx),
                                   ptr(dgamma), ptr(dbeta), static_cast<float*>(ptr(ng)), static_cast<float*>(ptr(nb)), B, T, d, dt, pdt, &q,
                                   ptr(ws), ws.numel(), stream(x));
  return {st, dx, dgamma, dbeta, ng, nb};
}
py::tuple layernorm_bwd(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& mean, const Tensor& rstd, int B, int T,
                        int dt, int pdt, const py::tuple& p, bool need_dx, bool need_dbeta, bool want_norms) {
  const fdp_dp_params q = params(p);
  LnBwd r;
  {
    py::gil_scoped_release nogil;
    r = layernorm_bwd_call(dy, x, w, mean, rstd, B, T, dt, pdt, q, need_dx, need_dbeta, want_norms);
  }
  return py::make_tuple(r.st, r.dx, r.dgamma, r.dbeta, r.ng, r.nb);
}

// ---- the layers' autograd nodes --------------------------------------------------------------------------------------
// What the Function classes of layers/*.py do, without a Python frame per tensor operation: a pass of a small layer is
// bound by the host, and of its 120 to 160 us those classes took a third.  Choices and noise bookkeeping stay in
// Python: one call a backward (`layers/_common.py`) takes the step and returns the parameters.  Both are tested to give
// the same bits.
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
struct PyCalls { py::object product, linear, layernorm, direct_done, check, dtype; }* py_calls = nullptr;    // (outlives the interpreter)

void bind_layers(const py::dict& f) {
  if (py_calls == nullptr) py_calls = new PyCalls;
  py_calls->product = f["product"]; py_calls->linear = f["linear"]; py_calls->layernorm = f["layernorm"];
  py_calls->direct_done = f["direct_done"]; py_calls->check = f["check"]; py_calls->dtype = f["dtype"];
}
// A Python exception on its way through the autograd engine, which knows python_error.
template <typename F>
auto python(F f) -> decltype(f()) {
  try {
    return f();
  } catch (py::error_already_set& e) {
    e.restore();
    python_error err;
    err.persist();
    throw err;
  }
}
// ... and back at the boundary to Python
template <typename F>
auto boundary(F f) -> decltype(f()) {
  try {
    return f();
  } catch (python_error& e) {
    e.restore();
    throw py::error_already_set();
  }
}
void check_status(int st, const char* what) {
  if (st == FDP_OK) return;
  py::gil_scoped_acquire gil;
  python([&] { py_calls->check(st, what); });
}
bool has_code(at::ScalarType t) { return t == at::kFloat || t == at::kBFloat16 || t == at::kHalf; }
int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return FDP_F32;
    case at::kBFloat16: return FDP_BF16;
    case at::kHalf: return FDP_F16;
    default: break;
  }
  py::gil_scoped_acquire gil;
  return python([&] { return py_calls->dtype(at::empty({0}, at::TensorOptions().dtype(t))).cast<int>(); });     // raises
}
int dtype_code(const Tensor& t) { return dtype_code(t.scalar_type()); }
Tensor aligned(const Tensor& t) {
  return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone(at::MemoryFormat::Contiguous);
}
// a Python object in a node's saved data
struct Holder final : c10::ivalue::PyObjectHolder {
  explicit Holder(PyObject* o) : o_(o) { Py_INCREF(o_); }
  ~Holder() override {
    if (!Py_IsInitialized()) return;
    py::gil_scoped_acquire gil;
    Py_DECREF(o_);
  }
  PyObject* getPyObject() override { return o_; }
  c10::InferredType tryToInferType() override { return c10::InferredType(std::string("a Python object")); }
  c10::IValue toIValue(const c10::TypePtr&, std::optional<int32_t>) override { return c10::IValue(); }
  std::string toStr() override { return "a Python object"; }
  std::vector<at::Tensor> extractTensors() override { return {}; }

 private:
  PyObject* o_;
};
c10::IValue hold(const py::object& o) { return c10::IValue(c10::intrusive_ptr<c10::ivalue::PyObjectHolder>(c10::make_intrusive<Holder>(o.ptr()))); }
py::object held(const c10::IValue& v) { return py::reinterpret_borrow<py::object>(v.toPyObject()); }
at::ScalarType autocast_type(const Tensor& input, const Tensor& weight) {
  if (!at::autocast::is_autocast_enabled(at::kCUDA) || !input.is_cuda() || !weight.is_cuda()) return at::ScalarType::Undefined;
  return at::autocast::get_autocast_dtype(at::kCUDA);
}
bool product_ok(const Tensor& a, int64_t rows, int64_t K, int64_t N) {
  if (!has_code(a.scalar_type())) return false;
  py::gil_scoped_acquire gil;
  return python([&] { return py_calls->product(dtype_code(a), rows, K, N).cast<bool>(); });
}

struct DpLinear : torch::autograd::Function<DpLinear> {
  // code: flags that an fp32 product takes; in_out: weight (in, out), as Conv1D's
  static Tensor forward(AutogradContext* ctx, const Tensor& input, const Tensor& weight, const OptTensor& bias, const c10::IValue& layer,
                        bool in_out, int64_t code) {
    const at::ScalarType dt = autocast_type(input, weight);
    const bool cast = dt != at::ScalarType::Undefined;
    const Tensor x = cast ? input.to(dt) : input, w = cast ? weight.to(dt) : weight;
    ctx->save_for_backward({x, weight, bias.has_value() ? *bias : Tensor(), cast ? w : Tensor()});
    ctx->saved_data["layer"] = layer;
    ctx->saved_data["in_out"] = in_out;
    ctx->saved_data["dtype"] = static_cast<int64_t>(input.scalar_type());
    const int64_t K = x.size(-1);
    if (K > 0 && w.dim() == 2 && product_ok(x, x.numel() / K, w.size(in_out ? 0 : 1), w.size(in_out ? 1 : 0))) {
      const Tensor X = aligned(x.contiguous()), W = aligned(w.to(x.scalar_type()).contiguous());
      OptTensor b;
      if (bias.has_value()) b = aligned(bias->to(x.scalar_type()).contiguous());
      const int t = dtype_code(x);
      const auto r = linear_fwd_call(X, W, b, static_cast<int>(X.numel() / K), t | (static_cast<int>(code) & (t == FDP_F32 ? ~0 : FDP_GEMM_SPLIT_K | FDP_PAD_16BIT)), t,
                                     in_out ? FDP_IN_OUT : FDP_OUT_IN);
      check_status(r.first, "fdp_linear_fwd");
      return r.second;
    }
    Tensor y = at::matmul(x, in_out ? w : w.t());
    if (!bias.has_value()) return y;
    const Tensor b = cast ? bias->to(dt) : *bias;
    return in_out ? y + b : y.add_(b);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &weight = saved[1], &bias = saved[2], &w = saved[3].defined() ? saved[3] : saved[1];
    const bool in_out = ctx->saved_data["in_out"].toBool();
    const bool need_dx = ctx->needs_input_grad(0), need_dw = ctx->needs_input_grad(1);
    const bool need_db = bias.defined() && ctx->needs_input_grad(2);
    Tensor x3 = x, g3 = grads[0];
    if (x.dim() == 2) {
      x3 = x.unsqueeze(1); g3 = g3.unsqueeze(1);
    } else if (x.dim() > 3) {
      x3 = x.reshape({x.size(0), -1, x.size(-1)}); g3 = g3.reshape({x.size(0), -1, g3.size(-1)});
    }
    const int64_t B = x3.size(0), K = w.size(in_out ? 1 : 0), N = w.size(in_out ? 0 : 1);
    // (a type the kernels do not know is refused only where they are asked: an input gradient alone is torch's then)
    const int t = has_code(g3.scalar_type()) ? dtype_code(g3) : -1;
    bool native_dx = false;
    OptTensor target;
    fdp_dp_params p{}, pb{};
    int algo = 0;
    {
      py::gil_scoped_acquire gil;
      python([&] {
        const py::tuple c = py_calls->linear(held(ctx->saved_data["layer"]), weight, B, t, K > 0 ? g3.numel() / K : 0, K, N, need_dx, need_dw, need_db);
        native_dx = c[0].cast<bool>();
        if (c.size() == 1) return;
        p = params(c[1]); pb = params(c[2]);
        algo = c[3].cast<int>();
        if (!c[4].is_none()) target = c[4].cast<Tensor>();
      });
    }
    Tensor dX;
    if (need_dx && !native_dx) {
      const Tensor wg = w.to(g3.scalar_type());
      dX = at::matmul(g3, in_out ? wg.t() : wg);
    }
    Tensor dW, db;
    if (native_dx || need_dw || need_db) {
      if (x3.dim() != 3 || g3.dim() != 3 || x3.size(0) != g3.size(0) || x3.size(1) != g3.size(1)) refuse("expected (B,T,in) and (B,T,out)", g3);
      dtype_code(g3);
      Tensor G = g3.contiguous();
      if (native_dx || need_dw) G = aligned(G);
      OptTensor X, W;
      if (need_dw) X = aligned(x3.to(G.scalar_type()).contiguous());
      if (native_dx) W = aligned(w.to(G.scalar_type()).contiguous());
      if (target.has_value() && (target->sizes() != weight.sizes() || !target->is_contiguous() || target->device() != G.device()))
        refuse("out must be a contiguous tensor of the weight's shape on its device", *target);
      const auto input_type = static_cast<at::ScalarType>(ctx->saved_data["dtype"].toInt());
      const int dx_dt = dtype_code(input_type);
      const Bwd r = linear_bwd_call(G, X, W, target, static_cast<int>(x3.size(-1)), t, dx_dt, dtype_code(target.has_value() ? *target : weight),
                                    need_db ? dtype_code(bias) : t, in_out ? FDP_IN_OUT : FDP_OUT_IN, algo, p, pb, native_dx, need_dw, need_db);
      check_status(r.st, "fdp_linear_bwd");
      if (native_dx) dX = *r.dX;
      if (need_dw && !target.has_value()) dW = *r.dW;       // else it is where the optimizer and the all-reduce read it
      if (need_db) db = *r.db;
      if (target.has_value()) {
        py::gil_scoped_acquire gil;
        python([&] { py_calls->direct_done(weight); });
      }
    }
    if (need_dx) dX = dX.reshape(x.sizes());
    return {dX, dW, db, Tensor(), Tensor(), Tensor()};
  }
};

struct DpLayerNorm : torch::autograd::Function<DpLayerNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& input, const Tensor& weight, const Tensor& bias, const c10::IValue& layer, double eps) {
    const Tensor x = input.contiguous(), w = weight.contiguous(), b = bias.to(w.scalar_type()).contiguous();
    const int64_t d = x.size(-1);
    if (d * x.element_size() >= 65536) throw std::runtime_error("This layer norm doesn't support feature dim >= 64KB.");
    const LnFwd r = layernorm_fwd_call(x, w, b, eps, d > 0 ? static_cast<int>(x.numel() / d) : 0, dtype_code(x), dtype_code(w));
    check_status(r.st, "fdp_layernorm_fwd");
    ctx->save_for_backward({input, weight, r.mean, r.rstd});
    ctx->saved_data["layer"] = layer;
    return r.y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor x = saved[0].contiguous(), w = saved[1].contiguous(), dy = grads[0].contiguous();
    const int64_t d = x.size(-1), B = x.dim() > 1 ? x.size(0) : 1;
    const bool need_dx = ctx->needs_input_grad(0), need_dw = ctx->needs_input_grad(1), need_db = ctx->needs_input_grad(2);
    fdp_dp_params p{};
    {
      py::gil_scoped_acquire gil;
      python([&] { p = params(py_calls->layernorm(held(ctx->saved_data["layer"]), B)); });
    }
    const LnBwd r = layernorm_bwd_call(dy, x, w, saved[2], saved[3], static_cast<int>(B), static_cast<int>(x.numel() / (B * d)), dtype_code(x),
                                       dtype_code(w), p, need_dx, need_db, false);
    check_status(r.st, "fdp_layernorm_bwd");
    return {need_dx ? *r.dx : Tensor(), need_dw ? r.dgamma : Tensor(), need_db ? *r.dbeta : Tensor(), Tensor(), Tensor()};
  }
};

// (the forward runs without the interpreter's lock, as the operator calls do: allocations and launches of one thread do not
// hold up the others)
Tensor dp_linear(const Tensor& input, const Tensor& weight, const OptTensor& bias, const py::object& layer, bool in_out, int64_t code) {
  const c10::IValue held_layer = hold(layer);
  return boundary([&] {
    py::gil_scoped_release nogil;
    return DpLinear::apply(input, weight, bias, held_layer, in_out, code);
  });
}
Tensor dp_layernorm(const Tensor& input, const Tensor& weight, const Tensor& bias, const py::object& layer, double eps) {
  const c10::IValue held_layer = hold(layer);
  return boundary([&] {
    py::gil_scoped_release nogil;
    return DpLayerNorm::apply(input, weight, bias, held_layer, eps);
  });
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.attr("built_for") = FDP_HOST_TAG;      // the build compares it with the torch it finds
  m.def("bind", &bind);
  m.def("linear_wgrad", &linear_wgrad);
  m.def("bias_grad", &bias_grad);
  m.def("linear_dgrad", &linear_dgrad);
  m.def("linear_bwd", &linear_bwd);
  m.def("linear_fwd", &linear_fwd);
  m.def("layernorm_fwd", &layernorm_fwd);
  m.def("layernorm_bwd", &layernorm_bwd);
  m.def("bind_layers", &bind_layers);
  m.def("dp_linear", &dp_linear);
  m.def("dp_layernorm", &dp_layernorm);
}
