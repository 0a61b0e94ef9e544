// Host layer of the public operators in native code: argument checks of the usual calls, output and workspace
// allocation, the argument structs of the C ABI and the autograd node.
//
// Why: a call through Python (autograd.Function, a ctypes struct filled field by field, one torch.empty per buffer) kept
// the host busy for 27 us per decode step, 66-118 us per forward and 240-310 us per training step (measured on a B200
// host, problems too small to keep the GPU busy), more than the kernels of every small call take.  Every entry point
// here returns None for anything but the plain case (separate decode weights, odd dtypes, arguments that must raise);
// the Python layer then serves the call and words the errors.
//
// The kernels are reached through the C ABI only; the addresses come from the library the Python layer has loaded.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <stdlib.h>
#include <string.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <cmath>
#include <string>

#include "../../include/flare_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;

// ---- the C ABI, bound once by the Python layer ---------------------------------------------------------------
struct Api {
  decltype(&flare_forward_workspace_bytes) forward_workspace_bytes = nullptr;
  decltype(&flare_forward_keep_bytes) forward_keep_bytes = nullptr;
  decltype(&flare_forward) forward = nullptr;
  decltype(&flare_forward_masked_workspace_bytes) forward_masked_workspace_bytes = nullptr;
  decltype(&flare_forward_masked) forward_masked = nullptr;
  decltype(&flare_backward_workspace_bytes) backward_workspace_bytes = nullptr;
  decltype(&flare_backward) backward = nullptr;
  decltype(&flare_decode_step) decode_step = nullptr;
  decltype(&flare_status_string) status_string = nullptr;
  decltype(&flare_last_cuda_error) last_cuda_error = nullptr;
} api;

template <typename F>
void take(F& f, const py::dict& table, const char* name) {
  f = reinterpret_cast<F>(table[name].cast<uintptr_t>());
}

void bind(const py::dict& table) {
  decltype(&flare_abi_version) version = nullptr;
  take(version, table, "flare_abi_version");
  if (version() != FLARE_ABI_VERSION) throw std::runtime_error("the native host layer was built for another version of the library");
  take(api.forward_workspace_bytes, table, "flare_forward_workspace_bytes");
  take(api.forward_keep_bytes, table, "flare_forward_keep_bytes");
  take(api.forward, table, "flare_forward");
  take(api.forward_masked_workspace_bytes, table, "flare_forward_masked_workspace_bytes");
  take(api.forward_masked, table, "flare_forward_masked");
  take(api.backward_workspace_bytes, table, "flare_backward_workspace_bytes");
  take(api.backward, table, "flare_backward");
  take(api.decode_step, table, "flare_decode_step");
  take(api.status_string, table, "flare_status_string");
  take(api.last_cuda_error, table, "flare_last_cuda_error");
}

// the exception classes of the Python binding (workspace and CUDA failures: RuntimeError, the rest: ValueError)
void check(int status, const char* what) {
  if (status == FLARE_OK) return;
  std::string msg = std::string(what) + " failed: " + api.status_string(status);
  if (status == FLARE_ERR_CUDA) msg += std::string(": ") + api.last_cuda_error();
  msg += " (status " + std::to_string(status) + ")";
  if (status == FLARE_ERR_WORKSPACE || status == FLARE_ERR_CUDA) throw std::runtime_error(msg);
  throw c10::ValueError({__func__, __FILE__, static_cast<uint32_t>(__LINE__)}, msg);
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return FLARE_F32;
    case at::kBFloat16: return FLARE_BF16;
    case at::kHalf: return FLARE_F16;
    default: return -1;
  }
}

// kernel path asked for by FLARE_B200_PATH; -1: not a value this layer knows (the Python layer reports it)
int path_from_env() {
  const char* e = getenv("FLARE_B200_PATH");
  if (e == nullptr || strcmp(e, "auto") == 0) return FLARE_PATH_AUTO;
  if (strcmp(e, "exact") == 0) return FLARE_PATH_EXACT;
  if (strcmp(e, "tensor") == 0) return FLARE_PATH_TENSOR;
  return -1;
}

// readable in place by the kernels: inner dimension contiguous, 16-byte aligned rows
bool readable(const Tensor& t) {
  const auto st = t.strides();
  if (st.back() != 1 || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u)) return false;
  for (size_t i = 0; i + 1 < st.size(); ++i)
    if (st[i] % 8) return false;
  return true;
}
Tensor ready(const Tensor& t) { return readable(t) ? t : t.contiguous(); }

bool same_kind(const Tensor& t, const Tensor& like) {
  return t.is_cuda() && t.device() == like.device() && t.scalar_type() == like.scalar_type();
}

// Storage that the kernels may read, and nothing that a call past the Python autograd functions would lose: no wrapper of a
// function transform or of a Python tensor class (no storage of its own), no forward-mode tangent (the Python functions
// refuse one; it would be dropped here).
bool ordinary(const Tensor& t) {
  constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                         c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize});
  return t.defined() && !t.key_set().has_any(wrapped) && !t._fw_grad(/*level=*/0).defined();
}

// Q [H, M, Dk], K [B, N, H, Dk], V [B, N, H, Dv] of one 16/32-bit float type on one GPU, not empty, sizes the kernels take
bool plain_qkv(const Tensor& q, const Tensor& k, const Tensor& v) {
  // (torch.jit.trace records the Python autograd functions as calls; of this layer it would record the empty output tensor)
  if (torch::jit::tracer::isTracing()) return false;
  if (!ordinary(q) || !ordinary(k) || !ordinary(v)) return false;
  if (q.dim() != 3 || k.dim() != 4 || v.dim() != 4 || !k.is_cuda()) return false;
  if (!same_kind(q, k) || !same_kind(v, k) || dtype_code(k.scalar_type()) < 0) return false;
  if (k.layout() != at::kStrided || v.layout() != at::kStrided || q.layout() != at::kStrided) return false;
  for (int i = 0; i < 3; ++i)
    if (k.size(i) != v.size(i) || k.size(i) == 0) return false;
  if (q.size(0) != k.size(2) || q.size(2) != k.size(3)) return false;
  return q.size(1) > 0 && q.size(1) % 16 == 0 && q.size(2) % 16 == 0 && v.size(3) > 0 && v.size(3) % 16 == 0 && k.size(3) > 0;
}

// float(scale), as the Python layer takes it (a text among others); false: it has to raise
bool to_scale(const py::object& scale, double* out) {
  PyObject* const f = PyNumber_Float(scale.ptr());
  if (f == nullptr) {
    PyErr_Clear();
    return false;
  }
  *out = PyFloat_AS_DOUBLE(f);
  Py_DECREF(f);
  return true;
}
bool default_scale(const py::object& scale, int64_t dk, double* out) {
  if (!scale.is_none()) return to_scale(scale, out);
  *out = dk <= 8 ? 1.0 : std::pow(static_cast<double>(dk), -0.5);
  return true;
}

struct Problem {
  Tensor q, k, v;
  double scale = 1.0, power = 2.0;
  int variant = FLARE_SOFTMAX, block = 1, path = FLARE_PATH_AUTO;
};

void fill(flare_fwd_args_t& a, const Problem& p) {
  memset(&a, 0, sizeof(a));
  a.q = p.q.data_ptr(); a.k = p.k.data_ptr(); a.v = p.v.data_ptr();
  a.B = (int32_t)p.k.size(0); a.N = (int32_t)p.k.size(1); a.H = (int32_t)p.k.size(2);
  a.M = (int32_t)p.q.size(1); a.Dk = (int32_t)p.k.size(3); a.Dv = (int32_t)p.v.size(3);
  a.q_stride_h = p.q.stride(0); a.q_stride_m = p.q.stride(1);
  a.k_stride_b = p.k.stride(0); a.k_stride_n = p.k.stride(1); a.k_stride_h = p.k.stride(2);
  a.v_stride_b = p.v.stride(0); a.v_stride_n = p.v.stride(1); a.v_stride_h = p.v.stride(2);
  a.scale = (float)p.scale; a.power = (float)p.power;
  a.dtype = dtype_code(p.k.scalar_type()); a.variant = p.variant; a.block_size = p.block; a.path = p.path;
}

struct State {
  Tensor m, d, u;
  bool given() const { return u.defined(); }
};

flare_state_t pointers(const State& s) {
  if (!s.given()) return flare_state_t{nullptr, nullptr, nullptr};
  return flare_state_t{s.m.data_ptr<float>(), s.d.data_ptr<float>(), s.u.data_ptr<float>()};
}

// {"m", "d", "u"} fp32 contiguous of the expected shapes on the device; false: anything else (the Python layer decides)
bool plain_state(const py::object& obj, int64_t B, int64_t H, int64_t M, int64_t Dv, const Tensor& like, State* out) {
  if (!PyDict_Check(obj.ptr())) return false;
  Tensor* const to[3] = {&out->m, &out->d, &out->u};
  const char* const names[3] = {"m", "d", "u"};
  for (int i = 0; i < 3; ++i) {
    PyObject* o = PyDict_GetItemString(obj.ptr(), names[i]);
    if (o == nullptr || !THPVariable_Check(o)) return false;
    const Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.device() != like.device() || t.scalar_type() != at::kFloat || !t.is_contiguous()) return false;
    if (t.dim() != (i == 2 ? 4 : 3) || t.size(0) != B || t.size(1) != H || t.size(2) != M || (i == 2 && t.size(3) != Dv))
      return false;
    *to[i] = t;
  }
  return (reinterpret_cast<uintptr_t>(out->u.data_ptr()) & 15u) == 0;
}

py::dict state_dict(const State& s) {
  py::dict d;
  d["m"] = s.m; d["d"] = s.d; d["u"] = s.u;
  return d;
}

struct Forward {
  Tensor y, lse_dec, lse_enc, keep;
  State out;
};

// mask: [B, N] int32, or undefined
Forward run_forward(const Problem& p, const State& in, bool want_state, bool want_lse, bool want_keep, const Tensor& mask = Tensor()) {
  const auto opts = p.k.options().requires_grad(false);
  const auto f32 = opts.dtype(at::kFloat);
  const int64_t B = p.k.size(0), N = p.k.size(1), H = p.k.size(2), M = p.q.size(1), Dv = p.v.size(3);
  Forward r;
  flare_fwd_args_t a;
  fill(a, p);
  r.y = at::empty({B, N, H, Dv}, opts);
  a.y = r.y.data_ptr();
  a.y_stride_b = N * H * Dv; a.y_stride_n = H * Dv; a.y_stride_h = Dv;
  a.state_in = pointers(in);
  if (want_state) {
    r.out = State{at::empty({B, H, M}, f32), at::empty({B, H, M}, f32), at::empty({B, H, M, Dv}, f32)};
    a.state_out = pointers(r.out);
  }
  size_t keep_bytes = want_keep ? api.forward_keep_bytes(&a) : 0;
  if (want_lse || keep_bytes > 0) {
    r.lse_dec = at::empty({B, H, N}, f32);
    a.lse_dec = r.lse_dec.data_ptr<float>();
  }
  if (want_lse && p.block > 1) {
    r.lse_enc = at::empty({B, H, N / p.block, M}, f32);
    a.lse_enc = r.lse_enc.data_ptr<float>();
    if (want_keep) keep_bytes = api.forward_keep_bytes(&a);
  }
  if (keep_bytes > 0) {
    r.keep = at::empty({(int64_t)keep_bytes}, opts.dtype(at::kByte));
    a.keep = r.keep.data_ptr();
    a.keep_bytes = keep_bytes;
  }
  Tensor ws;
  if (mask.defined()) a.mask = mask.data_ptr<int32_t>();
  if (const size_t need = mask.defined() ? api.forward_masked_workspace_bytes(&a) : api.forward_workspace_bytes(&a)) {
    ws = at::empty({(int64_t)need}, opts.dtype(at::kByte));  // stream-ordered memory: free once the launches are enqueued
    a.workspace = ws.data_ptr();
    a.workspace_bytes = need;
  }
  const auto stream = c10::cuda::getCurrentCUDAStream(p.k.device().index()).stream();
  check(mask.defined() ? api.forward_masked(&a, stream) : api.forward(&a, stream), "flare_forward");
  return r;
}

// ---- autograd node ---------------------------------------------------------------------------------------------
struct FlareNode : public torch::autograd::Function<FlareNode> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k,
                                                const Tensor& v, double scale, double power, int64_t variant, int64_t block,
                                                int64_t path, bool want_lse) {
    Problem p{ready(q), ready(k), ready(v), scale, power, (int)variant, (int)block, (int)path};
    Forward r = run_forward(p, State{}, false, want_lse, true);
    ctx->set_materialize_grads(false);  // (else zeros of the log-sum-exps' sizes are made for every backward)
    if (r.keep.defined()) ctx->save_for_backward({q, k, v, r.y, r.lse_dec, r.keep});
    else ctx->save_for_backward({q, k, v});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["power"] = power;
    ctx->saved_data["variant"] = variant;
    ctx->saved_data["block"] = block;
    ctx->saved_data["path"] = path;
    if (!want_lse) return {r.y};
    if (!r.lse_enc.defined()) return {r.y, r.lse_dec};
    ctx->mark_non_differentiable({r.lse_dec, r.lse_enc});
    return {r.y, r.lse_dec, r.lse_enc};
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    torch::autograd::variable_list out(9);
    const auto saved = ctx->get_saved_variables();
    const Tensor &q0 = saved[0], &k0 = saved[1], &v0 = saved[2];
    const c10::cuda::CUDAGuard guard(k0.device());
    if (!grads[0].defined()) {  // an undefined gradient of y stands for zeros
      out[0] = at::zeros(q0.sizes(), q0.options().requires_grad(false));
      out[1] = at::zeros(k0.sizes(), k0.options().requires_grad(false));
      out[2] = at::zeros(v0.sizes(), v0.options().requires_grad(false));
      return out;
    }
    const Problem p{ready(q0), ready(k0), ready(v0), ctx->saved_data["scale"].toDouble(), ctx->saved_data["power"].toDouble(),
                    (int)ctx->saved_data["variant"].toInt(), (int)ctx->saved_data["block"].toInt(),
                    (int)ctx->saved_data["path"].toInt()};
    const Tensor dy = ready(grads[0].scalar_type() == k0.scalar_type() ? grads[0] : grads[0].to(k0.scalar_type()));
    const auto opts = k0.options().requires_grad(false);
    flare_bwd_args_t a;
    memset(&a, 0, sizeof(a));
    fill(a.fwd, p);
    a.dy = dy.data_ptr();
    a.dy_stride_b = dy.stride(0); a.dy_stride_n = dy.stride(1); a.dy_stride_h = dy.stride(2);
    const Tensor dq = at::empty(q0.sizes(), opts), dk = at::empty(k0.sizes(), opts), dv = at::empty(v0.sizes(), opts);
    a.dq = dq.data_ptr(); a.dq_dtype = a.fwd.dtype; a.dk = dk.data_ptr(); a.dv = dv.data_ptr();
    if (saved.size() > 3) {
      const Tensor &y = saved[3], &lse = saved[4], &keep = saved[5];
      a.y = y.data_ptr();
      a.y_stride_b = y.stride(0); a.y_stride_n = y.stride(1); a.y_stride_h = y.stride(2);
      a.lse_dec = lse.data_ptr<float>();
      a.fwd.keep = keep.data_ptr();
      a.fwd.keep_bytes = (size_t)keep.numel();
    }
    Tensor ws;
    if (const size_t need = api.backward_workspace_bytes(&a)) {
      ws = at::empty({(int64_t)need}, opts.dtype(at::kByte));
      a.fwd.workspace = ws.data_ptr();
      a.fwd.workspace_bytes = need;
    }
    check(api.backward(&a, c10::cuda::getCurrentCUDAStream(k0.device().index()).stream()), "flare_backward");
    out[0] = dq;
    out[1] = dk;
    out[2] = dv;
    return out;
  }
};

bool wants_grad(const Tensor& q, const Tensor& k, const Tensor& v) {
  return at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
}

// ---- entry points ------------------------------------------------------------------------------------------------
// token-causal operator, shared decode weights: y, or None
py::object causal(const Tensor& q, const Tensor& k, const Tensor& v, const py::object& scale, int variant, double power) {
  const int path = path_from_env();
  if (path < 0 || !plain_qkv(q, k, v)) return py::none();
  double sc;
  if (!default_scale(scale, k.size(3), &sc)) return py::none();
  const c10::cuda::CUDAGuard guard(k.device());
  if (wants_grad(q, k, v))
    return py::cast(FlareNode::apply(q, k, v, sc, power, (int64_t)variant, (int64_t)1, (int64_t)path, false)[0]);
  const Problem p{ready(q), ready(k), ready(v), sc, power, variant, 1, path};
  return py::cast(run_forward(p, State{}, false, false, false).y);
}

// block-causal operator, shared decode weights: (y, lse_dec, lse_enc), or None
py::object block_causal(const Tensor& q, const Tensor& k, const Tensor& v, const py::object& scale, int64_t block, int64_t chunk) {
  const int path = path_from_env();
  if (path < 0 || !plain_qkv(q, k, v)) return py::none();
  if (block < 16 || block % 16 || k.size(1) % block || (chunk != 16 && chunk != 32 && chunk != 64 && chunk != 128) || block % chunk)
    return py::none();
  double sc;
  if (!default_scale(scale, k.size(3), &sc)) return py::none();
  const c10::cuda::CUDAGuard guard(k.device());
  if (wants_grad(q, k, v)) {
    const auto r = FlareNode::apply(q, k, v, sc, 2.0, (int64_t)FLARE_SOFTMAX, block, (int64_t)path, true);
    return py::make_tuple(r[0], r[1], r[2]);
  }
  const Problem p{ready(q), ready(k), ready(v), sc, 2.0, FLARE_SOFTMAX, (int)block, path};
  const Forward r = run_forward(p, State{}, false, true, false);
  return py::make_tuple(r.y, r.lse_dec, r.lse_enc);
}

// tokens on top of a state (None: empty), shared decode weights: (y, state), or None
py::object prefill(const Tensor& q, const Tensor& k, const Tensor& v, const py::object& state, const py::object& scale,
                   const py::object& mask) {
  const int path = path_from_env();
  double sc;
  if (path < 0 || !plain_qkv(q, k, v) || !to_scale(scale, &sc)) return py::none();
  Tensor valid;
  if (!mask.is_none()) {
    if (!THPVariable_Check(mask.ptr())) return py::none();
    valid = THPVariable_Unpack(mask.ptr());
    if (!ordinary(valid) || valid.device() != k.device() || valid.layout() != at::kStrided || valid.dim() != 2 ||
        valid.size(0) != k.size(0) || valid.size(1) != k.size(1))
      return py::none();
  }
  const c10::cuda::CUDAGuard guard(k.device());
  if (valid.defined()) valid = valid.to(at::kInt).contiguous();
  State in;
  if (!state.is_none() && !plain_state(state, k.size(0), k.size(2), q.size(1), v.size(3), k, &in)) return py::none();
  const Problem p{ready(q), ready(k), ready(v), sc, 2.0, FLARE_SOFTMAX, 1, path};
  const Forward r = run_forward(p, in, true, false, false, valid);
  return py::make_tuple(r.y, state_dict(r.out));
}

// one token on top of a state, which is updated in place: (y [B, 1, H, Dv], state), or None
py::object decode(const Tensor& q, const Tensor& k_in, const Tensor& v_in, const py::object& state, const py::object& scale) {
  // K, V: [B, H, D] or [B, 1, H, D]
  const bool k4 = k_in.dim() == 4 && k_in.size(1) == 1, v4 = v_in.dim() == 4 && v_in.size(1) == 1;
  if (!k_in.is_cuda() || q.dim() != 3 || !(k4 || k_in.dim() == 3) || !(v4 || v_in.dim() == 3)) return py::none();
  if (!same_kind(q, k_in) || !same_kind(v_in, k_in)) return py::none();
  const int dt = dtype_code(k_in.scalar_type());
  const int kh = k4 ? 2 : 1, vh = v4 ? 2 : 1;  // position of the head dimension
  const int64_t B = k_in.size(0), H = k_in.size(kh), Dk = k_in.size(kh + 1), M = q.size(1), Dv = v_in.size(vh + 1);
  if (dt < 0 || B == 0 || v_in.size(0) != B || v_in.size(vh) != H || q.size(0) != H || q.size(2) != Dk) return py::none();
  double sc;
  if (!to_scale(scale, &sc)) return py::none();
  if (k_in.stride(kh + 1) != 1 || v_in.stride(vh + 1) != 1 || !readable(q)) return py::none();
  const c10::cuda::CUDAGuard guard(k_in.device());
  State st;
  if (!plain_state(state, B, H, M, Dv, k_in, &st)) return py::none();
  const Tensor y = at::empty({B, 1, H, Dv}, k_in.options().requires_grad(false));
  flare_decode_args_t a;
  memset(&a, 0, sizeof(a));
  a.q = q.data_ptr(); a.k = k_in.data_ptr(); a.v = v_in.data_ptr(); a.y = y.data_ptr();
  a.state = pointers(st);
  a.B = (int32_t)B; a.H = (int32_t)H; a.M = (int32_t)M; a.Dk = (int32_t)Dk; a.Dv = (int32_t)Dv;
  a.q_stride_h = q.stride(0); a.q_stride_m = q.stride(1);
  a.k_stride_b = k_in.stride(0); a.k_stride_h = k_in.stride(kh);
  a.v_stride_b = v_in.stride(0); a.v_stride_h = v_in.stride(vh);
  a.scale = (float)sc;
  a.dtype = dt;
  const int rc = api.decode_step(&a, c10::cuda::getCurrentCUDAStream(k_in.device().index()).stream());
  if (rc == FLARE_ERR_UNSUPPORTED) return py::none();  // value width outside the streaming kernel: general walk
  check(rc, "flare_decode_step");
  return py::make_tuple(y, state_dict(st));
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.def("bind", &bind);
  m.def("causal", &causal);
  m.def("block_causal", &block_causal);
  m.def("prefill", &prefill);
  m.def("decode", &decode);
}
