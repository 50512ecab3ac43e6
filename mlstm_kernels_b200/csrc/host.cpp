// Host side of the PyTorch functions as a CPython module (_host.so): argument checks, output and scratch allocation,
// autograd node and launch of one call, without a Python frame in between.
//
// A decode step is 4.5 us of GPU time and a short prompt's forward some 20 us; checks, allocations and a
// foreign-function call made from Python cost 15 us a step, 86 us a forward and 260 us a forward + backward, so the
// GPU sat idle.  Here the whole call is native: tensors come straight from their Python objects, outputs from the
// caching allocator (one scratch block per call, carved here), and the backward runs as a C++ autograd node that needs
// no interpreter lock.  Signatures, defaults, return conventions and exception types are those of the Python wrappers
// (chunkwise.py, recurrent.py), which hand over to this module; the operands' sizes and memory are checked before anything
// touches the device.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <cstdlib>
#include <cstring>

#include "calls.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

int dtype_code(at::ScalarType t) {   // -1: not a kernel element type
  switch (t) {
    case at::kFloat: return MLSTM_F32;
    case at::kBFloat16: return MLSTM_BF16;
    case at::kHalf: return MLSTM_F16;
    default: return -1;
  }
}
at::ScalarType code_dtype(int code) {
  return code == MLSTM_F32 ? at::kFloat : code == MLSTM_BF16 ? at::kBFloat16 : at::kHalf;
}

const char* const kNeedsCuda = "mlstm_kernels_b200 kernels run on CUDA tensors only (there is no CPU fallback)";

Tensor empty(at::IntArrayRef size, at::ScalarType dt, const at::Device& dev) {
  return Tensor(at::detail::empty_cuda(size, dt, dev, std::nullopt));
}
Tensor conform(const Tensor& t, at::ScalarType dt) {
  if (t.scalar_type() != dt) return t.to(dt).contiguous();
  return t.is_contiguous() ? t : t.contiguous();
}
Tensor f32c(const Tensor& t) { return t.defined() ? conform(t, at::kFloat) : t; }
const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
const float* fptr(const Tensor& t) { return static_cast<const float*>(ptr(t)); }
float* fout(const Tensor& t) { return t.defined() ? static_cast<float*>(t.mutable_data_ptr()) : nullptr; }
void* current_stream(const at::Device& dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

void check(int rc, const char* what) {
  if (rc == MLSTM_OK) return;
  std::string msg = std::string(what) + ": " + mlstm_b200_error_string(rc);
  if (rc == MLSTM_ERR_CUDA) TORCH_CHECK(false, msg, ": ", mlstm_b200_last_cuda_error());
  C10_THROW_ERROR(ValueError, msg);
}

size_t up256(size_t n) { return (n + 255) / 256 * 256; }
Tensor bytes(size_t n, const at::Device& dev) { return empty({(int64_t)std::max<size_t>(n, 256)}, at::kByte, dev); }
// `need` bytes, and behind them (from up256(need)) `extra` that only make the call faster: where memory is too short for both,
// extra becomes 0 and the call does without.  (Asked for last: what a call allocates after it would have to fit beside the extra.)
Tensor bytes_and(size_t need, size_t& extra, const at::Device& dev) {
  if (extra > 0) {
    try {
      return bytes(up256(need) + extra, dev);
    } catch (const c10::OutOfMemoryError&) {
      extra = 0;
    }
  }
  return bytes(need, dev);
}

// ---- chunkwise ------------------------------------------------------------------------------------------
PyObject* g_select_chunk_size = nullptr;   // chunkwise.select_chunk_size: the rule of the portable kernels, and its errors
bool g_check_status = false;

struct Problem {   // one chunkwise problem, resolved
  mlstm::CallDims c;
  int NC;
  size_t states_bytes, n_states_bytes, m_states_bytes, inv_den_bytes, fw_bytes;
};

Problem resolve(const Tensor& q, const Tensor& v, const Tensor& i, int L, int variant, int impl, double eps) {
  Problem p{};
  p.c = mlstm::CallDims{(int)q.size(0), (int)q.size(1), (int)q.size(2), (int)q.size(3), (int)v.size(3), L,
                        dtype_code(q.scalar_type()), dtype_code(i.scalar_type()), variant, impl, (float)eps, nullptr};
  const auto& c = p.c;
  if (c.dtype < 0 || c.gate_dtype < 0)
    C10_THROW_ERROR(ValueError, c10::str("Unsupported kernel dtype ", c.dtype < 0 ? q.dtype() : i.dtype(), "."));
  p.NC = (c.S + L - 1) / L;
  const size_t bnh = (size_t)c.B * c.NH;
  const size_t sel = mlstm_b200_chunkwise_state_dtype(c.S, c.DHQK, c.DHHV, L, c.dtype, impl) == MLSTM_F32 ? 4 : 2;
  p.states_bytes = bnh * (p.NC + 1) * c.DHQK * c.DHHV * sel;
  p.n_states_bytes = bnh * (p.NC + 1) * c.DHQK * 4;
  p.m_states_bytes = bnh * (p.NC + 1) * 4;
  p.inv_den_bytes = up256(bnh * p.NC * L * 4);
  p.fw_bytes = up256(mlstm_b200_chunkwise_workspace_bytes(c.B, c.NH, c.S, c.DHQK, c.DHHV, L, c.dtype, variant, impl, 0));
  return p;
}


// What a forward leaves behind for its backward: the gate vectors and 1 / (denominator + eps) in one block, and the
// per-chunk states where they are kept.
struct Forward {
  Tensor h, c_last, n_last, m_last, kept, states;
};

// The tensors of a chunkwise call, before anything is launched or allocated for it.  Of the states c and n the kernels read
// as many elements as the sizes say, in memory order; m is one number per (batch, head), however it is shaped.
void check_chunkwise(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& i, const Tensor& f, const Tensor& c0,
                     const Tensor& n0, const Tensor& m0) {
  const auto B = q.size(0), NH = q.size(1), S = q.size(2), DHQK = q.size(3), DHHV = v.size(3);
  const std::array<int64_t, 3> tok_size{B, NH, S};
  const at::IntArrayRef tok(tok_size);
  if (k.sizes() != q.sizes() || v.sizes().slice(0, 3) != tok || i.sizes() != tok || f.sizes() != tok)
    C10_THROW_ERROR(ValueError, "q, k, v, i, f have inconsistent shapes");
  for (const Tensor* t : {&c0, &n0, &m0})
    TORCH_CHECK(!t->defined() || t->is_cuda(), kNeedsCuda);
  if (c0.defined() && c0.numel() < B * NH * DHQK * DHHV)
    C10_THROW_ERROR(ValueError, c10::str("c_initial of shape ", c0.sizes(), " is too small for (B, NH, DHQK, DHHV)"));
  if (n0.defined() && n0.numel() < B * NH * DHQK)
    C10_THROW_ERROR(ValueError, c10::str("n_initial of shape ", n0.sizes(), " is too small for (B, NH, DHQK)"));
  TORCH_CHECK(!m0.defined() || m0.numel() == B * NH, "m_initial: shape '[", B, ", ", NH, "]' is invalid for input of size ", m0.defined() ? m0.numel() : 0);
}

Forward run_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& i_, const Tensor& f_,
                    const Tensor& c0_, const Tensor& n0_, const Tensor& m0_, bool want_last, bool for_backward,
                    bool keep_states, int L, double eps, int variant, int impl) {
  const auto B = q_.size(0), NH = q_.size(1), S = q_.size(2), DHQK = q_.size(3), DHHV = v_.size(3);
  if (k_.scalar_type() != q_.scalar_type() || v_.scalar_type() != q_.scalar_type())
    C10_THROW_ERROR(ValueError, "q, k, v must share one dtype");
  const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous(), i = i_.contiguous();
  const Tensor f = conform(f_, i.scalar_type());
  const Tensor c0 = f32c(c0_), n0 = f32c(n0_), m0 = f32c(m0_);
  Problem p = resolve(q, v, i, L, variant, impl, eps);
  const at::Device dev = q.device();
  Forward out;
  out.h = empty({B, NH, S, DHHV}, q.scalar_type(), dev);
  if (want_last) {
    out.c_last = empty({B, NH, DHQK, DHHV}, at::kFloat, dev);
    out.n_last = empty({B, NH, DHQK}, at::kFloat, dev);
    if (variant == MLSTM_SIG_NONORM) out.n_last.zero_();   // no n without a normaliser: never written
    out.m_last = empty({B, NH, 1}, at::kFloat, dev);
  }
  // one block that dies with this call, one that lives on for the backward; every start 256-byte aligned
  size_t need = up256(p.n_states_bytes) + up256(p.m_states_bytes);
  const size_t states_at = need;
  if (!(for_backward && keep_states)) need += up256(p.states_bytes);
  const size_t ws_at = need;
  if (!for_backward) need += p.fw_bytes;
  size_t scores_bytes = mlstm::score_scratch_bytes(p.c, false);
  const size_t scores_at = up256(need);
  if (for_backward) out.kept = bytes(p.fw_bytes + p.inv_den_bytes, dev);
  if (for_backward && keep_states) out.states = bytes(p.states_bytes, dev);
  const Tensor scratch = bytes_and(need, scores_bytes, dev);
  char* sp = static_cast<char*>(scratch.mutable_data_ptr());
  char* kp = for_backward ? static_cast<char*>(out.kept.mutable_data_ptr()) : nullptr;
  p.c.stream = current_stream(dev);
  const mlstm::FwCall a{
      ptr(q), ptr(k), ptr(v), ptr(i), ptr(f), fptr(c0), fptr(n0), fptr(m0),
      out.h.mutable_data_ptr(), nullptr, nullptr,
      out.states.defined() ? out.states.mutable_data_ptr() : sp + states_at,
      reinterpret_cast<float*>(sp), reinterpret_cast<float*>(sp + up256(p.n_states_bytes)),
      fout(out.c_last), fout(out.n_last), fout(out.m_last),
      for_backward ? reinterpret_cast<float*>(kp + p.fw_bytes) : nullptr,
      for_backward ? kp : sp + ws_at, p.fw_bytes, true, scores_bytes > 0 ? sp + scores_at : nullptr};
  check(mlstm::run_chunkwise_fw(a, p.c), "mlstm_b200_chunkwise_fw");
  return out;
}

class ChunkwiseFn : public torch::autograd::Function<ChunkwiseFn> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& i,
                               const Tensor& f, const std::optional<Tensor>& c0_opt, const std::optional<Tensor>& n0_opt,
                               const std::optional<Tensor>& m0_opt, bool want_last, bool recompute, int64_t L, double eps, int64_t variant, int64_t impl,
                               std::optional<at::ScalarType> cast) {
    const Tensor c0 = c0_opt.value_or(Tensor()), n0 = n0_opt.value_or(Tensor()), m0 = m0_opt.value_or(Tensor());
    // inside an autocast region the inputs are cast and the kernels run with autocast off (torch.amp.custom_fwd)
    auto in = [&](const Tensor& t) { return t.defined() && cast && t.is_floating_point() && t.scalar_type() != at::kDouble ? t.to(*cast) : t; };
    const Tensor qc = in(q), kc = in(k), vc = in(v), ic = in(i), fc = in(f), c0c = in(c0), n0c = in(n0), m0c = in(m0);
    Forward o = run_forward(qc, kc, vc, ic, fc, c0c, n0c, m0c, want_last, true, !recompute, (int)L, eps, (int)variant, (int)impl);
    ctx->save_for_backward({qc, kc, vc, ic, fc, recompute ? c0c : Tensor(), m0c, o.states, o.kept});
    ctx->set_materialize_grads(false);
    auto& d = ctx->saved_data;
    d["cfg"] = std::vector<int64_t>{L, variant, impl, c0.defined() ? (int64_t)c0c.scalar_type() : -1,
                                    n0.defined() ? (int64_t)n0c.scalar_type() : -1, m0.defined() ? 1 : 0};
    d["eps"] = eps;
    if (want_last) return {o.h, o.c_last, o.n_last, o.m_last};
    return {o.h};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const auto cfg = ctx->saved_data["cfg"].toIntVector();
    const double eps = ctx->saved_data["eps"].toDouble();
    const Tensor &i_ = saved[3], &f_ = saved[4], &c0 = saved[5], &m0_ = saved[6], &states = saved[7], &kept = saved[8];
    const Tensor q = saved[0].contiguous(), k = saved[1].contiguous(), v = saved[2].contiguous(), i = i_.contiguous();
    const Tensor f = conform(f_, i.scalar_type()), m0 = f32c(m0_);
    const at::Device dev = q.device();
    c10::cuda::OptionalCUDAGuard guard(dev);
    Problem p = resolve(q, v, i, (int)cfg[0], (int)cfg[1], (int)cfg[2], eps);
    const auto& c = p.c;
    const Tensor dh = grads[0].defined() ? conform(grads[0], q.scalar_type())
                                         : at::zeros({c.B, c.NH, c.S, c.DHHV}, q.options());
    const Tensor dc_last = grads.size() > 1 ? f32c(grads[1]) : Tensor();
    const Tensor dq = empty(q.sizes(), q.scalar_type(), dev), dk = empty(q.sizes(), q.scalar_type(), dev);
    const Tensor dv = empty(v.sizes(), v.scalar_type(), dev);
    const Tensor di = empty(i.sizes(), i.scalar_type(), dev), df = empty(i.sizes(), i.scalar_type(), dev);
    const Tensor dc0 = cfg[3] >= 0 ? empty({c.B, c.NH, c.DHQK, c.DHHV}, at::kFloat, dev) : Tensor();
    const size_t ws_bytes = up256(mlstm_b200_chunkwise_workspace_bytes(c.B, c.NH, c.S, c.DHQK, c.DHHV, c.L, c.dtype, c.variant, c.impl, 1));
    const Tensor rc0 = f32c(c0);
    size_t scores_bytes = mlstm::score_scratch_bytes(c, true);
    const size_t scores_at = up256(ws_bytes + (states.defined() ? 0 : p.states_bytes));
    Tensor ws = bytes_and(scores_at, scores_bytes, dev);
    char* wp = static_cast<char*>(ws.mutable_data_ptr());
    const char* kp = static_cast<const char*>(kept.const_data_ptr());
    p.c.stream = current_stream(dev);
    const mlstm::BwCall a{
        ptr(q), ptr(k), ptr(v), ptr(i), ptr(f), fptr(m0), ptr(states), states.defined() ? nullptr : wp + ws_bytes,
        fptr(rc0), nullptr, reinterpret_cast<const float*>(kp + p.fw_bytes), kp, p.fw_bytes, ptr(dh), fptr(dc_last),
        dq.mutable_data_ptr(), dk.mutable_data_ptr(), dv.mutable_data_ptr(), di.mutable_data_ptr(), df.mutable_data_ptr(),
        c.gate_dtype, fout(dc0), wp, ws_bytes, scores_bytes > 0 ? wp + scores_at : nullptr};
    check(mlstm::run_chunkwise_bw(a, p.c), "mlstm_b200_chunkwise_bw");
    if (g_check_status && mlstm_b200_device_status(1) != 0)
      TORCH_CHECK(false, "mlstm_kernels_b200: a bounded wait of the tcgen05 kernels ran out; results invalid");
    ws.reset();
    Tensor dc0_out, dn0, dm0;
    if (dc0.defined()) dc0_out = dc0.to((at::ScalarType)cfg[3]);
    if (cfg[4] >= 0) dn0 = at::zeros({c.B, c.NH, c.DHQK}, q.options().dtype((at::ScalarType)cfg[4]));
    if (cfg[5]) dm0 = at::zeros_like(m0_);
    return {dq, dk, dv, di, f_.scalar_type() == df.scalar_type() ? df : df.to(f_.scalar_type()), dc0_out, dn0, dm0,
            Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---- Python glue ----------------------------------------------------------------------------------------
struct AssertionFailed { std::string what; };

Tensor arg(PyObject* o, const char* name) {
  if (o == Py_None) return Tensor();
  if (!THPVariable_Check(o)) throw torch::TypeError(c10::str(name, " must be a tensor, got ", Py_TYPE(o)->tp_name));
  return THPVariable_Unpack(o);
}
Tensor need(PyObject* o, const char* name) {
  Tensor t = arg(o, name);
  if (!t.defined()) throw torch::TypeError(c10::str(name, " must be a tensor, got None"));
  return t;
}
at::ScalarType dtype_arg(PyObject* o) {
  if (!THPDtype_Check(o)) throw torch::TypeError(c10::str("expected a torch.dtype, got ", Py_TYPE(o)->tp_name));
  return reinterpret_cast<THPDtype*>(o)->scalar_type;
}
PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
PyObject* state_tuple(PyObject* h, const Tensor& c, const Tensor& n, const Tensor& m) {
  return Py_BuildValue("(N(NNN))", h, wrap(c), wrap(n), wrap(m));
}
double double_arg(PyObject* o) {
  const double x = PyFloat_AsDouble(o);
  if (x == -1.0 && PyErr_Occurred()) throw python_error();
  return x;
}
long long_arg(PyObject* o) {
  const long x = PyLong_AsLong(o);
  if (x == -1 && PyErr_Occurred()) throw python_error();
  return x;
}
bool bool_arg(PyObject* o) {
  const int x = PyObject_IsTrue(o);
  if (x < 0) throw python_error();
  return x != 0;
}
void nargs_are(Py_ssize_t have, Py_ssize_t want) {
  if (have != want) throw torch::TypeError(c10::str("expected ", want, " arguments, got ", have));
}

// chunkwise(q, k, v, i, f, c0, n0, m0, return_last_states, eps, chunk_size, impl, recompute, cast_dtype, variant)
//   -> (h, c_last, n_last, m_last), the last three None without return_last_states
PyObject* py_chunkwise(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  nargs_are(n, 15);
  const Tensor q = need(a[0], "q"), k = need(a[1], "k"), v = need(a[2], "v"), i = need(a[3], "i"), f = need(a[4], "f");
  const Tensor c0 = arg(a[5], "c_initial"), n0 = arg(a[6], "n_initial"), m0 = arg(a[7], "m_initial");
  const bool want_last = bool_arg(a[8]), recompute = bool_arg(a[12]);
  const double eps = double_arg(a[9]);
  const char* impl_name = PyUnicode_Check(a[11]) ? PyUnicode_AsUTF8(a[11]) : "?";
  if (impl_name == nullptr) { PyErr_Clear(); impl_name = "?"; }   // text that has no UTF-8 form
  const int impl = !strcmp(impl_name, "auto") ? MLSTM_IMPL_AUTO : !strcmp(impl_name, "simt") ? MLSTM_IMPL_SIMT
                   : !strcmp(impl_name, "tcgen05") ? MLSTM_IMPL_TCGEN05 : -1;
  if (impl < 0) { PyErr_SetObject(PyExc_KeyError, a[11]); throw python_error(); }
  const at::ScalarType kdt = dtype_arg(a[13]);
  const int variant = (int)long_arg(a[14]);
  if (dtype_code(kdt) < 0) C10_THROW_ERROR(ValueError, c10::str("Unsupported kernel dtype ", kdt, "."));
  for (const Tensor* t : {&q, &k, &v, &i, &f})
    TORCH_CHECK(t->is_cuda(), kNeedsCuda);
  if (q.dim() != 4 || v.dim() != 4) C10_THROW_ERROR(ValueError, "q, k, v, i, f have inconsistent shapes");
  check_chunkwise(q, k, v, i, f, c0, n0, m0);
  // a forward-mode tangent would be dropped without a word
  for (const Tensor* t : {&q, &k, &v, &i, &f, &c0, &n0, &m0})
    if (t->defined() && t->_fw_grad(0).defined())
      C10_THROW_ERROR(NotImplementedError, "mlstm_kernels_b200 has no forward-mode derivative of the chunkwise functions");
  std::optional<at::ScalarType> cast;
  if (at::autocast::is_autocast_enabled(at::kCUDA)) cast = kdt;
  const at::ScalarType qdt = cast && q.scalar_type() != at::kDouble ? *cast : q.scalar_type();

  // Chunk size: 128 wherever the tcgen05 kernels run, else the portable kernels' rule
  int64_t L = 128;
  const int code = dtype_code(qdt);
  if (code < 0 || impl == MLSTM_IMPL_SIMT ||
      !mlstm_b200_chunkwise_has_tcgen05((int)q.size(2), (int)q.size(3), (int)v.size(3), 128, code)) {
    PyObject* r = PyObject_CallFunction(g_select_chunk_size, "LO", (long long)q.size(2), a[10]);
    if (r == nullptr) throw python_error();
    L = PyLong_AsLong(r);
    Py_DECREF(r);
  }
  const bool grad = at::GradMode::is_enabled() &&
                    (q.requires_grad() || k.requires_grad() || v.requires_grad() || i.requires_grad() || f.requires_grad() ||
                     (c0.defined() && c0.requires_grad()) || (n0.defined() && n0.requires_grad()) || (m0.defined() && m0.requires_grad()));
  Tensor h, c, nn, m;
  {
    pybind11::gil_scoped_release no_gil;
    c10::cuda::OptionalCUDAGuard guard(q.device());
    const bool was_on = cast.has_value();
    if (was_on) at::autocast::set_autocast_enabled(at::kCUDA, false);
    struct Restore { bool on; ~Restore() { if (on) at::autocast::set_autocast_enabled(at::kCUDA, true); } } restore{was_on};
    if (grad) {
      auto given = [](const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; };
      auto out = ChunkwiseFn::apply(q, k, v, i, f, given(c0), given(n0), given(m0), want_last, recompute, L, eps, (int64_t)variant, (int64_t)impl, cast);
      h = out[0];
      if (want_last) { c = out[1]; nn = out[2]; m = out[3]; }
    } else {
      at::AutoDispatchBelowADInplaceOrView below;
      auto in = [&](const Tensor& t) { return t.defined() && cast && t.is_floating_point() && t.scalar_type() != at::kDouble ? t.to(*cast) : t; };
      Forward o = run_forward(in(q), in(k), in(v), in(i), in(f), in(c0), in(n0), in(m0), want_last, false, false, (int)L, eps, variant, impl);
      h = o.h; c = o.c_last; nn = o.n_last; m = o.m_last;
    }
  }
  return Py_BuildValue("(NNNN)", wrap(h), wrap(c), wrap(nn), wrap(m));
  END_HANDLE_TH_ERRORS
}

std::string shape_text(const Tensor& t) { return c10::str("torch.Size(", t.sizes(), ")"); }

// step(c, n, m, q, k, v, i, f, c_new, n_new, m_new, eps, dtype_state, h_out) -> (h, (c_new, n_new, m_new))
PyObject* py_step(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  nargs_are(n_args, 14);
  try {
    Tensor c = need(a[0], "matC_old"), n = need(a[1], "vecN_old"), m = need(a[2], "scaM_old");
    Tensor q = need(a[3], "vecQ"), k = need(a[4], "vecK"), v = need(a[5], "vecV"), gi = need(a[6], "scaI"), gf = need(a[7], "scaF");
    Tensor cn = arg(a[8], "matC_new"), nn = arg(a[9], "vecN_new"), mn = arg(a[10], "scaM_new"), h = arg(a[13], "vecH_out");
    const double eps = double_arg(a[11]);
    const at::ScalarType sdt = dtype_arg(a[12]);
    for (const Tensor* t : {&q, &k, &v, &gi, &gf, &c, &n, &m, &cn, &nn, &mn, &h})
      TORCH_CHECK(!t->defined() || t->is_cuda(), kNeedsCuda);
    if (q.dim() != 3) throw AssertionFailed{"q must have shape (B, NH, DHQK)"};
    const auto B = q.size(0), NH = q.size(1), DHQK = q.size(2), DHHV = v.size(-1);
    const std::array<int64_t, 3> one_size{B, NH, 1};
    const at::IntArrayRef one(one_size);
    if (k.sizes() != q.sizes()) throw AssertionFailed{"q and k must have the same shape"};
    if (v.numel() < B * NH * DHHV) throw AssertionFailed{"vecV has wrong shape, got " + shape_text(v)};
    if (c.sizes() != at::IntArrayRef{B, NH, DHQK, DHHV}) throw AssertionFailed{"matC_old has wrong shape, got " + shape_text(c)};
    if (n.sizes() != q.sizes()) throw AssertionFailed{"vecN_old has wrong shape, got " + shape_text(n)};
    if (m.sizes() != one) throw AssertionFailed{"scaM_old has wrong shape, got " + shape_text(m)};
    if (gi.sizes() != one) throw AssertionFailed{"scaI has wrong shape, got " + shape_text(gi)};
    if (gf.sizes() != one) throw AssertionFailed{"scaF has wrong shape, got " + shape_text(gf)};
    if (sdt != at::kFloat && sdt != at::kBFloat16) C10_THROW_ERROR(ValueError, c10::str("Unsupported state dtype ", sdt, "."));
    const at::ScalarType qdt = q.scalar_type();
    const int dt = dtype_code(qdt);
    if (dt < 0) C10_THROW_ERROR(ValueError, c10::str("Unsupported kernel dtype ", qdt, "."));
    at::NoGradGuard no_grad;   // the step has no gradient: conversions of its inputs need none either
    q = conform(q, qdt); k = conform(k, qdt); v = conform(v, qdt);
    gi = conform(gi, dtype_code(gi.scalar_type()) < 0 ? at::kFloat : gi.scalar_type());
    gf = conform(gf, gi.scalar_type());
    c = conform(c, sdt); n = conform(n, sdt); m = conform(m, sdt);
    const at::Device dev = q.device();
    if (!cn.defined()) {
      if (nn.defined() || mn.defined()) throw AssertionFailed{"Initial states must be provided together."};
      cn = empty(c.sizes(), sdt, dev); nn = empty(n.sizes(), sdt, dev); mn = empty(one, sdt, dev);
    } else {
      if (!nn.defined() || !mn.defined()) throw AssertionFailed{"Initial states must be provided together."};
      for (const Tensor* t : {&cn, &nn, &mn})
        if (t->scalar_type() != sdt || !t->is_contiguous())
          C10_THROW_ERROR(ValueError, "output state tensors must be contiguous and of dtype_state");
      if (cn.numel() < c.numel() || nn.numel() < n.numel() || mn.numel() < m.numel())
        C10_THROW_ERROR(ValueError, "output state tensors are too small for the states");
    }
    if (!h.defined()) {
      h = empty(v.sizes(), qdt, dev);
    } else if (h.scalar_type() != qdt || h.sizes() != v.sizes() || !h.is_contiguous()) {
      C10_THROW_ERROR(ValueError, "vecH_out must be a contiguous (B, NH, DHHV) tensor of q's dtype");
    }
    int rc;
    {
      pybind11::gil_scoped_release no_gil;
      c10::cuda::OptionalCUDAGuard guard(dev);
      rc = mlstm_b200_step(ptr(q), ptr(k), ptr(v), ptr(gi), ptr(gf), ptr(c), ptr(n), ptr(m), h.mutable_data_ptr(),
                           cn.mutable_data_ptr(), nn.mutable_data_ptr(), mn.mutable_data_ptr(), (int)B, (int)NH, (int)DHQK,
                           (int)DHHV, dt, dtype_code(gi.scalar_type()), dtype_code(sdt), (float)eps, current_stream(dev));
    }
    check(rc, "mlstm_b200_step");
    return state_tuple(wrap(h), cn, nn, mn);
  } catch (const AssertionFailed& e) {
    PyErr_SetString(PyExc_AssertionError, e.what.c_str());
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// sequence(q, k, v, i, f, c0, n0, m0, eps, dtype_state) -> (h, (c, n, m))
PyObject* py_sequence(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  nargs_are(n_args, 10);
  Tensor q = need(a[0], "q"), k = need(a[1], "k"), v = need(a[2], "v"), gi = need(a[3], "i"), gf = need(a[4], "f");
  Tensor c0 = arg(a[5], "c_initial"), n0 = arg(a[6], "n_initial"), m0 = arg(a[7], "m_initial");
  const double eps = double_arg(a[8]);
  const at::ScalarType sdt = dtype_arg(a[9]);
  for (const Tensor* t : {&q, &k, &v, &gi, &gf, &c0, &n0, &m0}) TORCH_CHECK(!t->defined() || t->is_cuda(), kNeedsCuda);
  if (q.dim() != 4) C10_THROW_ERROR(ValueError, "q must have shape (B, NH, S, DHQK)");
  const auto B = q.size(0), NH = q.size(1), S = q.size(2), DHQK = q.size(3), DHHV = v.size(-1);
  // the kernel reads operands of these sizes in memory order, however they are shaped
  auto fits = [](const Tensor& t, int64_t n) { return !t.defined() || t.numel() >= n; };
  if (!fits(k, q.numel()) || !fits(v, B * NH * S * DHHV) || !fits(gi, B * NH * S) || !fits(gf, B * NH * S))
    C10_THROW_ERROR(ValueError, "q, k, v, i, f have inconsistent shapes");
  if (!fits(c0, B * NH * DHQK * DHHV) || !fits(n0, B * NH * DHQK) || !fits(m0, B * NH))
    C10_THROW_ERROR(ValueError, "c_initial, n_initial or m_initial is too small for the sizes of q and v");
  const int dt = dtype_code(q.scalar_type());
  if (dt < 0) C10_THROW_ERROR(ValueError, c10::str("Unsupported kernel dtype ", q.scalar_type(), "."));
  at::NoGradGuard no_grad;
  q = q.contiguous(); k = conform(k, q.scalar_type()); v = conform(v, q.scalar_type());
  gi = conform(gi, dtype_code(gi.scalar_type()) < 0 ? at::kFloat : gi.scalar_type());
  gf = conform(gf, gi.scalar_type());
  c0 = f32c(c0); n0 = f32c(n0); m0 = f32c(m0);
  const at::Device dev = q.device();
  const Tensor h = empty(v.sizes(), v.scalar_type(), dev), c = empty({B, NH, DHQK, DHHV}, at::kFloat, dev);
  const Tensor n = empty({B, NH, DHQK}, at::kFloat, dev), m = empty({B, NH, 1}, at::kFloat, dev);
  int rc;
  {
    pybind11::gil_scoped_release no_gil;
    c10::cuda::OptionalCUDAGuard guard(dev);
    rc = mlstm_b200_step_sequence(ptr(q), ptr(k), ptr(v), ptr(gi), ptr(gf), fptr(c0), fptr(n0), fptr(m0),
                                  h.mutable_data_ptr(), fout(c), fout(n), fout(m), (int)B, (int)NH, (int)S, (int)DHQK,
                                  (int)DHHV, dt, dtype_code(gi.scalar_type()), (float)eps, current_stream(dev));
  }
  check(rc, "mlstm_b200_step_sequence");
  if (sdt == at::kFloat) return state_tuple(wrap(h), c, n, m);
  return state_tuple(wrap(h), c.to(sdt), n.to(sdt), m.to(sdt));
  END_HANDLE_TH_ERRORS
}

// setup(select_chunk_size): once, when the package is first used
PyObject* py_setup(PyObject*, PyObject* fn) {
  Py_XDECREF(g_select_chunk_size);
  Py_INCREF(fn);
  g_select_chunk_size = fn;
  const char* e = getenv("MLSTM_B200_CHECK_STATUS");
  g_check_status = e != nullptr && !strcmp(e, "1");
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"chunkwise", (PyCFunction)(void (*)(void))py_chunkwise, METH_FASTCALL, nullptr},
    {"step", (PyCFunction)(void (*)(void))py_step, METH_FASTCALL, nullptr},
    {"sequence", (PyCFunction)(void (*)(void))py_sequence, METH_FASTCALL, nullptr},
    {"setup", py_setup, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&kModule); }
