// The autograd entry points' native route: attention on ordinary torch tensors, forward and backward, without Python in
// between.  Outputs, gradients and scratch come from torch's caching allocator, launches go to torch's current stream
// through the C++ operator API (include/aotriton/flash.h), the backward is a torch::autograd::Function: version checks and CUDA-graph
// capture see what they see of the Python Function, saved-tensor hooks the inputs, the output and the log-sum-exp.
//
// What bounds a small call is the host.  Measured, us a pass, the Python way against this: training step of 2 x 4 heads x 128 tokens of 64 (20
// of kernels) 160 / 77; cross attention, 4 x 8 heads x 1024 x 77 of 80 (47 of kernels), 332 / 78; one token of 4 sequences against 6007
// keys, 32:8 heads of 128 (14), 33.5 / 20.6.
//
// attend() returns None for whatever is not ordinary, and the caller then goes the Python way: tensors that are not plain CUDA tensors of
// one type on the current device with unit innermost stride, and every mode in which an operator call means more than its kernels
// (dispatch and function modes, functorch transforms, forward-mode gradients, tracing).  The backward asks the same of its
// gradient, of what was saved and of the modes it runs under, and otherwise leaves itself to the operator or to the Python Function's.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <aotriton/flash.h>
#include <aotriton/util.h>
#include <aotriton_b200.h>

#include <atomic>
#include <string>

namespace aotriton = AOTRITON_NS;
namespace flash = AOTRITON_NS::v3::flash;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

// Kernel family of the most recent backward: the library keeps it per thread, and autograd runs backwards on a thread of
// its own.
std::atomic<int> g_last_bwd_family{0};

// The Function's backward as Python has it (autograd.py), for what Attend::backward leaves to it.  Set once, at import.
PyObject* g_python_backward = nullptr;

// A call's numbers.  `packed`: token-packed sequences (cu_q, cu_k); `op`: the call stands for the registered operators, whose
// backward may use the fused form and is itself an operator.
struct Call {
  double sm_scale, dropout_p;
  int64_t causal_type, left, right, max_q, max_k;
  uint64_t seed, offset;      // of the dropout; offset is the whole of it
  bool packed, op;
};

aotriton::DType dtype_of(at::ScalarType t) {
  return t == at::kFloat ? aotriton::kFloat32 : (t == at::kHalf ? aotriton::kFloat16 : aotriton::kBFloat16);
}
template <int Rank>
aotriton::TensorView<Rank> view_of(const Tensor& t, aotriton::DType dt) {
  std::array<uint64_t, Rank> n, s;
  for (int i = 0; i < Rank; ++i) { n[i] = (uint64_t)t.size(i); s[i] = (uint64_t)t.stride(i); }
  return aotriton::TensorView<Rank>(reinterpret_cast<intptr_t>(t.data_ptr()), n, s, dt);
}
aotriton::TensorView<4> view_or_null(const Tensor& t, aotriton::DType dt) {
  return t.defined() ? view_of<4>(t, dt) : aotriton::TensorView<4>(0, {}, {}, dt);
}
Tensor fresh(at::IntArrayRef sizes, at::ScalarType dt) {
  return at::detail::empty_cuda(sizes, dt, c10::Device(c10::kCUDA, c10::cuda::current_device()), std::nullopt);
}
// torch.empty_like: the tensor's strides where they are dense
Tensor gradient_of(const Tensor& t) { return t.is_contiguous() ? fresh(t.sizes(), t.scalar_type()) : at::empty_like(t); }

void check(hipError_t e, const char* what) {
  if (e == hipSuccess) return;
  const char* name = e == hipErrorInvalidValue ? "hipErrorInvalidValue" : e == hipErrorNoBinaryForGpu ? "hipErrorNoBinaryForGpu"
                     : e == hipErrorNotSupported ? "hipErrorNotSupported" : e == hipErrorLaunchFailure ? "hipErrorLaunchFailure"
                                                                                                       : nullptr;
  throw std::runtime_error(std::string(what) + " failed: " + (name ? std::string("hipError_t.") + name : std::to_string((int)e)));
}

template <typename P>
void fill_common(P& p, const Call& c, const Tensor& cu_q, const Tensor& cu_k, const Tensor& seed) {
  p.Sm_scale = (float)c.sm_scale;
  p.dropout_p = (float)c.dropout_p;
  p.philox_seed_ptr = aotriton::TensorView<0>(seed.defined() ? reinterpret_cast<intptr_t>(seed.data_ptr()) : 0, aotriton::kUInt64);
  p.philox_offset1 = aotriton::TensorView<0>(0, aotriton::kUInt64);
  p.philox_offset2 = c.offset;
  p.causal_type = (int8_t)c.causal_type;
  p.window_left = (int32_t)c.left;
  p.window_right = (int32_t)c.right;
  p.varlen_type = c.packed ? AB200_VARLEN_COMPACT : AB200_VARLEN_NONE;
  if (c.packed) {
    p.cu_seqlens_q = view_of<1>(cu_q, aotriton::kInt32);
    p.cu_seqlens_k = view_of<1>(cu_k, aotriton::kInt32);
    p.Max_seqlen_q = (int32_t)c.max_q;
    p.Max_seqlen_k = (int32_t)c.max_k;
  }
}

aotriton::Stream current_stream() { return aotriton::Stream(c10::cuda::getCurrentCUDAStream().stream()); }

// `lse` is left undefined where nobody will read it.
void forward(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& cu_q, const Tensor& cu_k,
             bool want_lse, Tensor& out, Tensor& lse, Tensor& seed) {
  at::AutoDispatchBelowADInplaceOrView guard;
  const aotriton::DType dt = dtype_of(q.scalar_type());
  if (c.packed) {      // (1, H, tokens, D) views of (tokens, H, D) storage
    out = fresh({1, q.size(2), q.size(1), v.size(3)}, q.scalar_type()).transpose(1, 2);
    if (want_lse) lse = fresh({q.size(1), q.size(2)}, at::kFloat);
  } else {
    out = fresh({q.size(0), q.size(1), q.size(2), v.size(3)}, q.scalar_type());
    if (want_lse) lse = fresh({q.size(0) * q.size(1), q.size(2)}, at::kFloat);
  }
  // one fill on the stream; the offset goes by value
  if (c.dropout_p > 0) seed = at::full({1}, (int64_t)c.seed, out.options().dtype(at::kLong));
  flash::attn_fwd_params p;
  p.Q = view_of<4>(q, dt); p.K = view_of<4>(k, dt); p.V = view_of<4>(v, dt); p.B = view_or_null(b, dt); p.Out = view_of<4>(out, dt);
  p.L = want_lse ? view_of<2>(lse, aotriton::kFloat32) : aotriton::TensorView<2>(0, {}, {}, aotriton::kFloat32);
  p.encoded_softmax = aotriton::TensorView<4>(0, {}, {}, dt);
  fill_common(p, c, cu_q, cu_k, seed);
  check(flash::attn_fwd(p, flash::attn_fwd_params::kVersion, current_stream(), nullptr), c.packed ? "attn_fwd (varlen)" : "attn_fwd");
}

// The fp32 dQ accumulator of the fused form, made when the backward asks for it.
struct DqAcc {
  const Tensor* dq;
  Tensor acc;
  static aotriton::TensorView<4> acquire(aotriton::LazyTensor<4>* self) {
    auto* a = static_cast<DqAcc*>(self->cookie);
    a->acc = at::zeros(a->dq->sizes(), a->dq->options().dtype(at::kFloat));
    return view_of<4>(a->acc, aotriton::kFloat32);
  }
};

bool plain_modes() {
  const auto& tls = c10::impl::tls_local_dispatch_key_set();
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled() && !torch::jit::tracer::isTracing() &&
         !tls.included_.has(c10::DispatchKey::Python) && !tls.included_.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !tls.included_.has(c10::DispatchKey::Functionalize);
}

// Nothing but a strided CUDA tensor on device `dev`, with elements, without a forward-mode gradient.
bool plain(const Tensor& t, int dev) {
  static const uint64_t allowed =
      (c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
       c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) | c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)).raw_repr();
  return t.defined() && (t.key_set().raw_repr() & ~allowed) == 0 && t.is_cuda() && t.get_device() == dev && t.layout() == at::kStrided &&
         t.numel() != 0 && !t._fw_grad(0).defined();
}
// ... of this type and rank, with a unit innermost stride
bool plain_operand(const Tensor& t, int dev, at::ScalarType type, int64_t dim) {
  return plain(t, dev) && t.scalar_type() == type && t.dim() == dim && t.stride(-1) == 1;
}

struct Attend : torch::autograd::Function<Attend> {
  using Maybe = std::optional<Tensor>;      // (an undefined Tensor is no argument to apply())
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Maybe& bias,
                               const Maybe& seqs_q, const Maybe& seqs_k, const Call& c, bool return_lse) {
    const Tensor b = bias.value_or(Tensor()), cu_q = seqs_q.value_or(Tensor()), cu_k = seqs_k.value_or(Tensor());
    Tensor out, lse, seed;
    ::forward(c, q, k, v, b, cu_q, cu_k, true, out, lse, seed);
    ctx->save_for_backward({q, k, v, b, out, lse, cu_q, cu_k});
    if (seed.defined()) ctx->saved_data["seed"] = seed;      // (a number of the call, nothing for a saved-tensor hook to change)
    ctx->saved_data["numbers"] = std::vector<int64_t>{c.causal_type, c.left, c.right, c.max_q, c.max_k, (int64_t)c.seed,
                                                      (int64_t)c.offset, c.packed, c.op};
    ctx->saved_data["scales"] = std::vector<double>{c.sm_scale, c.dropout_p};
    ctx->set_materialize_grads(false);
    return return_lse ? variable_list{out, lse} : variable_list{out};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2], &b = saved[3], &out = saved[4], &lse = saved[5], &cu_q = saved[6], &cu_k = saved[7];
    const auto found = ctx->saved_data.find("seed");
    const Tensor seed = found == ctx->saved_data.end() ? Tensor() : found->second.toTensor();
    const auto n = ctx->saved_data["numbers"].toIntVector();
    const auto s = ctx->saved_data["scales"].toDoubleVector();
    const Call c{s[0], s[1], n[0], n[1], n[2], n[3], n[4], (uint64_t)n[5], (uint64_t)n[6], n[7] != 0, n[8] != 0};
    variable_list r(8);
    Tensor dout = grads[0].defined() ? grads[0] : at::zeros_like(out);
    // create_graph: the operator, which knows that it has no derivative
    if (c.op && at::GradMode::is_enabled()) {
      operator_backward(c, q, k, v, b, out, dout, lse, seed, r);
      return r;
    }
    // A gradient that is not an ordinary tensor (a batch of them under vmap), a mode that only this pass runs under, or a saved-tensor
    // hook that handed back something else than it was given: what the call stands for deals with it.
    if (!as_saved(q, k, v, b, out, dout, lse, cu_q, cu_k)) {
      if (c.op) operator_backward(c, q, k, v, b, out, dout, lse, seed, r);
      else python_backward(c, q, k, v, b, out, dout, lse, cu_q, cu_k, seed, r);
      return r;
    }
    if (dout.stride(-1) != 1) dout = dout.contiguous();
    const aotriton::DType dt = dtype_of(q.scalar_type());
    r[0] = gradient_of(q);
    r[1] = gradient_of(k);
    r[2] = gradient_of(v);
    if (b.defined()) r[3] = gradient_of(b);
    const Tensor delta = fresh(lse.sizes(), at::kFloat);
    DqAcc acc{&r[0], {}};
    flash::attn_options options;
    flash::attn_bwd_params p;
    p.Q = view_of<4>(q, dt); p.K = view_of<4>(k, dt); p.V = view_of<4>(v, dt); p.B = view_or_null(b, dt);
    p.Out = view_of<4>(out, dt); p.DO = view_of<4>(dout, dt);
    p.DQ = view_of<4>(r[0], dt); p.DK = view_of<4>(r[1], dt); p.DV = view_of<4>(r[2], dt); p.DB = view_or_null(r[3], dt);
    p.L = view_of<2>(lse, aotriton::kFloat32);
    p.D.eager = view_of<2>(delta, aotriton::kFloat32);
    if (c.op) {
      options.deterministic = at::globalContext().deterministicAlgorithms();
      p.DQ_ACC.cookie = &acc;
      p.DQ_ACC.acquire = &DqAcc::acquire;
    }
    fill_common(p, c, cu_q, cu_k, seed);
    check(flash::attn_bwd(p, flash::attn_bwd_params::kVersion, current_stream(), &options), c.packed ? "attn_bwd (varlen)" : "attn_bwd");
    g_last_bwd_family.store(ab200_last_bwd_family(), std::memory_order_relaxed);
    return r;
  }

  static bool as_saved(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& out, const Tensor& dout,
                       const Tensor& lse, const Tensor& cu_q, const Tensor& cu_k) {
    if (!plain_modes()) return false;
    const int dev = c10::cuda::current_device();
    const auto type = q.scalar_type();
    for (const Tensor* t : {&q, &k, &v, &out})
      if (!plain_operand(*t, dev, type, 4)) return false;
    for (const Tensor* t : {&cu_q, &cu_k})
      if (t->defined() && !plain_operand(*t, dev, at::kInt, 1)) return false;
    return (!b.defined() || plain_operand(b, dev, type, 4)) && plain_operand(lse, dev, at::kFloat, 2) && lse.is_contiguous() &&
           lse.numel() == q.size(0) * q.size(1) * q.size(2) && plain(dout, dev) && dout.scalar_type() == type && dout.sizes() == out.sizes();
  }

  static void python_backward(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& out,
                              const Tensor& dout, const Tensor& lse, const Tensor& cu_q, const Tensor& cu_k, const Tensor& seed,
                              variable_list& r) {
    pybind11::gil_scoped_acquire gil;
    auto wrap = [](const Tensor& t) {
      return t.defined() ? pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(t)) : pybind11::object(pybind11::none());
    };
    const pybind11::object t[] = {wrap(q), wrap(k), wrap(v), wrap(b), wrap(out), wrap(dout), wrap(lse), wrap(cu_q), wrap(cu_k), wrap(seed)};
    const auto result = pybind11::reinterpret_steal<pybind11::object>(PyObject_CallFunction(
        g_python_backward, "OOOOOOOOOOKddLLLLL", t[0].ptr(), t[1].ptr(), t[2].ptr(), t[3].ptr(), t[4].ptr(), t[5].ptr(), t[6].ptr(), t[7].ptr(),
        t[8].ptr(), t[9].ptr(), (unsigned long long)c.offset, c.sm_scale, c.dropout_p, (long long)c.causal_type, (long long)c.left,
        (long long)c.right, (long long)c.max_q, (long long)c.max_k));
    if (!result) {
      python_error e;
      e.persist();
      throw e;
    }
    for (int i = 0; i < (b.defined() ? 4 : 3); ++i) r[i] = THPVariable_Unpack(PyTuple_GET_ITEM(result.ptr(), i));
  }

  static void operator_backward(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& out,
                                const Tensor& dout, const Tensor& lse, const Tensor& seed, variable_list& r) {
    const auto one = lse.options().dtype(at::kLong);
    const Tensor sd = (seed.defined() ? seed : at::zeros({1}, one)).view(at::kUInt64);
    const Tensor off = at::full({1}, (int64_t)(c.dropout_p > 0 ? c.offset : 0), one).view(at::kUInt64);
    torch::jit::Stack stack;
    for (const Tensor& t : {q, k, v}) stack.emplace_back(t);
    stack.emplace_back(b.defined() ? c10::IValue(b) : c10::IValue());
    for (const Tensor& t : {out, dout, lse, sd, off}) stack.emplace_back(t);
    stack.emplace_back(c.sm_scale);
    stack.emplace_back(c.dropout_p);
    for (int64_t i : {c.causal_type, c.left, c.right}) stack.emplace_back(i);
    stack.emplace_back(at::globalContext().deterministicAlgorithms());
    c10::Dispatcher::singleton().findSchemaOrThrow("aotriton_b200::attn_bwd", "").callBoxed(&stack);
    for (int i = 0; i < (b.defined() ? 4 : 3); ++i) r[i] = stack[i].toTensor();
  }
};

// ---- from Python ------------------------------------------------------------------------------------------

// A torch.Tensor or Parameter (no subclass) that is plain().  The tensor itself goes to *out.
bool plain_tensor(PyObject* o, int dev, Tensor* out) {
  if (!THPVariable_CheckExact(o)) return false;
  const Tensor& t = THPVariable_Unpack(o);
  if (!plain(t, dev) || t.stride(-1) != 1) return false;
  *out = t;
  return true;
}
bool attention_operand(PyObject* o, int dev, Tensor* out) {
  if (!plain_tensor(o, dev, out)) return false;
  const auto t = out->scalar_type();
  return out->dim() == 4 && (t == at::kFloat || t == at::kHalf || t == at::kBFloat16);
}
bool small_int(PyObject* o, int64_t* out) {      // fits the C API's int32
  if (!PyLong_CheckExact(o)) return false;
  *out = PyLong_AsLongLong(o);
  if (*out == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return *out >= INT32_MIN && *out <= INT32_MAX;
}
bool u64(PyObject* o, uint64_t* out) {
  if (!PyLong_CheckExact(o)) return false;
  *out = PyLong_AsUnsignedLongLong(o);
  if (*out == (uint64_t)-1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}
bool number(PyObject* o, double* out) {
  if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
  *out = PyFloat_AsDouble(o);
  if (*out == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}

// attend(q, k, v, bias, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, sm_scale, dropout_p, causal_type, window_left,
// window_right, return_lse, philox_seed, philox_offset, op): out, or (out, lse), or None: not an ordinary call.
PyObject* attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 17) {
    PyErr_SetString(PyExc_TypeError, "attend takes 17 arguments");
    return nullptr;
  }
  Call c{};
  Tensor q, k, v, b, cu_q, cu_k;
  // (a process without a CUDA context yet has no tensor to look at either)
  if (!THPVariable_CheckExact(a[0]) || !THPVariable_Unpack(a[0]).is_cuda() || !plain_modes()) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  if (!attention_operand(a[0], dev, &q) || !attention_operand(a[1], dev, &k) || !attention_operand(a[2], dev, &v)) Py_RETURN_NONE;
  if (a[3] != Py_None && !attention_operand(a[3], dev, &b)) Py_RETURN_NONE;
  if (k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type() || (b.defined() && b.scalar_type() != q.scalar_type()))
    Py_RETURN_NONE;
  c.packed = a[4] != Py_None;
  if (c.packed) {
    for (int i = 0; i < 2; ++i) {
      Tensor& cu = i ? cu_k : cu_q;
      if (!plain_tensor(a[4 + i], dev, &cu) || cu.dim() != 1 || cu.numel() < 2 || cu.scalar_type() != at::kInt) Py_RETURN_NONE;
    }
    if (b.defined() || q.size(0) != 1 || !small_int(a[6], &c.max_q) || !small_int(a[7], &c.max_k)) Py_RETURN_NONE;
  }
  if (!number(a[8], &c.sm_scale) || !number(a[9], &c.dropout_p) || !small_int(a[10], &c.causal_type) || !small_int(a[11], &c.left) ||
      !small_int(a[12], &c.right))
    Py_RETURN_NONE;
  const bool return_lse = a[13] == Py_True;
  if (!return_lse && a[13] != Py_False) Py_RETURN_NONE;
  if (c.dropout_p > 0 && (!u64(a[14], &c.seed) || !u64(a[15], &c.offset))) Py_RETURN_NONE;
  c.op = a[16] == Py_True;
  Tensor out, lse;
  {
    pybind11::gil_scoped_release release;
    const bool grad = at::GradMode::is_enabled() &&
                      (q.requires_grad() || k.requires_grad() || v.requires_grad() || (b.defined() && b.requires_grad()));
    if (grad) {
      auto maybe = [](const Tensor& t) { return t.defined() ? Attend::Maybe(t) : Attend::Maybe(); };
      variable_list r = Attend::apply(q, k, v, maybe(b), maybe(cu_q), maybe(cu_k), c, return_lse);
      out = std::move(r[0]);
      if (return_lse) lse = std::move(r[1]);
    } else {
      Tensor seed;
      forward(c, q, k, v, b, cu_q, cu_k, return_lse, out, lse, seed);
    }
  }
  if (!return_lse) return THPVariable_Wrap(std::move(out));
  return PyTuple_Pack(2, pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(std::move(out))).ptr(),
                      pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(std::move(lse))).ptr());
  END_HANDLE_TH_ERRORS
}

PyObject* last_bwd_family(PyObject*, PyObject*) { return PyLong_FromLong(g_last_bwd_family.load(std::memory_order_relaxed)); }
// ... of a backward that ran on this thread by the Python way
PyObject* note_bwd_family(PyObject*, PyObject*) {
  g_last_bwd_family.store(ab200_last_bwd_family(), std::memory_order_relaxed);
  Py_RETURN_NONE;
}

// The Function's backward: (q, k, v, bias, out, dout, logsumexp, cu_seqlens_q, cu_seqlens_k, seed, offset, sm_scale, dropout_p, causal_type,
// window_left, window_right, max_seqlen_q, max_seqlen_k) -> (dq, dk, dv, dbias).  Kept for the life of the process.
PyObject* set_python_backward(PyObject*, PyObject* fn) {
  Py_INCREF(fn);
  std::swap(g_python_backward, fn);
  Py_XDECREF(fn);
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {{"attend", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&attend)), METH_FASTCALL, nullptr},
                          {"set_python_backward", &set_python_backward, METH_O, nullptr},
                          {"last_bwd_family", &last_bwd_family, METH_NOARGS, nullptr},
                          {"note_bwd_family", &note_bwd_family, METH_NOARGS, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_ops", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_ops() { return PyModule_Create(&kModule); }
