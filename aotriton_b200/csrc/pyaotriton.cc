// Python module `pyaotriton`: the same names the Python tests and the tuner of
// ROCm/aotriton import (bindings/module.cc:32-113, hipruntime.cc:11-95,
// hipmemory.cc:15-69, lazy_tensor/main.cc:17-34, modules/flash/bindings/v2.cc:26-50,
// v3.cc:21-186), bound to this library's C++ operator API.
//
// Differences a caller can observe:
//   * Stream(handle: int) is accepted in addition to Stream(); handle is a
//     cudaStream_t as an integer (torch.cuda.current_stream().cuda_stream).
//   * lazy_tensor.dq_acc / delta allocate through a small stream-keyed caching pool over
//     cudaMalloc, so the module does not link against libtorch; lazy_tensor.dq_acc_from /
//     delta_from take a Python callable instead, which is how the torch allocator is used
//     (the reference's lazy tensors call at::zeros / at::empty,
//     bindings/lazy_tensor/lazy_tensor_template.h:19-97).
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include <aotriton/flash.h>
#include <aotriton/util.h>
#include <aotriton_b200.h>
#include <cuda_runtime_api.h>

#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

namespace py = pybind11;
namespace aotriton = AOTRITON_NS;

namespace {

// ---- device scratch pool for lazy tensors -------------------------------------
// Blocks go back to a free list instead of cudaFree, so disposing a lazy tensor right after an
// asynchronous launch never synchronises the device.  The free lists are keyed by (device,
// stream): a block is only handed out again for work on the stream its previous user ran on,
// where the new kernels queue behind the old ones (what a stream-ordered caching allocator does).
class ScratchPool {
 public:
  using Key = std::pair<int, intptr_t>;
  void* take(int device, intptr_t stream, size_t bytes) {
    bytes = (bytes + 511) & ~size_t(511);
    if (bytes == 0) bytes = 512;
    {
      std::lock_guard<std::mutex> lock(mu_);
      auto& fl = free_[Key(device, stream)];
      auto it = fl.lower_bound(bytes);
      if (it != fl.end() && it->first <= 2 * bytes) {
        void* p = it->second;
        sizes_[p] = it->first;
        fl.erase(it);
        return p;
      }
    }
    int old = -1;
    cudaGetDevice(&old);
    if (device >= 0 && device != old) cudaSetDevice(device);
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (device >= 0 && device != old) cudaSetDevice(old);
    if (e != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
    std::lock_guard<std::mutex> lock(mu_);
    sizes_[p] = bytes;
    return p;
  }
  void give(int device, intptr_t stream, void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lock(mu_);
    free_[Key(device, stream)].emplace(sizes_[p], p);
  }

 private:
  std::mutex mu_;
  std::map<Key, std::multimap<size_t, void*>> free_;
  std::map<void*, size_t> sizes_;
};

ScratchPool& pool() {
  static ScratchPool* p = new ScratchPool;   // leaked on purpose: outlives CUDA teardown order issues
  return *p;
}

// Cookies of lazy tensors that have not been disposed yet.  A LazyTensor is a plain struct that
// callers copy around (into the params struct, for one); only the copy inside the operator call
// is cleared by free(), so a stale copy used for a second call must be recognised here.
class LiveCookies {
 public:
  void add(void* c) { std::lock_guard<std::mutex> l(mu_); live_.insert(c); }
  bool alive(void* c) { std::lock_guard<std::mutex> l(mu_); return live_.count(c) != 0; }
  bool remove(void* c) { std::lock_guard<std::mutex> l(mu_); return live_.erase(c) != 0; }
 private:
  std::mutex mu_;
  std::set<void*> live_;
};
LiveCookies& cookies() {
  static LiveCookies* c = new LiveCookies;
  return *c;
}

template <int Rank>
aotriton::TensorView<Rank> contiguous_f32_view(const aotriton::TensorView<Rank>& like, void* mem, uint64_t* numel) {
  std::array<uint64_t, Rank> sizes = like.sizes(), strides{};
  uint64_t n = 1;
  for (int i = Rank - 1; i >= 0; --i) { strides[i] = n; n *= sizes[i]; }
  if (numel) *numel = n;
  return aotriton::TensorView<Rank>(reinterpret_cast<intptr_t>(mem), sizes, strides, aotriton::kFloat32);
}

template <int Rank, bool Zeroed>
struct LazyHelper {
  struct Ctx {
    aotriton::TensorView<Rank> like;
    int device;
    intptr_t stream;      // the stream the operator call will launch on (0 = the default stream)
    void* mem = nullptr;
  };
  static aotriton::TensorView<Rank> acquire(aotriton::LazyTensor<Rank>* self) {
    auto* ctx = static_cast<Ctx*>(self->cookie);
    if (!ctx || !cookies().alive(ctx)) return aotriton::TensorView<Rank>();   // a lazy tensor serves one call
    uint64_t n = 0;
    contiguous_f32_view<Rank>(ctx->like, nullptr, &n);
    if (!ctx->mem) {
      ctx->mem = pool().take(ctx->device, ctx->stream, n * sizeof(float));
      if (ctx->mem && Zeroed)
        cudaMemsetAsync(ctx->mem, 0, n * sizeof(float), reinterpret_cast<cudaStream_t>(ctx->stream));
    }
    if (!ctx->mem) return aotriton::TensorView<Rank>();
    return contiguous_f32_view<Rank>(ctx->like, ctx->mem, nullptr);
  }
  static void dispose(aotriton::LazyTensor<Rank>* self) {
    auto* ctx = static_cast<Ctx*>(self->cookie);
    if (!ctx || !cookies().remove(ctx)) return;
    pool().give(ctx->device, ctx->stream, ctx->mem);
    delete ctx;
  }
  static aotriton::TensorView<Rank> acquire_eager(aotriton::LazyTensor<Rank>* self) { return self->eager; }

  static aotriton::LazyTensor<Rank> make(const aotriton::TensorView<Rank>& like, int device, intptr_t stream) {
    auto* ctx = new Ctx;
    ctx->like = like;
    ctx->device = device;
    ctx->stream = stream;
    cookies().add(ctx);
    aotriton::LazyTensor<Rank> lt;
    lt.cookie = ctx;
    lt.acquire = &acquire;
    lt.dispose = &dispose;
    return lt;
  }
  static aotriton::LazyTensor<Rank> make_eager(const aotriton::TensorView<Rank>& view) {
    aotriton::LazyTensor<Rank> lt;
    lt.acquire = &acquire_eager;
    lt.eager = view;
    return lt;
  }
};

// Lazy tensor whose memory comes from a Python callable (called at most once, when the operator
// really needs the tensor): the callable returns an object with data_ptr(), e.g. a torch tensor
// made by torch.empty / torch.zeros on the current stream, which the lazy tensor keeps alive until
// the operator disposes of it.  The operator runs with the GIL released, so both callbacks take it.
template <int Rank>
struct PyLazy {
  struct Ctx {
    aotriton::TensorView<Rank> like;
    py::object factory, tensor;
  };
  static aotriton::TensorView<Rank> acquire(aotriton::LazyTensor<Rank>* self) {
    auto* ctx = static_cast<Ctx*>(self->cookie);
    if (!ctx || !cookies().alive(ctx)) return aotriton::TensorView<Rank>();
    py::gil_scoped_acquire gil;
    try {
      if (!ctx->tensor || ctx->tensor.is_none()) ctx->tensor = ctx->factory();
      const intptr_t ptr = ctx->tensor.attr("data_ptr")().template cast<intptr_t>();
      return contiguous_f32_view<Rank>(ctx->like, reinterpret_cast<void*>(ptr), nullptr);
    } catch (py::error_already_set& e) {
      e.discard_as_unraisable("pyaotriton lazy tensor factory");
      return aotriton::TensorView<Rank>();
    }
  }
  static void dispose(aotriton::LazyTensor<Rank>* self) {
    auto* ctx = static_cast<Ctx*>(self->cookie);
    if (!ctx || !cookies().remove(ctx)) return;
    py::gil_scoped_acquire gil;
    delete ctx;
  }
  static aotriton::LazyTensor<Rank> make(const aotriton::TensorView<Rank>& like, py::object factory) {
    auto* ctx = new Ctx;
    ctx->like = like;
    ctx->factory = std::move(factory);
    cookies().add(ctx);
    aotriton::LazyTensor<Rank> lt;
    lt.cookie = ctx;
    lt.acquire = &acquire;
    lt.dispose = &dispose;
    return lt;
  }
};

// Plain cudaMalloc'ed buffer for callers that keep their tensors on the host.
class HipMemory {
 public:
  ~HipMemory() { release(); }
  void alloc(size_t size) {
    release();
    last_ = static_cast<hipError_t>(cudaMalloc(&mem_, size));
    if (last_ == hipSuccess) size_ = size;
  }
  void release() {
    if (mem_) last_ = static_cast<hipError_t>(cudaFree(mem_));
    mem_ = nullptr; size_ = 0;
  }
  intptr_t get_pointer() const { return reinterpret_cast<intptr_t>(mem_); }
  void load_from_host(intptr_t ptr, size_t nbytes) {
    if (mem_ && nbytes <= size_)
      last_ = static_cast<hipError_t>(cudaMemcpy(mem_, reinterpret_cast<void*>(ptr), nbytes, cudaMemcpyHostToDevice));
  }
  void store_to_host(intptr_t ptr, size_t nbytes) {
    if (mem_ && nbytes <= size_)
      last_ = static_cast<hipError_t>(cudaMemcpy(reinterpret_cast<void*>(ptr), mem_, nbytes, cudaMemcpyDeviceToHost));
  }
  void zero_memory() { if (mem_) last_ = static_cast<hipError_t>(cudaMemset(mem_, 0, size_)); }
  hipError_t last_state() const { return last_; }

 private:
  void* mem_ = nullptr;
  size_t size_ = 0;
  hipError_t last_ = hipSuccess;
};

template <int Rank>
void def_tensorview(py::module_& m, const char* name) {
  using TV = aotriton::TensorView<Rank>;
  py::class_<TV>(m, name)
      .def(py::init<intptr_t, std::array<uint64_t, Rank>, std::array<uint64_t, Rank>, aotriton::DType>())
      .def("size", &TV::size)
      .def("stride", &TV::stride)
      .def_property_readonly("sizes", &TV::sizes)
      .def_property_readonly("strides", &TV::strides)
      .def_property_readonly("data_ptr", [](const TV& t) { return reinterpret_cast<intptr_t>(t.data_ptr()); })
      .def_property_readonly("dtype", &TV::dtype);
}

void def_hip_errors(py::module_& m) {
  py::enum_<hipError_t> e(m, "hipError_t", py::module_local());
#define EV(name) e.value(#name, name)
  EV(hipSuccess); EV(hipErrorInvalidValue); EV(hipErrorOutOfMemory); EV(hipErrorMemoryAllocation);
  EV(hipErrorNotInitialized); EV(hipErrorInitializationError); EV(hipErrorDeinitialized);
  EV(hipErrorProfilerDisabled); EV(hipErrorProfilerNotInitialized); EV(hipErrorProfilerAlreadyStarted);
  EV(hipErrorProfilerAlreadyStopped); EV(hipErrorInvalidConfiguration); EV(hipErrorInvalidPitchValue);
  EV(hipErrorInvalidSymbol); EV(hipErrorInvalidDevicePointer); EV(hipErrorInvalidMemcpyDirection);
  EV(hipErrorInsufficientDriver); EV(hipErrorMissingConfiguration); EV(hipErrorPriorLaunchFailure);
  EV(hipErrorInvalidDeviceFunction); EV(hipErrorNoDevice); EV(hipErrorInvalidDevice); EV(hipErrorInvalidImage);
  EV(hipErrorInvalidContext); EV(hipErrorContextAlreadyCurrent); EV(hipErrorMapFailed);
  EV(hipErrorMapBufferObjectFailed); EV(hipErrorUnmapFailed); EV(hipErrorArrayIsMapped); EV(hipErrorAlreadyMapped);
  EV(hipErrorNoBinaryForGpu); EV(hipErrorAlreadyAcquired); EV(hipErrorNotMapped); EV(hipErrorNotMappedAsArray);
  EV(hipErrorNotMappedAsPointer); EV(hipErrorECCNotCorrectable); EV(hipErrorUnsupportedLimit);
  EV(hipErrorContextAlreadyInUse); EV(hipErrorPeerAccessUnsupported); EV(hipErrorInvalidKernelFile);
  EV(hipErrorInvalidGraphicsContext); EV(hipErrorInvalidSource); EV(hipErrorFileNotFound);
  EV(hipErrorSharedObjectSymbolNotFound); EV(hipErrorSharedObjectInitFailed); EV(hipErrorOperatingSystem);
  EV(hipErrorInvalidHandle); EV(hipErrorInvalidResourceHandle); EV(hipErrorIllegalState); EV(hipErrorNotFound);
  EV(hipErrorNotReady); EV(hipErrorIllegalAddress); EV(hipErrorLaunchOutOfResources); EV(hipErrorLaunchTimeOut);
  EV(hipErrorPeerAccessAlreadyEnabled); EV(hipErrorPeerAccessNotEnabled); EV(hipErrorSetOnActiveProcess);
  EV(hipErrorContextIsDestroyed); EV(hipErrorAssert); EV(hipErrorHostMemoryAlreadyRegistered);
  EV(hipErrorHostMemoryNotRegistered); EV(hipErrorLaunchFailure); EV(hipErrorCooperativeLaunchTooLarge);
  EV(hipErrorNotSupported); EV(hipErrorStreamCaptureUnsupported); EV(hipErrorStreamCaptureInvalidated);
  EV(hipErrorStreamCaptureMerge); EV(hipErrorStreamCaptureUnmatched); EV(hipErrorStreamCaptureUnjoined);
  EV(hipErrorStreamCaptureIsolation); EV(hipErrorStreamCaptureImplicit); EV(hipErrorCapturedEvent);
  EV(hipErrorStreamCaptureWrongThread); EV(hipErrorGraphExecUpdateFailure); EV(hipErrorUnknown);
  EV(hipErrorRuntimeMemory); EV(hipErrorRuntimeOther); EV(hipErrorTbd);
#undef EV
  e.export_values();
  m.def("hipDeviceSynchronize", []() { return static_cast<hipError_t>(::hipDeviceSynchronize()); });
  m.def("hipGetLastError", []() { return static_cast<hipError_t>(::hipGetLastError()); });
}

void def_v2(py::module_& root) {
  py::module_ v2 = root.def_submodule("v2", "v2 API namespace");
  py::module_ m = v2.def_submodule("flash", "Flash Attention API");
  m.def("check_gpu", &aotriton::v2::flash::check_gpu, py::arg("stream"));
  m.def("debug_simulate_encoded_softmax", &aotriton::v2::flash::debug_simulate_encoded_softmax,
        "Write +0.5/-0.5 according to the dropout keep bit", py::call_guard<py::gil_scoped_release>(),
        py::arg("r"), py::arg("dropout_p"), py::arg("philox_seed_ptr"), py::arg("philox_offset1"),
        py::arg("philox_offset2"), py::arg("stream") = aotriton::Stream());
  m.def("attn_fwd", &aotriton::v2::flash::attn_fwd, py::call_guard<py::gil_scoped_release>());
  m.def("attn_fwd_compact_varlen", &aotriton::v2::flash::attn_fwd_compact_varlen,
        py::call_guard<py::gil_scoped_release>());
  m.def("attn_bwd", &aotriton::v2::flash::attn_bwd, py::call_guard<py::gil_scoped_release>());
  m.def("attn_bwd_compact_varlen", &aotriton::v2::flash::attn_bwd_compact_varlen,
        py::call_guard<py::gil_scoped_release>());
}

void def_v3(py::module_& root) {
  using aotriton::v3::flash::attn_bwd_params;
  using aotriton::v3::flash::attn_fwd_params;
  using aotriton::v3::flash::attn_options;
  py::module_ v3 = root.def_submodule("v3", "v3 API namespace");
  py::module_ m = v3.def_submodule("flash", "Flash Attention Operators");
  py::class_<attn_options>(m, "attn_options")
      .def(py::init<>())
      .def_readwrite("force_backend_index", &attn_options::force_backend_index)
      .def_readwrite("deterministic", &attn_options::deterministic);
  py::class_<attn_fwd_params> f(m, "attn_fwd_params");
  f.def(py::init<>());
#define RW(name) f.def_readwrite(#name, &attn_fwd_params::name)
  RW(Q); RW(K); RW(V); RW(B); RW(Sm_scale); RW(L); RW(Out); RW(cu_seqlens_q); RW(cu_seqlens_k);
  RW(Max_seqlen_q); RW(Max_seqlen_k); RW(seq_strides_q); RW(seq_strides_k); RW(dropout_p);
  RW(philox_seed_ptr); RW(philox_offset1); RW(philox_offset2); RW(philox_seed_output);
  RW(philox_offset_output); RW(encoded_softmax); RW(persistent_atomic_counter); RW(causal_type);
  RW(varlen_type); RW(window_left); RW(window_right);
#undef RW
  f.def_readonly_static("kVersion", &attn_fwd_params::kVersion);
  py::class_<attn_bwd_params> b(m, "attn_bwd_params");
  b.def(py::init<>());
#define RW(name) b.def_readwrite(#name, &attn_bwd_params::name)
  RW(Q); RW(K); RW(V); RW(B); RW(Sm_scale); RW(Out); RW(DO); RW(DK); RW(DV); RW(DQ); RW(DB); RW(L); RW(D);
  RW(cu_seqlens_q); RW(cu_seqlens_k); RW(Max_seqlen_q); RW(Max_seqlen_k); RW(seq_strides_q);
  RW(seq_strides_k); RW(dropout_p); RW(philox_seed_ptr); RW(philox_offset1); RW(philox_offset2);
  RW(causal_type); RW(varlen_type); RW(window_left); RW(window_right); RW(DQ_ACC);
#undef RW
  b.def_readonly_static("kVersion", &attn_bwd_params::kVersion);
  m.def("attn_fwd", &aotriton::v3::flash::attn_fwd, "Flash Attention Operator Forward Pass",
        py::call_guard<py::gil_scoped_release>(), py::arg("params"), py::arg("params_version"),
        py::arg("stream") = aotriton::Stream(), py::arg("options") = nullptr);
  m.def("attn_bwd", &aotriton::v3::flash::attn_bwd, "Flash Attention Operator Backward Pass",
        py::call_guard<py::gil_scoped_release>(), py::arg("params"), py::arg("params_version"),
        py::arg("stream") = aotriton::Stream(), py::arg("options") = nullptr);
}

// ---- torch tensors straight into a parameter struct ----------------------------------------------
// Building every TensorView as a Python object (tuples to std::array and back) and assigning it costs 5 to 6
// us a tensor: 66 us of host time for a forward call and 91 us for a backward, several times what the kernels
// of a small call take.  These fill the structs from the tensors' data_ptr() / shape / stride() in one call (6 and
// 8 us).  They take the ordinary forms only and return false for everything else (the caller then goes the long
// way, which also words the errors).
struct TorchNames {
  PyObject *data_ptr = PyUnicode_InternFromString("data_ptr"), *shape = PyUnicode_InternFromString("shape"),
           *stride = PyUnicode_InternFromString("stride"), *dtype = PyUnicode_InternFromString("dtype");
};
const TorchNames& torch_names() {
  static const TorchNames* n = new TorchNames;
  return *n;
}

// `dtypes`: dict torch.dtype -> DType value as int.
class ViewReader {
 public:
  explicit ViewReader(py::dict dtypes) : dtypes_(std::move(dtypes)) {}

  template <int Rank>
  bool read(py::handle t, aotriton::TensorView<Rank>* out) const {
    const TorchNames& n = torch_names();
    aotriton::DType dt;
    if (t.is_none() || !dtype(t, &dt)) return false;
    const py::object shape = py::reinterpret_steal<py::object>(PyObject_GetAttr(t.ptr(), n.shape));
    if (!shape) throw py::error_already_set();
    if (!PyTuple_Check(shape.ptr()) || PyTuple_GET_SIZE(shape.ptr()) != Rank) return false;
    const py::object stride = py::reinterpret_steal<py::object>(PyObject_CallMethodNoArgs(t.ptr(), n.stride));
    if (!stride) throw py::error_already_set();
    if (!PyTuple_Check(stride.ptr()) || PyTuple_GET_SIZE(stride.ptr()) != Rank) return false;
    std::array<uint64_t, Rank> sizes, strides;
    for (int i = 0; i < Rank; ++i) {
      sizes[i] = PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(shape.ptr(), i));
      strides[i] = PyLong_AsUnsignedLongLong(PyTuple_GET_ITEM(stride.ptr(), i));
      if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    }
    if (strides[Rank - 1] != 1) return false;
    intptr_t ptr;
    if (!pointer(t, &ptr)) return false;
    *out = aotriton::TensorView<Rank>(ptr, sizes, strides, dt);
    return true;
  }

  // None: a null view of the other tensor's type
  template <int Rank>
  bool read_or_null(py::handle t, aotriton::DType like, aotriton::TensorView<Rank>* out) const {
    if (!t.is_none()) return read(t, out);
    *out = aotriton::TensorView<Rank>(0, {}, {}, like);
    return true;
  }

  // a device scalar: a rank-1 tensor of one element, or of none (null)
  bool read_scalar(py::handle t, aotriton::TensorView<0>* out) const {
    aotriton::DType dt;
    if (t.is_none() || !dtype(t, &dt)) return false;
    const py::object shape = py::reinterpret_steal<py::object>(PyObject_GetAttr(t.ptr(), torch_names().shape));
    if (!shape) throw py::error_already_set();
    if (!PyTuple_Check(shape.ptr()) || PyTuple_GET_SIZE(shape.ptr()) != 1) return false;
    const long long count = PyLong_AsLongLong(PyTuple_GET_ITEM(shape.ptr(), 0));
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    intptr_t ptr;
    if ((count != 0 && count != 1) || !pointer(t, &ptr)) return false;
    *out = aotriton::TensorView<0>(ptr, dt);
    return true;
  }

 private:
  bool dtype(py::handle t, aotriton::DType* out) const {
    const py::object d = py::reinterpret_steal<py::object>(PyObject_GetAttr(t.ptr(), torch_names().dtype));
    if (!d) throw py::error_already_set();
    PyObject* v = PyDict_GetItemWithError(dtypes_.ptr(), d.ptr());      // (borrowed)
    if (v == nullptr) { if (PyErr_Occurred()) throw py::error_already_set(); return false; }
    *out = static_cast<aotriton::DType>(PyLong_AsLong(v));
    return true;
  }
  static bool pointer(py::handle t, intptr_t* out) {
    const py::object p = py::reinterpret_steal<py::object>(PyObject_CallMethodNoArgs(t.ptr(), torch_names().data_ptr));
    if (!p) throw py::error_already_set();
    *out = (intptr_t)PyLong_AsUnsignedLongLong(p.ptr());
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
  }
  py::dict dtypes_;
};

bool set_fwd_views(aotriton::v3::flash::attn_fwd_params& p, py::dict dtypes, py::handle q, py::handle k, py::handle v,
                   py::handle b, py::handle lse, py::handle out, py::handle seed, py::handle off1, py::handle seed_out,
                   py::handle off_out, py::handle enc, py::handle atomic) {
  const ViewReader r(std::move(dtypes));
  if (!r.read(q, &p.Q)) return false;
  return r.read(k, &p.K) && r.read(v, &p.V) && r.read_or_null(b, p.Q.dtype(), &p.B) &&
         r.read_or_null(lse, aotriton::kFloat32, &p.L) && r.read(out, &p.Out) && r.read_scalar(seed, &p.philox_seed_ptr) &&
         r.read_scalar(off1, &p.philox_offset1) && r.read_scalar(seed_out, &p.philox_seed_output) &&
         r.read_scalar(off_out, &p.philox_offset_output) && r.read_or_null(enc, p.Q.dtype(), &p.encoded_softmax) &&
         r.read_scalar(atomic, &p.persistent_atomic_counter);
}

bool set_bwd_views(aotriton::v3::flash::attn_bwd_params& p, py::dict dtypes, py::handle q, py::handle k, py::handle v,
                   py::handle b, py::handle out, py::handle dout, py::handle dk, py::handle dv, py::handle dq, py::handle db,
                   py::handle lse, py::handle seed, py::handle off1) {
  const ViewReader r(std::move(dtypes));
  if (!r.read(q, &p.Q)) return false;
  return r.read(k, &p.K) && r.read(v, &p.V) && r.read_or_null(b, p.Q.dtype(), &p.B) && r.read(out, &p.Out) &&
         r.read(dout, &p.DO) && r.read(dk, &p.DK) && r.read(dv, &p.DV) && r.read(dq, &p.DQ) &&
         r.read_or_null(db, p.Q.dtype(), &p.DB) && r.read(lse, &p.L) && r.read_scalar(seed, &p.philox_seed_ptr) &&
         r.read_scalar(off1, &p.philox_offset1);
}

void def_lazy(py::module_& root) {
  py::module_ m = root.def_submodule("lazy_tensor", "lazy_tensor API namespace");
  py::class_<aotriton::LazyTensor<4>>(m, "LT4");
  py::class_<aotriton::LazyTensor<2>>(m, "LT2");
  m.def("dq_acc", &LazyHelper<4, true>::make, py::arg("like"), py::arg("device"), py::arg("stream") = 0);
  m.def("delta", &LazyHelper<2, false>::make, py::arg("like"), py::arg("device"), py::arg("stream") = 0);
  m.def("dq_acc_from", &PyLazy<4>::make, py::arg("like"), py::arg("factory"));
  m.def("delta_from", &PyLazy<2>::make, py::arg("like"), py::arg("factory"));
  m.def("eager_delta", &LazyHelper<2, false>::make_eager);
  // (the same straight from a tensor; None: not an ordinary one)
  m.def("dq_acc_of", [](py::dict dtypes, py::handle t, py::object factory) -> py::object {
    aotriton::TensorView<4> like;
    if (!ViewReader(std::move(dtypes)).read(t, &like)) return py::none();
    return py::cast(PyLazy<4>::make(like, std::move(factory)));
  });
  m.def("delta_of", [](py::dict dtypes, py::handle t, py::object factory) -> py::object {
    aotriton::TensorView<2> like;
    if (!ViewReader(std::move(dtypes)).read(t, &like)) return py::none();
    return py::cast(PyLazy<2>::make(like, std::move(factory)));
  });
  m.def("eager_delta_of", [](py::dict dtypes, py::handle t) -> py::object {
    aotriton::TensorView<2> view;
    if (!ViewReader(std::move(dtypes)).read(t, &view)) return py::none();
    return py::cast(LazyHelper<2, false>::make_eager(view));
  });
  m.def("eager_null_dq_acc", &LazyHelper<4, false>::make_eager);
}

}  // namespace

PYBIND11_MODULE(pyaotriton, m) {
  m.doc() = "aotriton operator API backed by sm_100a CUDA kernels";
  py::class_<aotriton::Stream>(m, "Stream")
      .def(py::init<>())
      .def(py::init([](intptr_t handle) { return aotriton::Stream(reinterpret_cast<hipStream_t>(handle)); }));
  py::enum_<aotriton::DType>(m, "DType")
      .value("kUnknown", aotriton::kUnknown)
      .value("kFloat32", aotriton::kFloat32)
      .value("kFloat16", aotriton::kFloat16)
      .value("kBFloat16", aotriton::kBFloat16)
      .value("kInt8", aotriton::kInt8)
      .value("kInt16", aotriton::kInt16)
      .value("kInt32", aotriton::kInt32)
      .value("kInt64", aotriton::kInt64)
      .value("kUInt8", aotriton::kUInt8)
      .value("kUInt16", aotriton::kUInt16)
      .value("kUInt32", aotriton::kUInt32)
      .value("kUInt64", aotriton::kUInt64)
      .export_values();
  def_hip_errors(m);
  def_tensorview<4>(m, "T4");
  def_tensorview<2>(m, "T2");
  def_tensorview<1>(m, "T1");
  py::class_<HipMemory>(m, "HipMemory")
      .def(py::init<>())
      .def("alloc", &HipMemory::alloc)
      .def("free", &HipMemory::release)
      .def("get_pointer", &HipMemory::get_pointer)
      .def("last_state", &HipMemory::last_state)
      .def("load_from_host", &HipMemory::load_from_host)
      .def("store_to_host", &HipMemory::store_to_host)
      .def("zero_memory", &HipMemory::zero_memory);
  using T0 = aotriton::TensorView<0>;
  py::class_<T0>(m, "T0")
      .def(py::init<intptr_t, aotriton::DType>())
      .def("size", &T0::size)
      .def("stride", &T0::stride)
      .def_property_readonly("sizes", &T0::sizes)
      .def_property_readonly("strides", &T0::strides)
      .def_property_readonly("data_ptr", [](const T0& t) { return reinterpret_cast<intptr_t>(t.data_ptr()); })
      .def_property_readonly("dtype", &T0::dtype);
#define AB200_STR2(x) #x
#define AB200_STR(x) AB200_STR2(x)
  m.def("get_name_suffix", []() -> std::string { return AB200_STR(AOTRITON_NAME_SUFFIX); });
  m.def("set_fwd_views", &set_fwd_views);
  m.def("set_bwd_views", &set_bwd_views);
  m.def("launch_count", []() { return ab200_launch_count(); });
  m.def("set_kernel_family", [](int f) { return ab200_set_kernel_family(f); });
  m.def("last_fwd_family", []() { return ab200_last_fwd_family(); });
  m.def("last_bwd_family", []() { return ab200_last_bwd_family(); });
  m.def("stream_check", [](aotriton::Stream s) { return static_cast<hipError_t>(ab200_stream_check(s.native())); },
        py::call_guard<py::gil_scoped_release>(), py::arg("stream") = aotriton::Stream());
  m.def("kernel_status", [](bool reset) { return ab200_kernel_status(reset ? 1 : 0); }, py::arg("reset") = false);
  def_v2(m);
  def_v3(m);
  def_lazy(m);
}
