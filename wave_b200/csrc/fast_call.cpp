// Repeated calls of the Python front ends, in native code: `wave_b200._fast`.
//
// A scaled GEMM of a small problem runs for 5 to 30 microseconds on the GPU, and so long did the Python code take that leads
// to it (the counterpart of the reference's invoke path, wave_lang/kernel/wave/utils/run_utils.py:62-134, which it
// measures with profile_python_wrapper): building the key of a call from shapes and strides, the look-up of the weight's packed
// scales and of the workspace, sixteen arguments through ctypes. Here a call that was made before is recognised from the
// tensors themselves and goes straight to the C ABI of include/wave_b200.h; whatever is not recognised returns None, and the
// Python code does what it always did (all checks, all error messages) and then registers what it found.
//
// What is kept: per kernel object, the signatures (sizes, strides, types, device, stream, alignment of the output) of at most
// kMaxPlans calls with their scratch, and at most kMaxWeights packings of weight scales, each found by the tensor it was made from
// (a weak reference), its version counter, address, sizes and strides, as WeightScaleCache does. Nothing about activations or outputs
// is kept but their shapes. A call notes whose scratch and workspace it used where the Python code notes it (`marks`): a captured call takes the
// memory of the eager call before it. Calls under stream capture, on another device than the current one, with tensor subclasses, under
// functional transforms, or with weight scales that are inference tensors (which have no version) are left to the Python code.
// us per call, calls back to back, before and after this module: 1024^3 f32 16.9 -> 8.2, MXFP4Linear 8 x 14336 x 4096 26.8 -> 15.6 (since then 6.9 and 10.8: the
// GPU's time).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <iterator>
#include <unordered_map>
#include <vector>

namespace {

// A model that walks all its layers through one kernel object uses one or two packings per layer, and one plan per distinct row count. Those of weights
// that are gone are given back at the next registration.
constexpr size_t kMaxPlans = 1024, kMaxWeights = 512;
constexpr int kF32 = 0, kBF16 = 1;  // WB200_F32, WB200_BF16

struct Abi {
  int (*gemm_repack_a)(int, int, int, const void*, const void*, long long, void*, const void*, const void*, void*, int, long long, void*, size_t,
                       unsigned, void*);
  int (*mxfp8_gemm_repack_a)(int, int, int, const void*, const void*, long long, void*, const void*, const void*, void*, int, long long, int, void*,
                             size_t, unsigned, void*);
  int (*gemm_quantize_a)(int, int, int, const void*, int, long long, void*, void*, const void*, const void*, void*, int, long long, void*, size_t,
                         unsigned, void*);
  size_t (*gemm_workspace_bytes)(int, int, int);
  int (*decode_tile_rows_for)(int, int, int, int, int, int);
} abi;

// A reference to a Python object; copied and dropped with the interpreter lock held.
struct Ref {
  PyObject* o = nullptr;
  Ref() = default;
  explicit Ref(PyObject* p) : o(p) { Py_XINCREF(o); }
  Ref(const Ref& r) : Ref(r.o) {}
  Ref(Ref&& r) noexcept : o(r.o) { r.o = nullptr; }
  Ref& operator=(Ref r) noexcept {
    std::swap(o, r.o);
    return *this;
  }
  ~Ref() { Py_XDECREF(o); }
};
// A mark is a pair (list of one element, value): setting it makes the value the list's element.
bool is_mark(PyObject* m) {
  return PyTuple_Check(m) && PyTuple_GET_SIZE(m) == 2 && PyList_Check(PyTuple_GET_ITEM(m, 0)) && PyList_GET_SIZE(PyTuple_GET_ITEM(m, 0)) == 1;
}
void set_mark(PyObject* m) { PyList_SetItem(PyTuple_GET_ITEM(m, 0), 0, Py_NewRef(PyTuple_GET_ITEM(m, 1))); }

// An ordinary CUDA tensor: no subclass, no wrapper of a functional transform. Tensors made in inference mode count (a layer's output there is the
// next one's input): they only lack the autograd keys.
bool plain(PyObject* o) {
  if (Py_TYPE(o) != reinterpret_cast<PyTypeObject*>(THPVariableClass)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  static const c10::DispatchKeySet inference = c10::DispatchKeySet(c10::DispatchKey::CUDA) |
                                               c10::getAutocastRelatedKeySetFromBackend(c10::BackendComponent::CUDABit);
  static const c10::DispatchKeySet ordinary = inference | c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) |
                                              c10::getAutogradRelatedKeySetFromBackend(c10::BackendComponent::CUDABit);
  return (t.key_set() == ordinary || t.key_set() == inference) && t.layout() == at::kStrided;
}

struct Signature {
  int64_t size[2], stride[2];
  at::ScalarType type;
  bool operator==(const Signature& o) const {
    return size[0] == o.size[0] && size[1] == o.size[1] && stride[0] == o.stride[0] && stride[1] == o.stride[1] && type == o.type;
  }
};
bool signature_of(const at::Tensor& t, int device, Signature* s) {
  if (t.dim() != 2 || t.device().index() != device) return false;
  s->size[0] = t.size(0);
  s->size[1] = t.size(1);
  s->stride[0] = t.stride(0);
  s->stride[1] = t.stride(1);
  s->type = t.scalar_type();
  return true;
}

// Every row of a matrix with unit column stride starts on 16 bytes.
bool rows_aligned(const at::Tensor& c) {
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 == 0 && (c.size(0) == 1 || c.stride(0) * int64_t(c.element_size()) % 16 == 0);
}

struct CallKey {  // order: a, a_scale, b, b_scale, c
  Signature sig[5];
  int device;
  cudaStream_t stream;
  bool aligned, tiled;
  long path;
  bool operator==(const CallKey& o) const {
    return stream == o.stream && device == o.device && aligned == o.aligned && tiled == o.tiled && path == o.path && std::equal(sig, sig + 5, o.sig);
  }
};
struct CallKeyHash {
  size_t operator()(const CallKey& k) const {
    uint64_t h = reinterpret_cast<uintptr_t>(k.stream) + uint64_t(k.device) * 4 + k.aligned * 2 + k.tiled + uint64_t(k.path) * 64;
    auto mix = [&h](uint64_t v) { h = (h ^ v) * 0x9e3779b97f4a7c15ull, h ^= h >> 29; };
    for (const Signature& s : k.sig) {
      for (int i = 0; i < 2; ++i) mix(uint64_t(s.size[i])), mix(uint64_t(s.stride[i]));
      mix(uint64_t(s.type));
    }
    return size_t(h);
  }
};
struct Plan {
  int M, N, K;
  int elem_format;  // -1: MXFP4
  unsigned flags;
  at::Tensor scratch, workspace;  // packed activation scales; workspace (undefined: none)
  size_t workspace_bytes;
  int tile_rows;
  Ref marks;  // a tuple of marks
};
struct Weight {
  c10::weak_intrusive_ptr<c10::TensorImpl> owner;
  Signature sig;
  const void* ptr;
  uint32_t version;
  int tile_rows;
  at::Tensor packed;
  cudaStream_t stream;  // the one that the packing was filled on,
  bool complete;        // and whether that is known to be done: until then the Python code orders other streams behind it
  uint64_t used;        // when the last call read it
};

struct Calls {
  std::unordered_map<CallKey, Plan, CallKeyHash> plans;
  std::unordered_multimap<const c10::TensorImpl*, Weight> weights;
  uint64_t now = 0, asked = 0;  // calls so far, and when the Python code last asked which packings were used
  const std::pair<const CallKey, Plan>* last = nullptr;  // the plan of the last call (entries keep their place until they are erased)

  const Plan* find(const CallKey& key) {
    if (last && last->first == key) return &last->second;
    const auto it = plans.find(key);
    if (it == plans.end()) return nullptr;
    last = &*it;
    return &it->second;
  }
  Weight* find(const at::Tensor& scale, const Signature& sig, int tile_rows) {
    const auto [first, last] = weights.equal_range(scale.unsafeGetTensorImpl());
    for (auto it = first; it != last; ++it) {
      Weight& w = it->second;
      // (an address that another tensor has taken over belongs to a new object, and the reference to the old one has expired)
      if (w.tile_rows == tile_rows && w.sig == sig && !w.owner.expired() && w.ptr == scale.data_ptr() && w.version == scale._version()) return &w;
    }
    return nullptr;
  }
  void insert(const c10::TensorImpl* impl, Weight w) {
    for (auto it = weights.begin(); it != weights.end();)
      it = it->second.owner.expired() || (it->first == impl && it->second.tile_rows == w.tile_rows) ? weights.erase(it) : std::next(it);
    if (weights.size() >= kMaxWeights) {  // the one that was not used for longest
      auto oldest = weights.begin();
      for (auto it = weights.begin(); it != weights.end(); ++it)
        if (it->second.used < oldest->second.used) oldest = it;
      weights.erase(oldest);
    }
    weights.emplace(impl, std::move(w));
  }
};

struct PyCalls {
  PyObject_HEAD
  Calls* calls;
};

bool key_of(PyObject* const* args, CallKey* key) {
  for (int i = 0; i < 5; ++i)
    if (!plain(args[i])) return false;
  if (THPVariable_Unpack(args[3]).is_inference()) return false;
  const at::Tensor& a = THPVariable_Unpack(args[0]);
  key->device = a.device().index();
  if (key->device != c10::cuda::current_device()) return false;
  for (int i = 0; i < 5; ++i)
    if (!signature_of(THPVariable_Unpack(args[i]), key->device, &key->sig[i])) return false;
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return false;
  key->stream = c10::cuda::getCurrentCUDAStream(key->device).stream();
  key->aligned = rows_aligned(THPVariable_Unpack(args[4]));
  key->tiled = PyObject_IsTrue(args[5]) == 1;
  key->path = PyLong_AsLong(args[6]);
  return !PyErr_Occurred();
}

PyObject* fail(const std::exception& e) {
  PyErr_SetString(PyExc_RuntimeError, e.what());
  return nullptr;
}

// call(a, a_scale, b, b_scale, c, tiled, path) -> status of the launch, or None: not a call that is known here
PyObject* calls_call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  if (n != 7) {
    PyErr_SetString(PyExc_TypeError, "call takes 7 arguments");
    return nullptr;
  }
  try {
    Calls& calls = *reinterpret_cast<PyCalls*>(self)->calls;
    CallKey key;
    if (calls.plans.empty() || !key_of(args, &key)) {
      if (PyErr_Occurred()) return nullptr;
      Py_RETURN_NONE;
    }
    const Plan* found = calls.find(key);
    Weight* weight = found ? calls.find(THPVariable_Unpack(args[3]), key.sig[3], found->tile_rows) : nullptr;
    if (!weight || !(weight->complete || weight->stream == key.stream)) Py_RETURN_NONE;
    weight->used = ++calls.now;
    // another thread may change the tables while the lock is released: what the launch reads is held here
    const at::Tensor scratch = found->scratch, workspace = found->workspace, packed = weight->packed;
    const int M = found->M, N = found->N, K = found->K, elem_format = found->elem_format;
    const size_t ws_bytes = found->workspace_bytes;
    const unsigned flags = found->flags;
    const void* ptr[4];
    for (int i = 0; i < 3; ++i) ptr[i] = THPVariable_Unpack(args[i]).data_ptr();
    void* c = THPVariable_Unpack(args[4]).data_ptr();
    const int c_type = key.sig[4].type == at::kFloat ? kF32 : kBF16;
    const long long a_scale_stride = M > 1 ? key.sig[1].stride[0] : K / 32, ldc = M > 1 ? key.sig[4].stride[0] : N;
    void* ws = workspace.defined() ? workspace.data_ptr() : nullptr;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(found->marks.o); ++i) set_mark(PyTuple_GET_ITEM(found->marks.o, i));
    if (weight->stream != key.stream)  // its memory may be given back on the stream it was made on while this one reads it
      c10::cuda::CUDACachingAllocator::recordStream(packed.storage().data_ptr(), c10::cuda::getCurrentCUDAStream(key.device));
    int rc;
    Py_BEGIN_ALLOW_THREADS
    if (elem_format < 0)
      rc = abi.gemm_repack_a(M, N, K, ptr[0], ptr[1], a_scale_stride, scratch.data_ptr(), ptr[2], packed.data_ptr(), c, c_type, ldc, ws, ws_bytes, flags,
                             key.stream);
    else
      rc = abi.mxfp8_gemm_repack_a(M, N, K, ptr[0], ptr[1], a_scale_stride, scratch.data_ptr(), ptr[2], packed.data_ptr(), c, c_type, ldc, elem_format,
                                   ws, ws_bytes, flags, key.stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
  } catch (const std::exception& e) {
    return fail(e);
  }
}

// add(a, a_scale, b, b_scale, c, tiled, path, (M, N, K, elem_format, flags, tile_rows, workspace_bytes), packed, scratch, workspace or None, marks,
//     stream that the packing was filled on, whether it is complete):
// the Python code has just made this call with these arguments.
PyObject* calls_add(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  bool marks_ok = n == 14 && PyTuple_Check(args[11]);
  for (Py_ssize_t i = 0; marks_ok && i < PyTuple_GET_SIZE(args[11]); ++i) marks_ok = is_mark(PyTuple_GET_ITEM(args[11], i));
  if (!marks_ok) {
    PyErr_SetString(PyExc_TypeError, "add takes 14 arguments, the twelfth a tuple of (list of one element, value) pairs");
    return nullptr;
  }
  try {
    Calls& calls = *reinterpret_cast<PyCalls*>(self)->calls;
    Plan p;
    CallKey key;
    Py_ssize_t ws_bytes = 0;
    if (!PyArg_ParseTuple(args[7], "iiiiIin", &p.M, &p.N, &p.K, &p.elem_format, &p.flags, &p.tile_rows, &ws_bytes)) return nullptr;
    if (!key_of(args, &key) || !THPVariable_Check(args[8]) || !THPVariable_Check(args[9])) {
      if (PyErr_Occurred()) return nullptr;
      Py_RETURN_NONE;
    }
    const at::ScalarType c_type = key.sig[4].type;
    if (key.sig[4].stride[1] != 1 || (c_type != at::kFloat && c_type != at::kBFloat16)) Py_RETURN_NONE;
    p.scratch = THPVariable_Unpack(args[9]);
    if (args[10] != Py_None) p.workspace = THPVariable_Unpack(args[10]);
    p.workspace_bytes = size_t(ws_bytes);
    p.marks = Ref(args[11]);
    if (calls.plans.size() >= kMaxPlans && !calls.plans.count(key)) {
      calls.last = nullptr;
      calls.plans.erase(calls.plans.begin());
    }
    const int tile_rows = p.tile_rows;
    calls.plans[key] = std::move(p);
    const at::Tensor& scale = THPVariable_Unpack(args[3]);
    const auto filled_on = reinterpret_cast<cudaStream_t>(PyLong_AsUnsignedLongLong(args[12]));
    const bool complete = PyObject_IsTrue(args[13]) == 1;
    if (PyErr_Occurred()) return nullptr;
    Weight* known = calls.find(scale, key.sig[3], tile_rows);
    if (known && known->packed.is_same(THPVariable_Unpack(args[8]))) {
      known->complete = known->complete || complete;
    } else {
      calls.insert(scale.unsafeGetTensorImpl(),
                   Weight{c10::weak_intrusive_ptr<c10::TensorImpl>(scale.getIntrusivePtr()), key.sig[3], scale.data_ptr(), uint32_t(scale._version()),
                          tile_rows, THPVariable_Unpack(args[8]), filled_on, complete, ++calls.now});
    }
    Py_RETURN_NONE;
  } catch (const std::exception& e) {
    return fail(e);
  }
}

PyObject* calls_clear(PyObject* self, PyObject*) {
  Calls& calls = *reinterpret_cast<PyCalls*>(self)->calls;
  calls.last = nullptr;
  calls.plans.clear();
  calls.weights.clear();
  Py_RETURN_NONE;
}

// recent() -> addresses of the packings that calls have read since it was asked last, the one used last at the end
PyObject* calls_recent(PyObject* self, PyObject*) {
  Calls& calls = *reinterpret_cast<PyCalls*>(self)->calls;
  std::vector<std::pair<uint64_t, const void*>> used;
  for (const auto& [impl, w] : calls.weights)
    if (w.used > calls.asked) used.emplace_back(w.used, w.packed.data_ptr());
  calls.asked = calls.now;
  std::sort(used.begin(), used.end());
  PyObject* list = PyList_New(Py_ssize_t(used.size()));
  for (size_t i = 0; list && i < used.size(); ++i) {
    PyObject* address = PyLong_FromVoidPtr(const_cast<void*>(used[i].second));
    if (!address) {
      Py_DECREF(list);
      return nullptr;
    }
    PyList_SET_ITEM(list, Py_ssize_t(i), address);
  }
  return list;
}

// ---------------------------------------------------------------------------------------------
// What stands behind the work that the current stream of a device has been given so far: Fence(device)
// ---------------------------------------------------------------------------------------------
struct PyFence {
  PyObject_HEAD
  int device;
  cudaStream_t stream;
  cudaEvent_t event;
};
PyObject* fence_new(PyTypeObject* type, PyObject* args, PyObject*) {
  int device;
  if (!PyArg_ParseTuple(args, "i", &device)) return nullptr;
  auto* self = reinterpret_cast<PyFence*>(type->tp_alloc(type, 0));
  if (!self) return nullptr;
  try {
    const c10::cuda::CUDAGuard guard{c10::DeviceIndex(device)};
    self->device = device;
    self->stream = c10::cuda::getCurrentCUDAStream(device).stream();
    cudaError_t rc = cudaEventCreateWithFlags(&self->event, cudaEventDisableTiming);
    if (rc == cudaSuccess) rc = cudaEventRecord(self->event, self->stream);
    if (rc == cudaSuccess) return reinterpret_cast<PyObject*>(self);
    (void)cudaGetLastError();
    PyErr_Format(PyExc_RuntimeError, "wave_b200: no event behind the work of stream %p: %s", self->stream, cudaGetErrorString(rc));
  } catch (const std::exception& e) {
    fail(e);
  }
  Py_DECREF(self);
  return nullptr;
}
void fence_free(PyObject* o) {
  auto* self = reinterpret_cast<PyFence*>(o);
  if (self->event && cudaEventDestroy(self->event) != cudaSuccess) (void)cudaGetLastError();
  Py_TYPE(o)->tp_free(o);
}
PyObject* fence_stream(PyObject* o, PyObject*) { return PyLong_FromVoidPtr(reinterpret_cast<PyFence*>(o)->stream); }
// done() -> whether that work is complete; may be asked while a stream is being captured (the event is not part of the capture)
PyObject* fence_done(PyObject* o, PyObject*) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // of this thread: a query does not end a capture then
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) {
    (void)cudaGetLastError();
    Py_RETURN_FALSE;
  }
  const cudaError_t status = cudaEventQuery(reinterpret_cast<PyFence*>(o)->event);
  (void)cudaGetLastError();
  (void)cudaThreadExchangeStreamCaptureMode(&mode);
  return PyBool_FromLong(status == cudaSuccess);
}
// wait(): what the current stream of the device does next comes after that work
PyObject* fence_wait(PyObject* o, PyObject*) {
  auto* self = reinterpret_cast<PyFence*>(o);
  try {
    const c10::cuda::CUDAGuard guard{c10::DeviceIndex(self->device)};
    const cudaError_t rc = cudaStreamWaitEvent(c10::cuda::getCurrentCUDAStream(self->device).stream(), self->event, 0);
    if (rc == cudaSuccess) Py_RETURN_NONE;
    (void)cudaGetLastError();
    PyErr_SetString(PyExc_RuntimeError, cudaGetErrorString(rc));
    return nullptr;
  } catch (const std::exception& e) {
    return fail(e);
  }
}

// ---------------------------------------------------------------------------------------------
// workspaces of the functional entry points, as WorkspacePool holds them
// ---------------------------------------------------------------------------------------------
struct Workspaces {
  struct Entry {
    int device;
    cudaStream_t stream;
    at::Tensor ws;
    Ref mark;
  };
  std::vector<Entry> entries;
};
struct PyWorkspaces {
  PyObject_HEAD
  Workspaces* table;
};
// put(device, stream, workspace, mark)
PyObject* workspaces_put(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  if (n != 4 || !THPVariable_Check(args[2]) || !is_mark(args[3])) {
    PyErr_SetString(PyExc_TypeError, "put takes a device index, a stream, a tensor and a (list of one element, value) pair");
    return nullptr;
  }
  const int device = int(PyLong_AsLong(args[0]));
  auto stream = reinterpret_cast<cudaStream_t>(PyLong_AsUnsignedLongLong(args[1]));
  if (PyErr_Occurred()) return nullptr;
  auto& entries = reinterpret_cast<PyWorkspaces*>(self)->table->entries;
  for (auto& e : entries)
    if (e.device == device && e.stream == stream) {
      e.ws = THPVariable_Unpack(args[2]);
      e.mark = Ref(args[3]);
      Py_RETURN_NONE;
    }
  entries.push_back({device, stream, THPVariable_Unpack(args[2]), Ref(args[3])});
  Py_RETURN_NONE;
}
PyObject* workspaces_clear(PyObject* self, PyObject*) {
  reinterpret_cast<PyWorkspaces*>(self)->table->entries.clear();
  Py_RETURN_NONE;
}

template <typename Object, typename Data, Data* Object::*Field>
PyObject* object_new(PyTypeObject* type, PyObject*, PyObject*) {
  PyObject* self = type->tp_alloc(type, 0);
  if (self) reinterpret_cast<Object*>(self)->*Field = new Data;
  return self;
}
template <typename Object, typename Data, Data* Object::*Field>
void object_free(PyObject* self) {
  delete (reinterpret_cast<Object*>(self)->*Field);
  Py_TYPE(self)->tp_free(self);
}

bool is_workspaces(PyObject* o);

// Packed scales of N rows and K values in tiles of tile_rows (at most 128) rows: a 512-byte atom per 128 K and tile, K padded to 256.
// (The kernel's tensor map covers all of it, whatever the array holds.)
bool holds_scales(const at::Tensor& packed, int64_t N, int64_t K, int64_t tile_rows) {
  return packed.scalar_type() == at::kByte && packed.is_contiguous() && packed.numel() >= (N + tile_rows - 1) / tile_rows * ((K + 255) / 256) * 1024;
}

// linear(x, weight_codes, (rows and K that the scales were packed for, packed scales, those per tile of low_rows rows, low_rows), output dtype,
//        workspaces)
// -> dequant(quantise(x)) @ dequant(W)^T, or None: left to the Python code.
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 5 || !PyTuple_Check(args[2]) || PyTuple_GET_SIZE(args[2]) != 5 || !is_workspaces(args[4])) {
    PyErr_SetString(PyExc_TypeError, "linear takes 5 arguments, the third a tuple of 5 and the last one a Workspaces object");
    return nullptr;
  }
  PyObject* const* scales = reinterpret_cast<PyTupleObject*>(args[2])->ob_item;
  try {
    if (!plain(args[0]) || !plain(args[1]) || !plain(scales[2]) || !THPDtype_Check(args[3])) Py_RETURN_NONE;
    const at::Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]);
    at::Tensor packed = THPVariable_Unpack(scales[2]);
    const long long rows = PyLong_AsLongLong(scales[0]), of_k = PyLong_AsLongLong(scales[1]);
    if (PyErr_Occurred()) return nullptr;
    const int device = x.device().index();
    const at::ScalarType x_type = x.scalar_type(), out_type = reinterpret_cast<THPDtype*>(args[3])->scalar_type;
    const int64_t dims = x.dim();
    if (device != c10::cuda::current_device() || w.device().index() != device || packed.device().index() != device || dims < 1 || w.dim() != 2 ||
        !w.is_contiguous() || w.element_size() != 1 || (x_type != at::kFloat && x_type != at::kBFloat16) || (out_type != at::kFloat && out_type != at::kBFloat16))
      Py_RETURN_NONE;
    const int64_t K = w.size(1) * 2, N = w.size(0);
    if (N != rows || K != of_k) Py_RETURN_NONE;  // refused there: the scales belong to another matrix
    if (x.size(dims - 1) != K || K == 0 || x.numel() == 0) Py_RETURN_NONE;
    const int64_t M = x.numel() / K;
    const bool strided = dims == 2 && x.stride(1) == 1 && x.stride(0) >= K;
    if (!(strided || x.is_contiguous()) || M > 0x7fffffff || N > 0x7fffffff) Py_RETURN_NONE;
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) Py_RETURN_NONE;
    const auto stream = c10::cuda::getCurrentCUDAStream(device);
    at::Tensor ws;
    Ref mark;
    size_t ws_bytes = 0;
    if (M <= 128) {
      ws_bytes = abi.gemm_workspace_bytes(int(M), int(N), int(K));
      for (const auto& e : reinterpret_cast<PyWorkspaces*>(args[4])->table->entries)
        if (e.device == device && e.stream == stream.stream()) {
          ws = e.ws;
          mark = e.mark;
        }
      if (!ws.defined() || size_t(ws.numel()) < ws_bytes) Py_RETURN_NONE;
    }
    // (a fresh output starts on 16 bytes: its rows are aligned when N says so)
    const bool aligned = M == 1 || N * (out_type == at::kFloat ? 4 : 2) % 16 == 0;
    int tile_rows = 128;
    if (M <= 128 && (tile_rows = abi.decode_tile_rows_for(int(M), int(N), int(K), 4, 4, aligned)) != 128) {
      if (PyLong_AsLong(scales[4]) != tile_rows || !plain(scales[3])) {
        if (PyErr_Occurred()) return nullptr;
        Py_RETURN_NONE;
      }
      packed = THPVariable_Unpack(scales[3]);
      if (packed.device().index() != device) Py_RETURN_NONE;
    }
    if (!holds_scales(packed, N, K, tile_rows)) Py_RETURN_NONE;
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = N;
    const at::Tensor out = at::detail::empty_cuda(shape, out_type, x.device(), c10::nullopt);
    const int64_t q_bytes = (M * K / 2 + 255) / 256 * 256;
    const at::Tensor scratch = at::detail::empty_cuda({q_bytes + (M + 127) / 128 * ((K + 255) / 256) * 1024}, at::kByte, x.device(), c10::nullopt);
    uint8_t* q = static_cast<uint8_t*>(scratch.data_ptr());
    if (mark.o) set_mark(mark.o);
    const unsigned flags = tile_rows == 128 ? 0u : unsigned(tile_rows / 8) << 16;  // WB200_B_TILE_ROWS
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = abi.gemm_quantize_a(int(M), int(N), int(K), x.data_ptr(), x_type == at::kFloat ? kF32 : kBF16, strided && M > 1 ? x.stride(0) : K, q, q + q_bytes,
                             w.data_ptr(), packed.data_ptr(), out.data_ptr(), out_type == at::kFloat ? kF32 : kBF16, N,
                             ws.defined() ? ws.data_ptr() : nullptr, ws_bytes, flags, stream.stream());
    Py_END_ALLOW_THREADS
    if (rc) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
  } catch (const std::exception& e) {
    return fail(e);
  }
}

// bind(gemm_repack_a, mxfp8_gemm_repack_a, gemm_quantize_a, gemm_workspace_bytes, decode_tile_rows_for): addresses in the loaded library
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long p[5];
  if (!PyArg_ParseTuple(args, "KKKKK", &p[0], &p[1], &p[2], &p[3], &p[4])) return nullptr;
  abi.gemm_repack_a = reinterpret_cast<decltype(abi.gemm_repack_a)>(p[0]);
  abi.mxfp8_gemm_repack_a = reinterpret_cast<decltype(abi.mxfp8_gemm_repack_a)>(p[1]);
  abi.gemm_quantize_a = reinterpret_cast<decltype(abi.gemm_quantize_a)>(p[2]);
  abi.gemm_workspace_bytes = reinterpret_cast<decltype(abi.gemm_workspace_bytes)>(p[3]);
  abi.decode_tile_rows_for = reinterpret_cast<decltype(abi.decode_tile_rows_for)>(p[4]);
  Py_RETURN_NONE;
}

#define FASTCALL(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL
PyMethodDef calls_methods[] = {{"call", FASTCALL(calls_call), nullptr}, {"add", FASTCALL(calls_add), nullptr},
                               {"clear", calls_clear, METH_NOARGS, nullptr}, {"recent", calls_recent, METH_NOARGS, nullptr},
                               {nullptr, nullptr, 0, nullptr}};
PyMethodDef workspaces_methods[] = {{"put", FASTCALL(workspaces_put), nullptr}, {"clear", workspaces_clear, METH_NOARGS, nullptr},
                                    {nullptr, nullptr, 0, nullptr}};
PyMethodDef fence_methods[] = {{"stream", fence_stream, METH_NOARGS, nullptr}, {"done", fence_done, METH_NOARGS, nullptr},
                               {"wait", fence_wait, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyMethodDef module_methods[] = {{"bind", bind, METH_VARARGS, nullptr}, {"linear", FASTCALL(linear), nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_fast", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

bool is_workspaces(PyObject* o) {
  return Py_TYPE(o)->tp_dealloc == object_free<PyWorkspaces, Workspaces, &PyWorkspaces::table>;
}

template <typename Object>
bool add_type(PyObject* module, const char* name, const char* qualified, PyMethodDef* methods, newfunc make, destructor free) {
  static PyTypeObject type = {PyVarObject_HEAD_INIT(nullptr, 0)};
  type.tp_name = qualified;
  type.tp_basicsize = sizeof(Object);
  type.tp_flags = Py_TPFLAGS_DEFAULT;
  type.tp_methods = methods;
  type.tp_new = make;
  type.tp_dealloc = free;
  if (PyType_Ready(&type) < 0) return false;
  return PyModule_AddObjectRef(module, name, reinterpret_cast<PyObject*>(&type)) == 0;
}

}  // namespace

PyMODINIT_FUNC PyInit__fast() {
  PyObject* m = PyModule_Create(&module_def);
  if (!m) return nullptr;
  if (!add_type<PyCalls>(m, "Calls", "wave_b200._fast.Calls", calls_methods, object_new<PyCalls, Calls, &PyCalls::calls>,
                         object_free<PyCalls, Calls, &PyCalls::calls>) ||
      !add_type<PyWorkspaces>(m, "Workspaces", "wave_b200._fast.Workspaces", workspaces_methods, object_new<PyWorkspaces, Workspaces, &PyWorkspaces::table>,
                              object_free<PyWorkspaces, Workspaces, &PyWorkspaces::table>) ||
      !add_type<PyFence>(m, "Fence", "wave_b200._fast.Fence", fence_methods, fence_new, fence_free)) {
    Py_DECREF(m);
    return nullptr;
  }
  if (PyModule_AddStringConstant(m, "target", WB200_FAST_TARGET) < 0) {  // what this was compiled against
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
