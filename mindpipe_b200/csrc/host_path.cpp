// The host side of the module forwards, in native code.
//
// A forward of a small linear is 5-10 us of GPU work; checking the arguments, allocating the result and making the
// C-ABI call from Python took about 30 us (one 4096 x 4096 W4A16 linear at one token: 31 us per call, 6 us of them on
// the GPU).  A Plan holds what does not change between calls (weight-side tensors, sizes, which module attributes it
// was derived from) and one call of Plan.run does what the Python wrappers in ops.py do: check the input, allocate
// the output, find the stream's scratch buffer and call the C ABI.  Everything out of the ordinary -- another dtype or
// device, a non-contiguous or empty input, a tensor subclass, weights that were replaced or edited since the plan was
// made, an error status -- makes run() return None, and the module then takes the checked Python path, which rebuilds
// the plan or raises.  No arithmetic happens here.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/mindpipe_b200.h"

namespace {

// ------------------------------------------------------------------------------------------------- scratch buffers
// Zero-initialised scratch, one per (device, stream, kind) and one per captured stream of a graph, grown on demand.  The
// decode kernels leave their part zeroed where it has to be, so it is cleared only when it is (re)allocated; the kinds whose
// kernels overwrite theirs freely (split-K partial sums) have buffers of their own.  Launches of one stream run in order, so
// they may share.
enum WorkspaceKind { kDecode = 0, kPrefill = 1, kW8A8 = 2, kKinds = 3 };
const char* const kKindNames[kKinds] = {"decode", "prefill", "w8a8"};

std::mutex g_workspace_mutex;
std::map<std::tuple<int, cudaStream_t, int>, at::Tensor> g_workspaces;

// Scratch of a graph capture.  A captured launch holds the address for as long as its graph lives, and graphs that were
// captured on one stream may be replayed side by side; so a capture never takes the stream's buffer, which a later call that
// wants more replaces, but one of its own per captured stream.  It does not come from the graph's memory pool, where memory of
// other tensors of the capture is used again: its words have to stay zero from one replay to the next.  It is given back at
// the first capture after that pool's memory has gone back to the driver, which happens when the pool has no graph any more
// and waits for the device, so no replay is in flight.  (A capture without a pool of torch's keeps its scratch.  A user object
// of the graph would tell of its end at once, and costs 6.5 us a replay: a 7B layer's four linears at 16 rows 41.1 -> 47.4.)
// Cleared once, outside the graph: a fill in front of every linear, 1.2 MB up to 16 rows and up to 10 MB beyond, also kept the
// linear from starting before the end of the kernel before (that layer at 1 / 8 / 16 / 77 / 128 rows, us, with the fills
// 51.2 / 50.8 / 53.4 / 80.0 / 106, without 38.7 / 39.0 / 41.1 / 62.7 / 86.3).
struct CaptureScratch {
  std::vector<at::Tensor> buffers;                   // the last is in use; launches captured before it grew hold the others
  c10::MempoolId_t pool{0, 0};                       // of the graph; {0, 0}: none that is known
};
using CaptureKey = std::tuple<int, cudaStream_t, int, unsigned long long>;
std::map<CaptureKey, CaptureScratch> g_captures;

// The memory pool of the capture on the current stream; scratch of pools that are gone is given back.
c10::MempoolId_t look_at_pools(int device) {
  const at::Tensor probe = at::empty({1}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
  const auto address = reinterpret_cast<size_t>(probe.data_ptr());
  c10::MempoolId_t pool{0, 0};
  std::set<std::pair<int, c10::MempoolId_t>> there;
  if (c10::cuda::CUDACachingAllocator::name() != "native") return pool;          // (the other allocator has no snapshots)
  for (const auto& segment : c10::cuda::CUDACachingAllocator::snapshot({0, 0}, false).segments) {
    there.emplace(segment.device, segment.owner_private_pool_id);
    if (address >= segment.address && address - segment.address < segment.total_size) pool = segment.owner_private_pool_id;
  }
  for (auto it = g_captures.begin(); it != g_captures.end();) {
    const c10::MempoolId_t of = it->second.pool;
    const bool keep = of == c10::MempoolId_t{0, 0} || there.count({std::get<0>(it->first), of});
    it = keep ? std::next(it) : g_captures.erase(it);
  }
  return pool;
}

// A stream of this library's own, on which captures' scratch is allocated and cleared while another stream captures.
cudaStream_t clearing_stream(int device) {
  static auto* streams = new std::map<int, cudaStream_t>;
  cudaStream_t& st = (*streams)[device];
  if (!st) C10_CUDA_CHECK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  return st;
}

// The caller holds g_workspace_mutex.
at::Tensor capture_workspace(size_t nbytes, int device, cudaStream_t stream, int kind, unsigned long long id) {
  const CaptureKey key(device, stream, kind, id);
  auto at = g_captures.find(key);
  if (at != g_captures.end() && static_cast<size_t>(at->second.buffers.back().numel()) >= nbytes) return at->second.buffers.back();
  // at least twice the one before, so that those that are kept for earlier launches add up to less than the last
  size_t bytes = at == g_captures.end() ? size_t(1) << 20 : 2 * static_cast<size_t>(at->second.buffers.back().numel());
  if (bytes < nbytes) bytes = nbytes;
  // the capture's mode may forbid allocation and synchronisation, also of streams that do not capture
  c10::cuda::CUDAStreamCaptureModeGuard relaxed{cudaStreamCaptureModeRelaxed};
  c10::cuda::CUDAGuard on(static_cast<c10::DeviceIndex>(device));
  CaptureScratch fresh;
  if (at == g_captures.end()) fresh.pool = look_at_pools(device);
  const cudaStream_t clearing = clearing_stream(device);
  at::Tensor buffer;
  {
    c10::cuda::CUDAStreamGuard guard(c10::cuda::getStreamFromExternal(clearing, static_cast<c10::DeviceIndex>(device)));
    buffer = at::empty({static_cast<int64_t>(bytes)},
                       at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
  }
  C10_CUDA_CHECK(cudaMemsetAsync(buffer.data_ptr(), 0, bytes, clearing));
  C10_CUDA_CHECK(cudaStreamSynchronize(clearing));
  if (at == g_captures.end()) at = g_captures.emplace(key, std::move(fresh)).first;
  at->second.buffers.push_back(buffer);
  return buffer;
}

// A copy of the tensor handle: it keeps the buffer alive until the launch is in the stream even if another thread
// replaces it by a larger one meanwhile (the allocator hands freed memory on in stream order).
// own_in_capture: whether a capture may begin on a stream that has no scratch yet.  (A linear that could do without scratch is
// not to fail there for the sake of a faster kernel; the other calls ask for a first call outside the capture, as for their
// error word.)
at::Tensor workspace(size_t nbytes, int device, cudaStream_t stream, int kind, bool own_in_capture = false) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  // (the legacy stream cannot capture; the question takes 0.1 us, which a call of 6 us that the host bounds would show)
  if (stream && cudaStreamGetCaptureInfo(stream, &capturing, &id) != cudaSuccess) cudaGetLastError();    // the launch will tell
  std::lock_guard<std::mutex> lock(g_workspace_mutex);
  at::Tensor& ws = g_workspaces[std::make_tuple(device, stream, kind)];
  const bool there = ws.defined() && static_cast<size_t>(ws.numel()) >= nbytes;
  if (capturing == cudaStreamCaptureStatusActive && (there || own_in_capture))
    return capture_workspace(nbytes, device, stream, kind, id);
  if (!there) {
    TORCH_CHECK(capturing == cudaStreamCaptureStatusNone,
                "scratch memory would be allocated during CUDA graph capture; "
                "pass a preallocated workspace= (see new_workspace)");
    const int64_t bytes = static_cast<int64_t>(nbytes > (size_t(1) << 20) ? nbytes : (size_t(1) << 20));
    ws = at::zeros({bytes}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
  }
  return ws;
}

// ------------------------------------------------------------------------------------------------------------ plans
// An attribute the plan was derived from: dict[key] must still be the same object and, for a tensor, have the same
// storage address and version (in-place edits and load_state_dict advance the version counter).  A null dict is the
// attribute dict of the module run() is called with: the plan lives in that dict, and a reference from here would keep
// a dropped module's weights allocated until the next garbage collection.
struct Guard {
  PyObject* dict;
  PyObject* key;
  PyObject* value;      // null: the key was absent
  const void* data;
  uint32_t version;
};

const void* address_of(const at::Tensor& t) { return t.has_storage() ? t.unsafeGetTensorImpl()->data() : nullptr; }
uint32_t version_of(const at::Tensor& t) {
  const auto& v = t.unsafeGetTensorImpl()->version_counter();
  return v.enabled() ? v.current_version() : 0u;
}

struct Plan {
  std::vector<Guard> guards;
  int device = 0;
  virtual ~Plan() {
    for (Guard& g : guards) {
      Py_XDECREF(g.dict);
      Py_XDECREF(g.key);
      Py_XDECREF(g.value);
    }
  }
  // null with a Python error set, or a new reference (None = take the checked path)
  virtual PyObject* run(PyObject* module, PyObject* const* args, Py_ssize_t n) = 0;

  bool fresh(PyObject* module) const {
    PyObject* own = PyObject_GenericGetDict(module, nullptr);
    if (!own) {
      PyErr_Clear();
      return false;
    }
    const bool ok = fresh_in(own);
    Py_DECREF(own);
    return ok;
  }

 private:
  bool fresh_in(PyObject* own) const {
    for (const Guard& g : guards) {
      if (PyDict_GetItemWithError(g.dict ? g.dict : own, g.key) != g.value) return false;
      if (g.value && THPVariable_Check(g.value)) {
        const at::Tensor& t = THPVariable_Unpack(g.value);
        if (address_of(t) != g.data || version_of(t) != g.version) return false;
      }
    }
    return true;
  }
};

// The input as a dense CUDA tensor on the plan's (current) device, or null.
const at::Tensor* plain_input(PyObject* o, int device, at::ScalarType dtype) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (t.scalar_type() != dtype || !t.is_cuda() || t.get_device() != device || t.dim() < 1 || !t.is_contiguous() ||
      t.numel() == 0 || c10::cuda::current_device() != device)
    return nullptr;
  return &t;
}

at::Tensor output_like(const at::Tensor& x, int64_t last, at::ScalarType dtype) {
  c10::SmallVector<int64_t, 6> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = last;
  return at::empty(shape, x.options().dtype(dtype).requires_grad(false));
}

PyObject* none() { Py_RETURN_NONE; }

size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

at::Tensor scratch(size_t bytes, const at::Tensor& like) {
  return at::empty({static_cast<int64_t>(bytes)}, like.options().dtype(at::kByte).requires_grad(false));
}

const void* data_or_null(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// Scratch of the current stream for a call that wants `bytes` of it (0: none).
struct Scratch {
  at::Tensor hold;
  void* ptr = nullptr;
  size_t bytes = 0;
  Scratch(size_t wanted, int device, cudaStream_t st, int kind, bool own_in_capture = false) {
    if (!wanted) return;
    hold = workspace(wanted, device, st, kind, own_in_capture);
    ptr = hold.data_ptr();
    bytes = static_cast<size_t>(hold.numel());
  }
};

struct W4Plan : Plan {
  at::Tensor packed, scale_zero, bias;
  int n = 0, k = 0, group = 0;
  int* error_word = nullptr;
  PyObject* run(PyObject* module, PyObject* const* args, Py_ssize_t nargs) override {
    const at::Tensor* xp = nargs == 1 ? plain_input(args[0], device, at::kHalf) : nullptr;
    if (!xp || xp->size(-1) != k || !fresh(module)) return none();
    const at::Tensor& x = *xp;
    const int64_t rows = x.numel() / k;
    if (rows > (int64_t(1) << 30)) return none();
    const int m = static_cast<int>(rows);
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
    at::Tensor y = output_like(x, n, at::kHalf);
    Scratch ws(mp_w4a16_linear_workspace_bytes(m, n, k, group), device, st, kDecode, true);
    const int rc = mp_w4a16_linear(x.data_ptr(), packed.data_ptr(), scale_zero.data_ptr(), data_or_null(bias), y.data_ptr(),
                                   m, n, k, group, ws.ptr, ws.bytes, error_word, st);
    return rc == MP_OK ? THPVariable_Wrap(std::move(y)) : none();
  }
};

// Symmetric W8A8: per-token quantisation, then the int8 GEMM; codes and token scales live in one scratch tensor.
struct W8Plan : Plan {
  at::Tensor weight, weight_scale, bias;
  int n = 0, k = 0;
  int* error_word = nullptr;
  PyObject* run(PyObject* module, PyObject* const* args, Py_ssize_t nargs) override {
    const at::Tensor* xp = nargs == 1 ? plain_input(args[0], device, at::kHalf) : nullptr;
    if (!xp || xp->size(-1) != k || !fresh(module)) return none();
    const at::Tensor& x = *xp;
    const int64_t rows = x.numel() / k;
    if (rows > (int64_t(1) << 30)) return none();
    const int m = static_cast<int>(rows);
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
    at::Tensor y = output_like(x, n, at::kHalf);
    const size_t codes = align256(static_cast<size_t>(m) * k);
    at::Tensor q = scratch(codes + static_cast<size_t>(m) * 4, x);
    char* qp = static_cast<char*>(q.data_ptr());
    Scratch ws(mp_w8a8_linear_workspace_bytes(m, n, k), device, st, kDecode);
    const int rc = mp_w8a8_linear(x.data_ptr(), weight.data_ptr(), weight_scale.data_ptr(), data_or_null(bias), y.data_ptr(),
                                  m, n, k, qp, qp + codes, ws.ptr, ws.bytes, error_word, st);
    return rc == MP_OK ? THPVariable_Wrap(std::move(y)) : none();
  }
};

// Asymmetric W8A8 (OmniQuant): the same with zero points and code sums.
struct AffinePlan : Plan {
  at::Tensor weight, scale, zero, rowsum, bias;
  int n = 0, k = 0;
  int* error_word = nullptr;
  PyObject* run(PyObject* module, PyObject* const* args, Py_ssize_t nargs) override {
    const at::Tensor* xp = nargs == 1 ? plain_input(args[0], device, at::kHalf) : nullptr;
    if (!xp || xp->size(-1) != k || !fresh(module)) return none();
    const at::Tensor& x = *xp;
    const int64_t rows = x.numel() / k;
    if (rows > (int64_t(1) << 30)) return none();
    const int m = static_cast<int>(rows);
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
    at::Tensor y = output_like(x, n, at::kHalf);
    const size_t codes = align256(static_cast<size_t>(m) * k), per_row = align256(static_cast<size_t>(m) * 4);
    at::Tensor q = scratch(codes + 3 * per_row, x);
    char* qp = static_cast<char*>(q.data_ptr());
    char *sp = qp + codes, *zp = sp + per_row, *rp = zp + per_row;
    Scratch ws(mp_w8a8_affine_linear_workspace_bytes(m, n, k), device, st, kDecode);
    const int rc = mp_w8a8_affine_linear(x.data_ptr(), weight.data_ptr(), scale.data_ptr(), zero.data_ptr(),
                                         rowsum.data_ptr(), data_or_null(bias), y.data_ptr(), m, n, k, qp, sp, zp, rp, ws.ptr,
                                         ws.bytes, error_word, st);
    return rc == MP_OK ? THPVariable_Wrap(std::move(y)) : none();
  }
};

// W8A8 experts; one scratch tensor for the whole layer.
struct MoePlan : Plan {
  at::Tensor w13, w13_scale, w2, w2_scale;
  int h = 0, i = 0, lo = 0, hi = 0;
  int* error_word = nullptr;
  PyObject* run(PyObject* module, PyObject* const* args, Py_ssize_t nargs) override {
    const at::Tensor* xp = nargs == 3 ? plain_input(args[0], device, at::kHalf) : nullptr;
    const at::Tensor* idp = xp ? plain_input(args[1], device, at::kInt) : nullptr;
    const at::Tensor* wp = idp ? plain_input(args[2], device, at::kHalf) : nullptr;
    if (!wp || xp->size(-1) != h || !fresh(module)) return none();
    const at::Tensor& x = *xp;
    const int64_t rows = x.numel() / h;
    const int64_t entries = idp->numel();
    if (entries != wp->numel() || entries % rows != 0 || entries > (int64_t(1) << 24)) return none();
    const int t = static_cast<int>(rows), k = static_cast<int>(entries / rows), e = hi - lo;
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
    at::Tensor out = output_like(x, h, at::kHalf);
    const size_t bytes = mp_moe_experts_scratch_bytes(t, h, k, e, i);
    at::Tensor buf = scratch(bytes, x);
    Scratch ws(mp_moe_experts_workspace_bytes(t), device, st, kDecode);
    const int rc = mp_moe_experts(x.data_ptr(), idp->data_ptr(), wp->data_ptr(), t, h, k, lo, hi, w13.data_ptr(),
                                  w13_scale.data_ptr(), w2.data_ptr(), w2_scale.data_ptr(), i, out.data_ptr(), buf.data_ptr(),
                                  bytes, ws.ptr, ws.bytes, error_word, st);
    return rc == MP_OK ? THPVariable_Wrap(std::move(out)) : none();
  }
};

// ----------------------------------------------------------------------------------------------------- Python object
struct PlanObject {
  PyObject_HEAD
  Plan* plan;
};

void plan_dealloc(PyObject* self) {
  delete reinterpret_cast<PlanObject*>(self)->plan;
  PyTypeObject* type = Py_TYPE(self);
  type->tp_free(self);
  Py_DECREF(type);
}

PyObject* plan_run(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 1) return none();
  return reinterpret_cast<PlanObject*>(self)->plan->run(args[0], args + 1, n - 1);
  END_HANDLE_TH_ERRORS
}

PyObject* plan_fresh(PyObject* self, PyObject* module) {
  HANDLE_TH_ERRORS
  return PyBool_FromLong(reinterpret_cast<PlanObject*>(self)->plan->fresh(module));
  END_HANDLE_TH_ERRORS
}

// Copied or pickled with its module, a plan becomes None: the copy builds its own at its first forward.
PyObject* plan_reduce(PyObject*, PyObject*) {
  return Py_BuildValue("(O())", reinterpret_cast<PyObject*>(Py_TYPE(Py_None)));
}

PyMethodDef plan_methods[] = {
    {"run", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(plan_run)), METH_FASTCALL, nullptr},
    {"fresh", plan_fresh, METH_O, nullptr},
    {"__reduce__", plan_reduce, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyType_Slot plan_slots[] = {{Py_tp_dealloc, reinterpret_cast<void*>(plan_dealloc)},
                            {Py_tp_methods, plan_methods},
                            {0, nullptr}};
PyType_Spec plan_spec = {"mindpipe_b200._host.Plan", sizeof(PlanObject), 0,
                         Py_TPFLAGS_DEFAULT | Py_TPFLAGS_DISALLOW_INSTANTIATION, plan_slots};
PyTypeObject* plan_type = nullptr;

// guards: a sequence of (dict or None for the module's own, key) pairs whose present values the plan depends on
bool take_guards(Plan* p, PyObject* module, PyObject* guards) {
  PyObject* own = PyObject_GenericGetDict(module, nullptr);
  if (!own) return false;
  Py_DECREF(own);                                  // the module keeps it
  PyObject* seq = PySequence_Fast(guards, "guards must be a sequence");
  if (!seq) return false;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) {
    PyObject *dict, *key;
    if (!PyArg_ParseTuple(PySequence_Fast_GET_ITEM(seq, i), "OU", &dict, &key) ||
        (dict != Py_None && !PyDict_Check(dict))) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "a guard is a (dict or None, key) pair");
      Py_DECREF(seq);
      return false;
    }
    if (dict == Py_None) dict = nullptr;
    Guard g{dict, key, PyDict_GetItemWithError(dict ? dict : own, key), nullptr, 0};
    Py_XINCREF(dict);
    Py_INCREF(key);
    Py_XINCREF(g.value);
    if (g.value && THPVariable_Check(g.value)) {
      const at::Tensor& t = THPVariable_Unpack(g.value);
      g.data = address_of(t);
      g.version = version_of(t);
    }
    p->guards.push_back(g);
  }
  Py_DECREF(seq);
  return true;
}

PyObject* wrap_plan(std::unique_ptr<Plan> p, PyObject* module, PyObject* guards, const at::Tensor& on) {
  p->device = on.get_device();
  if (!take_guards(p.get(), module, guards)) return nullptr;
  PlanObject* o = PyObject_New(PlanObject, plan_type);
  if (!o) return nullptr;
  o->plan = p.release();
  return reinterpret_cast<PyObject*>(o);
}

bool tensor_arg(PyObject* o, at::Tensor& t, at::ScalarType dtype, bool optional = false) {
  if (optional && o == Py_None) return true;
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "expected a tensor");
    return false;
  }
  t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.scalar_type() != dtype || !t.is_contiguous()) {
    PyErr_SetString(PyExc_ValueError, "expected a contiguous CUDA tensor of the kernel's dtype");
    return false;
  }
  return true;
}

int* int_pointer(unsigned long long v) { return reinterpret_cast<int*>(static_cast<uintptr_t>(v)); }

PyObject* w4_plan(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  PyObject *module, *guards, *packed, *sz, *bias;
  int group;
  unsigned long long err;
  if (!PyArg_ParseTuple(args, "OOOOOiK", &module, &guards, &packed, &sz, &bias, &group, &err)) return nullptr;
  auto p = std::make_unique<W4Plan>();
  if (!tensor_arg(packed, p->packed, at::kInt) || !tensor_arg(sz, p->scale_zero, at::kHalf) ||
      !tensor_arg(bias, p->bias, at::kHalf, true))
    return nullptr;
  p->n = static_cast<int>(p->packed.size(0));
  p->k = static_cast<int>(p->packed.size(1) * 8);
  p->group = group;
  p->error_word = int_pointer(err);
  const at::Tensor on = p->packed;
  return wrap_plan(std::move(p), module, guards, on);
  END_HANDLE_TH_ERRORS
}

PyObject* w8_plan(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  PyObject *module, *guards, *weight, *scale, *bias;
  unsigned long long err;
  if (!PyArg_ParseTuple(args, "OOOOOK", &module, &guards, &weight, &scale, &bias, &err)) return nullptr;
  auto p = std::make_unique<W8Plan>();
  if (!tensor_arg(weight, p->weight, at::kChar) || !tensor_arg(scale, p->weight_scale, at::kFloat) ||
      !tensor_arg(bias, p->bias, at::kHalf, true))
    return nullptr;
  p->n = static_cast<int>(p->weight.size(0));
  p->k = static_cast<int>(p->weight.size(1));
  p->error_word = int_pointer(err);
  const at::Tensor on = p->weight;
  return wrap_plan(std::move(p), module, guards, on);
  END_HANDLE_TH_ERRORS
}

PyObject* affine_plan(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  PyObject *module, *guards, *weight, *scale, *zero, *rowsum, *bias;
  unsigned long long err;
  if (!PyArg_ParseTuple(args, "OOOOOOOK", &module, &guards, &weight, &scale, &zero, &rowsum, &bias, &err)) return nullptr;
  auto p = std::make_unique<AffinePlan>();
  if (!tensor_arg(weight, p->weight, at::kByte) || !tensor_arg(scale, p->scale, at::kFloat) ||
      !tensor_arg(zero, p->zero, at::kFloat) || !tensor_arg(rowsum, p->rowsum, at::kInt) ||
      !tensor_arg(bias, p->bias, at::kHalf, true))
    return nullptr;
  p->n = static_cast<int>(p->weight.size(0));
  p->k = static_cast<int>(p->weight.size(1));
  p->error_word = int_pointer(err);
  const at::Tensor on = p->weight;
  return wrap_plan(std::move(p), module, guards, on);
  END_HANDLE_TH_ERRORS
}

PyObject* moe_plan(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  PyObject *module, *guards, *w13, *s13, *w2, *s2;
  int lo, hi;
  unsigned long long err;
  if (!PyArg_ParseTuple(args, "OOOOOOiiK", &module, &guards, &w13, &s13, &w2, &s2, &lo, &hi, &err)) return nullptr;
  auto p = std::make_unique<MoePlan>();
  if (!tensor_arg(w13, p->w13, at::kChar) || !tensor_arg(s13, p->w13_scale, at::kFloat) ||
      !tensor_arg(w2, p->w2, at::kChar) || !tensor_arg(s2, p->w2_scale, at::kFloat))
    return nullptr;
  p->h = static_cast<int>(p->w13.size(2));
  p->i = static_cast<int>(p->w2.size(2));
  p->lo = lo;
  p->hi = hi;
  p->error_word = int_pointer(err);
  const at::Tensor on = p->w13;
  return wrap_plan(std::move(p), module, guards, on);
  END_HANDLE_TH_ERRORS
}

// (packed, scale, zero) of an fp16 weight the caller has checked, or the error status as an int
PyObject* w4_quantize(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  PyObject* weight;
  int group;
  if (!PyArg_ParseTuple(args, "Oi", &weight, &group)) return nullptr;
  at::Tensor w;
  if (!tensor_arg(weight, w, at::kHalf)) return nullptr;
  const int64_t n = w.size(0), k = w.size(1), groups = k / group;
  const auto opt = w.options().requires_grad(false);
  at::Tensor packed = at::empty({n, k / 8}, opt.dtype(at::kInt));
  at::Tensor scale = at::empty({n, groups}, opt);
  at::Tensor zero = at::empty({n, (groups + 7) / 8}, opt.dtype(at::kInt));
  const int rc = mp_w4a16_quantize(w.data_ptr(), static_cast<int>(n), static_cast<int>(k), group, packed.data_ptr(),
                                   scale.data_ptr(), zero.data_ptr(), c10::cuda::getCurrentCUDAStream().stream());
  if (rc != MP_OK) return PyLong_FromLong(rc);
  return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(packed)), THPVariable_Wrap(std::move(scale)),
                       THPVariable_Wrap(std::move(zero)));
  END_HANDLE_TH_ERRORS
}

// the expanded fp16 weight of checked buffers, or the error status as an int
PyObject* w4_dequant(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  PyObject *po, *so, *zo;
  int n, k, group;
  if (!PyArg_ParseTuple(args, "OOOiii", &po, &so, &zo, &n, &k, &group)) return nullptr;
  at::Tensor packed, scale, zero;
  if (!tensor_arg(po, packed, at::kInt) || !tensor_arg(so, scale, at::kHalf) || !tensor_arg(zo, zero, at::kInt, true))
    return nullptr;
  at::Tensor out = at::empty({n, k}, scale.options().requires_grad(false));
  const int rc = mp_w4a16_dequant(packed.data_ptr(), scale.data_ptr(), data_or_null(zero), n, k, group, out.data_ptr(),
                                  c10::cuda::getCurrentCUDAStream().stream());
  if (rc != MP_OK) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyObject* py_workspace(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  unsigned long long nbytes;
  int device, own_in_capture = 0;
  const char* name;
  if (!PyArg_ParseTuple(args, "Kis|p", &nbytes, &device, &name, &own_in_capture)) return nullptr;
  for (int kind = 0; kind < kKinds; ++kind)
    if (std::string(name) == kKindNames[kind]) {
      const cudaStream_t st = c10::cuda::getCurrentCUDAStream().stream();
      return THPVariable_Wrap(workspace(static_cast<size_t>(nbytes), device, st, kind, own_in_capture != 0));
    }
  PyErr_Format(PyExc_ValueError, "unknown workspace kind %s", name);
  return nullptr;
  END_HANDLE_TH_ERRORS
}

// every cached scratch buffer and every graph's, as (device index, tensor)
PyObject* py_workspaces(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  std::vector<std::pair<int, at::Tensor>> all;
  {
    std::lock_guard<std::mutex> lock(g_workspace_mutex);
    for (auto& kv : g_workspaces)
      if (kv.second.defined()) all.emplace_back(std::get<0>(kv.first), kv.second);
    for (auto& kv : g_captures)
      for (auto& t : kv.second.buffers) all.emplace_back(std::get<0>(kv.first), t);
  }
  PyObject* list = PyList_New(0);
  for (auto& it : all) {
    PyObject* t = THPVariable_Wrap(it.second);
    PyObject* pair = t ? Py_BuildValue("(iN)", it.first, t) : nullptr;
    if (!pair || PyList_Append(list, pair) != 0) {
      Py_XDECREF(pair);
      Py_DECREF(list);
      return nullptr;
    }
    Py_DECREF(pair);
  }
  return list;
  END_HANDLE_TH_ERRORS
}

PyMethodDef module_methods[] = {{"w4_plan", w4_plan, METH_VARARGS, nullptr},
                                {"w8_plan", w8_plan, METH_VARARGS, nullptr},
                                {"affine_plan", affine_plan, METH_VARARGS, nullptr},
                                {"moe_plan", moe_plan, METH_VARARGS, nullptr},
                                {"w4_quantize", w4_quantize, METH_VARARGS, nullptr},
                                {"w4_dequant", w4_dequant, METH_VARARGS, nullptr},
                                {"workspace", py_workspace, METH_VARARGS, nullptr},
                                {"workspaces", py_workspaces, METH_NOARGS, nullptr},
                                {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  plan_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&plan_spec));
  if (!plan_type) return nullptr;
  return PyModule_Create(&module_def);
}
