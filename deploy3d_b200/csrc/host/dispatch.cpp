// Host path of a plugin call: torch tensors in, C-ABI enqueue out, without the interpreter in between.
//
// The Python classes of plugins.py used to build two descriptor arrays, two pointer arrays and three foreign-function
// calls per enqueue: 35-45 us of interpreter time, more than the kernels of most single operators take.  `enqueue`
// below does the same steps natively (B200 host: 5 us plus the launches).  What only depends on the shapes and types
// of the inputs and on the plugin's parameters -- output descriptors, workspace size -- is kept per plugin for the
// last few signatures seen and compared in full on every call.
//
// The library's entry points arrive as addresses (the package decides which build of the library is loaded), so this
// module links against torch only.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string.h>
#include <unistd.h>

#include <atomic>
#include <condition_variable>
#include <mutex>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "../../../include/deploy3d_b200.h"

namespace {

using DescFn = int (*)(const void*, const d3d_tensor_desc*, int, int, d3d_tensor_desc*);
using WorkspaceFn = int (*)(const void*, const d3d_tensor_desc*, int, size_t*);
using EnqueueFn = int (*)(const void*, const d3d_tensor_desc*, int, const d3d_tensor_desc*, int, const void* const*,
                          void* const*, void*, size_t, void*);

constexpr int kMaxTensors = 32;
constexpr size_t kSignatures = 8;  // shapes a plugin object is called with in turn before the oldest is dropped

struct Signature {
  std::vector<unsigned char> params;
  std::vector<d3d_tensor_desc> in, out;
  size_t workspace = 0;
};

struct Call {
  PyObject_HEAD
  std::string* name;    // plugin name, for messages
  std::string* prefix;  // C-ABI prefix, for messages
  DescFn desc;
  WorkspaceFn workspace;
  EnqueueFn enqueue;
  std::vector<Signature>* seen;
  size_t oldest;
};

PyObject* g_check = nullptr;      // check(function name, status): raises
PyObject* g_workspace = nullptr;  // interned "_workspace"

int dtype_of(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return D3D_FLOAT;
    case at::kHalf: return D3D_HALF;
    case at::kInt: return D3D_INT32;
    case at::kBFloat16: return D3D_BF16;
    case at::kChar: return D3D_INT8;
    case at::kBool: return D3D_BOOL;
    default: return -1;
  }
}
at::ScalarType scalar_of(int dtype) {
  switch (dtype) {
    case D3D_FLOAT: return at::kFloat;
    case D3D_HALF: return at::kHalf;
    case D3D_INT32: return at::kInt;
    case D3D_BF16: return at::kBFloat16;
    case D3D_INT8: return at::kChar;
    default: return at::kBool;
  }
}

bool describe(const at::Tensor& t, d3d_tensor_desc* d) {
  const int dt = dtype_of(t);
  if (dt < 0) {
    PyErr_Format(PyExc_TypeError, "unsupported tensor dtype %s", c10::toString(t.scalar_type()));
    return false;
  }
  if (t.dim() > D3D_MAX_DIMS) {
    PyErr_Format(PyExc_IndexError, "tensors of at most %d dimensions, got %d", D3D_MAX_DIMS, (int)t.dim());
    return false;
  }
  memset(d, 0, sizeof(*d));
  d->dtype = dt;
  d->nb_dims = (int32_t)t.dim();
  for (int i = 0; i < d->nb_dims; ++i) d->dims[i] = t.size(i);
  return true;
}

// Raises through the package's own check(); always returns null.
PyObject* fail(const Call* c, const char* what, int status) {
  PyObject* r = PyObject_CallFunction(g_check, "si", (*c->prefix + what).c_str(), status);
  Py_XDECREF(r);
  if (r) PyErr_SetString(PyExc_RuntimeError, "plugin call failed");
  return nullptr;
}

// The kept signature of these inputs, made on first sight; null with an exception set when the library refuses.
const Signature* signature(Call* c, const void* params, size_t params_size, const d3d_tensor_desc* in, int n_in,
                           int n_out) {
  const unsigned char* pb = params_size ? reinterpret_cast<const unsigned char*>(params)
                                        : reinterpret_cast<const unsigned char*>(&params);
  const size_t pn = params_size ? params_size : sizeof(params);
  for (const Signature& s : *c->seen)
    if ((int)s.in.size() == n_in && (int)s.out.size() == n_out && s.params.size() == pn &&
        memcmp(s.params.data(), pb, pn) == 0 && memcmp(s.in.data(), in, n_in * sizeof(*in)) == 0)
      return &s;
  Signature s;
  s.params.assign(pb, pb + pn);
  s.in.assign(in, in + n_in);
  s.out.resize(n_out);
  for (int i = 0; i < n_out; ++i) {
    const int rc = c->desc(params, in, n_in, i, &s.out[i]);
    if (rc != D3D_OK) return fail(c, "_output_desc", rc), nullptr;
  }
  if (c->workspace) {
    const int rc = c->workspace(params, in, n_in, &s.workspace);
    if (rc != D3D_OK) return fail(c, "_workspace", rc), nullptr;
  }
  if (c->seen->size() < kSignatures) {
    c->seen->push_back(std::move(s));
    return &c->seen->back();
  }
  Signature& slot = (*c->seen)[c->oldest];
  c->oldest = (c->oldest + 1) % kSignatures;
  slot = std::move(s);
  return &slot;
}

// Whether a kernel can follow the tensor's address: on a GPU, in pinned host memory, or without elements (a shape).
bool reachable(const at::Tensor& t) { return t.is_cuda() || t.numel() == 0 || (t.is_cpu() && t.is_pinned()); }

int64_t volume(const d3d_tensor_desc& d) {
  int64_t v = 1;
  for (int i = 0; i < d.nb_dims; ++i) v *= d.dims[i];
  return v;
}

bool stream_of(PyObject* obj, c10::Device device, void** out) {
  if (obj == Py_None) {
    *out = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    return true;
  }
  PyObject* v = PyObject_GetAttrString(obj, "cuda_stream");
  if (!v) {
    PyErr_Clear();
    v = PyNumber_Long(obj);
    if (!v) return false;
  }
  *out = PyLong_AsVoidPtr(v);
  Py_DECREF(v);
  return !PyErr_Occurred();
}

}  // namespace

namespace {

// enqueue(plugin, params address, params size (0: an opaque handle), number of outputs, inputs, outputs | None,
//         stream | None, keep the workspace) -> tuple of the output tensors
// The workspace is the plugin's `_workspace`, replaced when it is too small.  With keep = False the call takes one of its
// own and never looks at that attribute: calls of one plugin from several threads or streams then share nothing.
PyObject* call_enqueue(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Call* c = reinterpret_cast<Call*>(self);
  if (nargs != 8) {
    PyErr_SetString(PyExc_TypeError, "enqueue takes eight arguments");
    return nullptr;
  }
  PyObject* plugin = args[0];
  const void* params = PyLong_AsVoidPtr(args[1]);
  const size_t params_size = PyLong_AsSize_t(args[2]);
  const long n_out = PyLong_AsLong(args[3]);
  PyObject *inputs = args[4], *outputs = args[5];
  const int keep = PyObject_IsTrue(args[7]);
  if (PyErr_Occurred()) return nullptr;
  const Py_ssize_t n_in = PyTuple_Check(inputs) ? PyTuple_GET_SIZE(inputs) : -1;
  if (n_in < 0 || n_in > kMaxTensors || n_out < 0 || n_out > kMaxTensors) {
    PyErr_SetString(PyExc_TypeError, "too many tensors");
    return nullptr;
  }
  at::Tensor in[kMaxTensors];
  d3d_tensor_desc in_desc[kMaxTensors];
  const void* in_ptr[kMaxTensors];
  for (Py_ssize_t i = 0; i < n_in; ++i) {
    PyObject* o = PyTuple_GET_ITEM(inputs, i);
    if (!THPVariable_Check(o)) {
      PyErr_Format(PyExc_TypeError, "%s: input %zd is no tensor", c->name->c_str(), i);
      return nullptr;
    }
    in[i] = THPVariable_Unpack(o);
  }
  if (n_in == 0 || !in[0].is_cuda()) {
    PyErr_Format(PyExc_RuntimeError, "%s: inputs must be CUDA tensors; this library has no CPU path", c->name->c_str());
    return nullptr;
  }
  const c10::Device device = in[0].device();
  c10::cuda::CUDAGuard guard(device);
  for (Py_ssize_t i = 0; i < n_in; ++i) {
    if (!reachable(in[i])) {
      PyErr_Format(PyExc_RuntimeError, "%s: input %zd is not in CUDA memory", c->name->c_str(), i);
      return nullptr;
    }
    if (!in[i].is_contiguous()) in[i] = in[i].contiguous();
    if (!describe(in[i], &in_desc[i])) return nullptr;
    in_ptr[i] = in[i].numel() ? in[i].data_ptr() : nullptr;
  }
  const Signature* s = signature(c, params, params_size, in_desc, (int)n_in, (int)n_out);
  if (!s) return nullptr;
  // Copied before anything below can run Python code or let another thread in: a call of the same plugin with another
  // shape may take the entry over.
  const size_t ws_bytes = s->workspace;
  d3d_tensor_desc out_desc[kMaxTensors];
  void* out_ptr[kMaxTensors] = {};
  memcpy(out_desc, s->out.data(), n_out * sizeof(d3d_tensor_desc));
  s = nullptr;
  PyObject* result;
  if (outputs == Py_None) {
    result = PyTuple_New(n_out);
    if (!result) return nullptr;
    for (long i = 0; i < n_out; ++i) {
      at::Tensor t = at::empty(at::IntArrayRef(out_desc[i].dims, out_desc[i].nb_dims),
                               at::TensorOptions().dtype(scalar_of(out_desc[i].dtype)).device(device));
      out_ptr[i] = t.numel() ? t.data_ptr() : nullptr;
      PyTuple_SET_ITEM(result, i, THPVariable_Wrap(std::move(t)));
    }
  } else {  // the caller's buffers say which of the accepted output types it wants (GatherBack can widen)
    result = PySequence_Tuple(outputs);
    if (!result) return nullptr;
    const Py_ssize_t given = PyTuple_GET_SIZE(result);
    for (Py_ssize_t i = given; i < n_out; ++i)
      if (volume(out_desc[i]) != 0) {
        PyErr_Format(PyExc_ValueError, "%s: %zd of %ld outputs given", c->name->c_str(), given, n_out);
        Py_DECREF(result);
        return nullptr;
      }
    for (Py_ssize_t i = 0; i < given && i < n_out; ++i) {
      PyObject* o = PyTuple_GET_ITEM(result, i);
      if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s: output %zd is no tensor", c->name->c_str(), i);
        Py_DECREF(result);
        return nullptr;
      }
      const at::Tensor& t = THPVariable_Unpack(o);
      const int dt = dtype_of(t);
      if (dt < 0) {
        PyErr_Format(PyExc_KeyError, "unsupported tensor dtype %s", c10::toString(t.scalar_type()));
        Py_DECREF(result);
        return nullptr;
      }
      if (!reachable(t)) {
        PyErr_Format(PyExc_RuntimeError, "%s: output %zd is not in CUDA memory", c->name->c_str(), i);
        Py_DECREF(result);
        return nullptr;
      }
      out_desc[i].dtype = dt;
      out_ptr[i] = t.numel() ? t.data_ptr() : nullptr;
    }
  }
  at::Tensor ws;  // held until the launches are in the stream, whatever another thread does to the plugin meanwhile
  if (ws_bytes && !keep) {
    ws = at::empty({(int64_t)ws_bytes}, at::TensorOptions().dtype(at::kByte).device(device));
  } else if (ws_bytes) {
    PyObject* have = PyObject_GetAttr(plugin, g_workspace);
    if (!have) {
      Py_DECREF(result);
      return nullptr;
    }
    if (THPVariable_Check(have)) {
      const at::Tensor& t = THPVariable_Unpack(have);
      if ((size_t)t.numel() >= ws_bytes && t.device() == device) ws = t;
    }
    Py_DECREF(have);
    if (!ws.defined()) {
      ws = at::empty({(int64_t)ws_bytes}, at::TensorOptions().dtype(at::kByte).device(device));
      PyObject* o = THPVariable_Wrap(ws);
      const int rc = o ? PyObject_SetAttr(plugin, g_workspace, o) : -1;
      Py_XDECREF(o);
      if (rc) {
        Py_DECREF(result);
        return nullptr;
      }
    }
  }
  void* ws_ptr = ws_bytes ? ws.data_ptr() : nullptr;
  void* stream;
  if (!stream_of(args[6], device, &stream)) {
    Py_DECREF(result);
    return nullptr;
  }
  int status;
  Py_BEGIN_ALLOW_THREADS;
  status = c->enqueue(params, in_desc, (int)n_in, out_desc, (int)n_out, in_ptr, out_ptr, ws_ptr, ws_bytes, stream);
  Py_END_ALLOW_THREADS;
  if (status != D3D_OK) {
    Py_DECREF(result);
    return fail(c, "_enqueue", status);
  }
  return result;
  END_HANDLE_TH_ERRORS
}

PyObject* call_new(PyTypeObject* type, PyObject* args, PyObject*) {
  const char *name, *prefix;
  unsigned long long desc, workspace, enqueue;
  if (!PyArg_ParseTuple(args, "ssKKK", &name, &prefix, &desc, &workspace, &enqueue)) return nullptr;
  Call* c = reinterpret_cast<Call*>(type->tp_alloc(type, 0));
  if (!c) return nullptr;
  c->name = new std::string(name);
  c->prefix = new std::string(prefix);
  c->desc = reinterpret_cast<DescFn>(desc);
  c->workspace = reinterpret_cast<WorkspaceFn>(workspace);
  c->enqueue = reinterpret_cast<EnqueueFn>(enqueue);
  c->seen = new std::vector<Signature>();
  c->seen->reserve(kSignatures);
  c->oldest = 0;
  return reinterpret_cast<PyObject*>(c);
}
void call_dealloc(PyObject* self) {
  Call* c = reinterpret_cast<Call*>(self);
  delete c->name;
  delete c->prefix;
  delete c->seen;
  Py_TYPE(self)->tp_free(self);
}

PyMethodDef call_methods[] = {
    {"enqueue", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_enqueue)), METH_FASTCALL,
     "enqueue(plugin, params, params_size, n_out, inputs, outputs, stream, keep) -> tuple of output tensors"},
    {nullptr, nullptr, 0, nullptr}};
PyTypeObject call_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// Compares two large buffers with up to three helper threads beside the caller: one core reads two 1.8 MB weight arrays in
// 93 us (they come from its neighbours' caches), four in 30-40 us.  The buffers are dealt out in pieces and the caller takes
// pieces too, so it waits only for helpers that are in the middle of one: a helper that is asleep, or was never started
// because the process may have no more threads, costs nothing but its share.  Helpers sleep between calls; a second caller
// that finds them busy compares alone.  They are started at first use, and not in a forked child.
class Comparer {
 public:
  static constexpr int kHelpers = 3;
  static constexpr size_t kWorthIt = 256 << 10, kPiece = 64 << 10;

  bool same(const char* a, const char* b, size_t n) {
    const uint64_t pieces = (n + kPiece - 1) / kPiece;
    if (n < kWorthIt || pieces > kPieces || getpid() != pid_ || !turn_.try_lock()) return memcmp(a, b, n) == 0;
    std::lock_guard<std::mutex> turn(turn_, std::adopt_lock);
    if (!started_) {
      started_ = true;
      try {
        for (int i = 0; i < kHelpers; ++i) std::thread([this] { help(); }).detach();
      } catch (const std::system_error&) {  // as many as there are
      }
    }
    a_ = a, b_ = b, n_ = n;
    differ_.store(false, std::memory_order_relaxed);
    done_.store(0, std::memory_order_relaxed);
    uint64_t job;
    {
      std::lock_guard<std::mutex> g(lock_);
      job = ++job_;
      left_.store(job << 32 | pieces, std::memory_order_release);
    }
    wake_.notify_all();
    work(job);
    while (done_.load(std::memory_order_acquire) < pieces) std::this_thread::yield();  // pieces in helpers' hands
    return !differ_.load(std::memory_order_relaxed);
  }

 private:
  static constexpr uint64_t kPieces = 0xffffffffu;

  // Takes pieces of `job` while there are any.  `left_` holds the job and the number of its pieces nobody has taken in one
  // word: a helper that comes late finds another job or none left, and reads nothing else.  The buffers of a job stay as
  // they are while one of its pieces is taken and not done.
  void work(uint64_t job) {
    uint64_t at = left_.load(std::memory_order_acquire);
    while ((uint32_t)(at >> 32) == (uint32_t)job && (at & kPieces) != 0) {
      if (!left_.compare_exchange_weak(at, at - 1, std::memory_order_acq_rel, std::memory_order_acquire)) continue;
      const size_t from = ((at & kPieces) - 1) * kPiece, len = n_ - from < kPiece ? n_ - from : kPiece;
      if (!differ_.load(std::memory_order_relaxed) && memcmp(a_ + from, b_ + from, len) != 0)
        differ_.store(true, std::memory_order_relaxed);
      done_.fetch_add(1, std::memory_order_release);
      at = left_.load(std::memory_order_acquire);
    }
  }
  void help() {
    uint64_t seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> g(lock_);
        wake_.wait(g, [&] { return job_ != seen; });
        seen = job_;
      }
      work(seen);
    }
  }
  const pid_t pid_ = getpid();
  std::mutex turn_, lock_;
  std::condition_variable wake_;
  std::atomic<uint64_t> left_{0}, done_{0};
  std::atomic<bool> differ_{false};
  bool started_ = false;
  uint64_t job_ = 0;
  const char *a_ = nullptr, *b_ = nullptr;
  size_t n_ = 0;
};
Comparer* comparer() {
  static Comparer* c = new Comparer();  // never destroyed: the helpers outlive the module's statics
  return c;
}

// same_bytes(a, b, offset of b): whether the buffer `a` equals the bytes of `b` from `offset` on.
PyObject* same_bytes(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  Py_buffer a, b;
  if (nargs != 3) {
    PyErr_SetString(PyExc_TypeError, "same_bytes takes three arguments");
    return nullptr;
  }
  const Py_ssize_t off = PyLong_AsSsize_t(args[2]);
  if (PyErr_Occurred()) return nullptr;
  if (PyObject_GetBuffer(args[0], &a, PyBUF_SIMPLE) != 0) return nullptr;  // contiguous buffers only
  if (PyObject_GetBuffer(args[1], &b, PyBUF_SIMPLE) != 0) {
    PyBuffer_Release(&a);
    return nullptr;
  }
  bool same = off >= 0 && off <= b.len && a.len <= b.len - off;
  if (same) {
    Py_BEGIN_ALLOW_THREADS;
    same = comparer()->same(static_cast<const char*>(a.buf), static_cast<const char*>(b.buf) + off, (size_t)a.len);
    Py_END_ALLOW_THREADS;
  }
  PyBuffer_Release(&a);
  PyBuffer_Release(&b);
  return PyBool_FromLong(same);
}

PyObject* set_check(PyObject*, PyObject* fn) {
  Py_INCREF(fn);
  Py_XSETREF(g_check, fn);
  Py_RETURN_NONE;
}

PyMethodDef module_methods[] = {
    {"same_bytes", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(same_bytes)), METH_FASTCALL,
     "same_bytes(a, b, offset): whether buffer a equals the bytes of b from offset on"},
    {"set_check", set_check, METH_O, "set_check(check): the function that raises for a C-ABI status"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_d3d_host", nullptr, -1, module_methods};

}  // namespace

PyMODINIT_FUNC PyInit__d3d_host() {
  call_type.tp_name = "_d3d_host.Call";
  call_type.tp_basicsize = sizeof(Call);
  call_type.tp_flags = Py_TPFLAGS_DEFAULT;
  call_type.tp_new = call_new;
  call_type.tp_dealloc = call_dealloc;
  call_type.tp_methods = call_methods;
  if (PyType_Ready(&call_type) < 0) return nullptr;
  g_workspace = PyUnicode_InternFromString("_workspace");
  PyObject* m = PyModule_Create(&module_def);
  if (!m) return nullptr;
  Py_INCREF(&call_type);
  if (PyModule_AddObject(m, "Call", reinterpret_cast<PyObject*>(&call_type)) < 0) return nullptr;
  return m;
}
