// The module calls' host path in native code.
//
// One eager LinearQ call spent 19 us in Python (attribute lookups through nn.Module, argument checks, an allocation, a
// fifteen-argument ctypes call) around a launch of 2 us and, for decode sizes, a kernel of 4 us: a program calling layer
// after layer was bound by the interpreter up to about 1500 tokens.  The functions here do the same work -- the same
// checks, the same allocation, the same C-ABI call -- for the ordinary case, and return None for everything else (wrong
// types, CPU tensors, other devices, non-contiguous operands, empty inputs, tensor subclasses, dispatch modes), which the
// Python code then handles and reports exactly as before.
//
// The interpreter lock is held while Python objects are looked at, and given up around the allocations and the C-ABI calls, as
// torch's own operators and ctypes do: an allocation or a launch may wait (for memory, for room in the launch queue), and
// neither the program's other threads nor a host function on the stream that needs the lock may have to wait with it.  What
// the call uses is held by reference across it, since another thread may replace a layer's buffers or grow the workspace.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <map>
#include <mutex>

#include "../../include/asrq_b200.h"

namespace {

std::atomic<long long> g_calls{0};   // C-ABI calls made here
PyObject* g_workspaces = nullptr;    // linear._workspaces: (device index, stream) -> uint8 tensor
PyObject* g_check = nullptr;         // _lib.check(function name, status): raises AsrqError

struct Names {
  PyObject *buffers, *weight, *scales, *zeros, *bias, *in_features, *out_features, *bits, *group_size, *hadamard, *operand, *w8;
} N;

bool intern_names() {
  auto s = [](const char* t) { return PyUnicode_InternFromString(t); };
  N = {s("_buffers"), s("weight"), s("scales"), s("zeros"), s("bias"), s("in_features"), s("out_features"), s("bits"), s("group_size"),
       s("hadamard"), s("operand"), s("_w8")};
  return !PyErr_Occurred();
}

// Plain strided tensors outside any tensor-subclass or dispatch mode; everything else takes the Python path.
inline const at::Tensor* plain(PyObject* o) { return o && THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
inline bool modes_active() {
  return at::impl::PythonTorchFunctionTLS::stack_len() != 0 || c10::impl::TorchDispatchModeTLS::any_modes_set();
}
inline bool int_of(PyObject* dict, PyObject* name, long long* out) {
  PyObject* v = PyDict_GetItemWithError(dict, name);
  if (!v || !PyLong_Check(v)) return false;
  *out = PyLong_AsLongLong(v);
  return true;
}

// Gives up the interpreter lock for a scope (an exception takes it again on its way out).
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  Unlocked() = default;
  Unlocked(const Unlocked&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// A tensor held by its Python object.  (Copies of the at::Tensor, an atomic count each that reaches the Python object too, made a
// call of 4.9 us one of 5.2.)
class Held {
 public:
  Held() = default;
  Held(const Held&) = delete;
  ~Held() { Py_XDECREF(o_); }
  void operator=(PyObject* o) {
    Py_INCREF(o);
    Py_XDECREF(o_);
    o_ = o;
  }
  explicit operator bool() const { return o_ != nullptr; }
  const at::Tensor& operator*() const { return THPVariable_Unpack(o_); }
  const at::Tensor* operator->() const { return &THPVariable_Unpack(o_); }

 private:
  PyObject* o_ = nullptr;
};

struct Layer {
  Held weight, scales, zeros, bias;  // bias empty: none
  PyObject* dict;
  long long k, n, bits, group;
};

// The layer's operands as module attributes hold them (registered buffers, or plain attributes).  False: not the ordinary case.
bool layer_of(PyObject* self, const c10::Device& dev, Layer* L) {
  PyObject** dp = _PyObject_GetDictPtr(self);
  if (!dp || !*dp) return false;
  PyObject* d = L->dict = *dp;
  PyObject* buf = PyDict_GetItemWithError(d, N.buffers);
  if (!buf || !PyDict_Check(buf)) return false;
  auto operand = [&](PyObject* name, PyObject** obj) {
    *obj = PyDict_GetItemWithError(buf, name);
    if (!*obj) *obj = PyDict_GetItemWithError(d, name);
    return *obj != nullptr;
  };
  PyObject *w, *s, *z, *b;
  if (!operand(N.weight, &w) || !operand(N.scales, &s) || !operand(N.zeros, &z) || !operand(N.bias, &b)) return false;
  const at::Tensor *wt = plain(w), *st = plain(s), *zt = plain(z), *bt = plain(b);
  if (!wt || !st || !zt || (b != Py_None && !bt)) return false;
  if (wt->scalar_type() != at::kByte || st->scalar_type() != at::kHalf || zt->scalar_type() != at::kHalf) return false;
  for (const at::Tensor* t : {wt, st, zt})
    if (t->device() != dev || !t->is_contiguous()) return false;
  if (bt && (bt->scalar_type() != at::kHalf || bt->device() != dev)) return false;
  L->weight = w;
  L->scales = s;
  L->zeros = z;
  if (bt) L->bias = b;
  return int_of(d, N.in_features, &L->k) && int_of(d, N.out_features, &L->n) && int_of(d, N.bits, &L->bits) && int_of(d, N.group_size, &L->group);
}

// fp16 / bf16 activations on the current CUDA device, contiguous, at least one row
bool activations(PyObject* o, Held* x, int* dtype) {
  const at::Tensor* t = plain(o);
  if (!t || !t->is_cuda() || t->dim() < 1 || !t->is_contiguous() || t->numel() == 0) return false;
  const auto st = t->scalar_type();
  if (st != at::kHalf && st != at::kBFloat16) return false;
  *x = o;
  *dtype = st == at::kHalf ? ASRQ_F16 : ASRQ_BF16;
  return t->device().index() == c10::cuda::current_device() && !modes_active();
}

// The stream's workspace if it is there and large enough.
bool workspace(int dev, cudaStream_t stream, size_t need, Held* ws) {
  PyObject* key = PyTuple_New(2);
  if (!key) return false;
  PyTuple_SET_ITEM(key, 0, PyLong_FromLong(dev));
  PyTuple_SET_ITEM(key, 1, PyLong_FromVoidPtr(stream));
  PyObject* v = PyDict_GetItemWithError(g_workspaces, key);
  Py_DECREF(key);
  const at::Tensor* t = plain(v);
  if (!t || size_t(t->numel()) < need) return false;
  *ws = v;
  return true;
}

bool contains(PyObject* streams, cudaStream_t stream) {
  PyObject* handle = PyLong_FromVoidPtr(stream);
  if (!handle) return false;
  const int in = PySet_Contains(streams, handle);
  Py_DECREF(handle);
  return in == 1;
}

at::Tensor output_like(const at::Tensor& x, int64_t n) {
  c10::SmallVector<int64_t, 5> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = n;
  return at::detail::empty_cuda(shape, x.scalar_type(), x.device(), std::nullopt);
}

// Memory of a large call's own for its weights as 16-bit values, from torch's allocator: on a shared stream a block that no other call
// has, under capture the graph's.  Undefined where the call needs none, and where there is none to be had: the kernels that unpack inside
// the GEMM run then.
at::Tensor weights_scratch(int64_t bytes, const c10::Device& device) {
  if (bytes == 0) return at::Tensor();
  try {
    return at::detail::empty_cuda({bytes}, at::kByte, device, std::nullopt);
  } catch (const c10::OutOfMemoryError&) {
    return at::Tensor();
  }
}

PyObject* failed(const char* fn, int rc) {
  PyObject* r = PyObject_CallFunction(g_check, "si", fn, rc);
  Py_XDECREF(r);
  if (r) PyErr_Format(PyExc_RuntimeError, "%s failed with status %d", fn, rc);
  return nullptr;
}

// linearq_forward(layer, input, residual or None, gelu) -> output, or None: not the ordinary case
PyObject* linearq_forward(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  if (n_args != 4) {
    PyErr_SetString(PyExc_TypeError, "linearq_forward(layer, input, residual, gelu)");
    return nullptr;
  }
  Held x;
  int dtype;
  Layer L;
  if (!activations(a[1], &x, &dtype) || !layer_of(a[0], x->device(), &L) || (L.bits != 2 && L.bits != 4) || x->size(-1) != L.k) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const int64_t m = x->numel() / L.k;
  Held res;
  if (a[2] != Py_None) {
    const at::Tensor* r = plain(a[2]);
    if (!r || r->scalar_type() != x->scalar_type() || r->device() != x->device() || r->numel() != m * L.n || !r->is_contiguous()) Py_RETURN_NONE;
    res = a[2];
  }
  const bool gelu = a[3] == Py_True, fused = bool(res) || gelu;
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  Held ws;
  if (!workspace(x->device().index(), stream, asrq_workspace_bytes(ASRQ_WS_LINEARQ, m, L.n, L.k), &ws)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;  // the Python path makes it
  }
  at::Tensor y;
  int rc;
  {
    Unlocked unlocked;
    y = output_like(*x, L.n);
    g_calls.fetch_add(1, std::memory_order_relaxed);
    const void* bias = L.bias ? L.bias->data_ptr() : nullptr;
    const int act = gelu ? ASRQ_ACT_GELU : ASRQ_ACT_NONE;
    const at::Tensor w16 = weights_scratch(int64_t(asrq_linearq_a16_scratch_bytes(m, L.n, L.k, int(L.group), act, bool(res))), x->device());
    rc = asrq_linearq_a16_scratch(int(L.bits), x->data_ptr(), static_cast<const uint8_t*>(L.weight->data_ptr()), L.scales->data_ptr(), L.zeros->data_ptr(),
                                  bias, res ? res->data_ptr() : nullptr, y.data_ptr(), m, L.n, L.k, int(L.group), dtype, act, ws->data_ptr(),
                                  size_t(ws->numel()), w16.defined() ? w16.data_ptr() : nullptr, w16.defined() ? size_t(w16.numel()) : 0, stream);
  }
  if (rc) return failed(fused ? "asrq_linearq_a16_fused" : "asrq_linearq_a16", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// linearqq_forward(layer, input) -> output, or None
PyObject* linearqq_forward(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  if (n_args != 2) {
    PyErr_SetString(PyExc_TypeError, "linearqq_forward(layer, input)");
    return nullptr;
  }
  Held x;
  int dtype;
  Layer L;
  if (!activations(a[1], &x, &dtype) || !layer_of(a[0], x->device(), &L) || x->size(-1) != L.k || L.group <= 0) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  PyObject* had_o = PyDict_GetItemWithError(L.dict, N.hadamard);
  if (had_o != Py_True && had_o != Py_False) Py_RETURN_NONE;
  const int had = had_o == Py_True;
  const int64_t m = x->numel() / L.k;
  const int dev = x->device().index();
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  const void* bias = L.bias ? L.bias->data_ptr() : nullptr;
  Held ws, w8;
  at::Tensor sc, y;
  const char* fn;
  int rc;
  // the activation codes and their scales: one scratch allocation (codes first, the scales at the next multiple of 256 bytes)
  auto scratch = [&](int64_t code_bytes) {
    return at::detail::empty_cuda({(code_bytes + 255) / 256 * 256 + m * 4}, at::kByte, x->device(), std::nullopt);
  };
  if (m >= 64 && L.n % 128 == 0 && L.k % 128 == 0 && L.group % 128 == 0 && L.k % L.group == 0) {
    PyObject* op = PyObject_GetAttr(a[0], N.operand);
    if (!op) return nullptr;
    const bool f8 = PyUnicode_Check(op) && PyUnicode_CompareWithASCIIString(op, "f8") == 0;
    const bool i8 = PyUnicode_Check(op) && PyUnicode_CompareWithASCIIString(op, "int8") == 0;
    // the prepared weight (linear._Prepared), if it was derived from this very buffer in this state and this stream is behind that
    PyObject* prepared = PyDict_GetItemWithError(L.dict, N.w8);
    if ((f8 || i8) && prepared && PyTuple_Check(prepared) && PyTuple_GET_SIZE(prepared) == 6) {
      const at::Tensor *t = plain(PyTuple_GET_ITEM(prepared, 0)), *src = plain(PyTuple_GET_ITEM(prepared, 1));
      if (t && src && t->device() == x->device() && src->device() == x->device() && src->data_ptr() == L.weight->data_ptr() &&
          PyLong_AsLongLong(PyTuple_GET_ITEM(prepared, 2)) == (long long)L.weight->_version() && PyUnicode_Compare(PyTuple_GET_ITEM(prepared, 3), op) == 0 &&
          contains(PyTuple_GET_ITEM(prepared, 4), stream))
        w8 = PyTuple_GET_ITEM(prepared, 0);
    }
    Py_DECREF(op);
    if (PyErr_Occurred()) return nullptr;
    if (!w8 || !workspace(dev, stream, 256, &ws)) {
      if (PyErr_Occurred()) return nullptr;
      Py_RETURN_NONE;
    }
    Unlocked unlocked;
    sc = scratch(m * L.k);
    y = output_like(*x, L.n);
    uint8_t* a8 = static_cast<uint8_t*>(sc.data_ptr());
    float* sa = reinterpret_cast<float*>(a8 + (m * L.k + 255) / 256 * 256);
    g_calls.fetch_add(2, std::memory_order_relaxed);
    fn = f8 ? "asrq_hadamard_quant_f8" : "asrq_hadamard_quant_int8";
    rc = (f8 ? asrq_hadamard_quant_f8 : asrq_hadamard_quant_int8)(x->data_ptr(), a8, sa, m, L.k, had, dtype, stream);
    if (!rc) {
      fn = f8 ? "asrq_w4a4_gemm_f8" : "asrq_w4a4_gemm_int8";
      rc = (f8 ? asrq_w4a4_gemm_f8 : asrq_w4a4_gemm_int8)(a8, sa, static_cast<const uint8_t*>(w8->data_ptr()), L.scales->data_ptr(), bias, y.data_ptr(), nullptr, m,
                                                          L.n, L.k, int(L.group), dtype, ws->data_ptr(), size_t(ws->numel()), stream);
    }
  } else {
    if (!workspace(dev, stream, asrq_workspace_bytes(ASRQ_WS_W4A4_GEMM, m, L.n, L.k), &ws)) {
      if (PyErr_Occurred()) return nullptr;
      Py_RETURN_NONE;
    }
    Unlocked unlocked;
    sc = scratch(m * (L.k / 2));
    y = output_like(*x, L.n);
    uint8_t* qa = static_cast<uint8_t*>(sc.data_ptr());
    float* sa = reinterpret_cast<float*>(qa + (m * (L.k / 2) + 255) / 256 * 256);
    g_calls.fetch_add(2, std::memory_order_relaxed);
    fn = "asrq_hadamard_quant_int4";
    rc = asrq_hadamard_quant_int4(x->data_ptr(), qa, sa, m, L.k, had, dtype, stream);
    if (!rc) {
      fn = "asrq_w4a4_gemm";
      rc = asrq_w4a4_gemm(qa, sa, static_cast<const uint8_t*>(L.weight->data_ptr()), L.scales->data_ptr(), bias, y.data_ptr(), nullptr, m, L.n, L.k, int(L.group),
                          dtype, ws->data_ptr(), size_t(ws->numel()), stream);
    }
  }
  if (rc) return failed(fn, rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

PyObject* calls(PyObject*, PyObject*) { return PyLong_FromLongLong(g_calls.load(std::memory_order_relaxed)); }

// A stream of this file's own per device: never under capture, which one of the pool that torch hands out round and round may be.
c10::cuda::CUDAStream own_stream(c10::DeviceIndex device) {
  static std::mutex mu;
  static std::map<int, cudaStream_t> streams;
  std::lock_guard<std::mutex> lock(mu);
  auto it = streams.find(device);
  if (it == streams.end()) {
    c10::cuda::CUDAGuard guard(device);
    cudaStream_t s;
    C10_CUDA_CHECK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    it = streams.emplace(device, s).first;
  }
  return c10::cuda::getStreamFromExternal(it->second, device);
}

// zeros_now(bytes, device) -> uint8 tensor that is zero on return, also while a stream is under capture: zeros made on that stream
// would be the graph's, there only once it has run, in memory of the graph's.
PyObject* zeros_now(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  long long bytes;
  int device;
  if (!PyArg_ParseTuple(args, "Li", &bytes, &device)) return nullptr;
  at::Tensor t;
  {
    Unlocked unlocked;
    c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    const c10::cuda::CUDAStream side = own_stream(c10::DeviceIndex(device));
    c10::cuda::CUDAStreamGuard guard(side);
    t = at::detail::empty_cuda({bytes}, at::kByte, c10::Device(c10::kCUDA, c10::DeviceIndex(device)), std::nullopt);
    C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, size_t(bytes), side.stream()));
    C10_CUDA_CHECK(cudaStreamSynchronize(side.stream()));
  }
  return THPVariable_Wrap(std::move(t));
  END_HANDLE_TH_ERRORS
}

// bind(workspaces dict, check function)
PyObject* bind(PyObject*, PyObject* args) {
  PyObject *ws, *check;
  if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &ws, &check)) return nullptr;
  Py_INCREF(ws);
  Py_INCREF(check);
  Py_XDECREF(g_workspaces);
  Py_XDECREF(g_check);
  g_workspaces = ws;
  g_check = check;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"linearq_forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linearq_forward)), METH_FASTCALL, nullptr},
    {"linearqq_forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linearqq_forward)), METH_FASTCALL, nullptr},
    {"calls", calls, METH_NOARGS, nullptr},
    {"zeros_now", zeros_now, METH_VARARGS, nullptr},
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return intern_names() ? PyModule_Create(&kModule) : nullptr; }
