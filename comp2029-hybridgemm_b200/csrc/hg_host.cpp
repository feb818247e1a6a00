// Host path of one layer call (`DualLinear.__call__`, `DualLinear.silu_linear`) as a CPython extension.
//
// A call at decode sizes is bounded by the host: 3.4 us of GPU time at 8 tokens of 896 -> 4864.  Through ctypes and
// torch's Python bindings the host needed 7.3 us a call, of which 2.4 us are the launch itself; the rest was the output
// allocation (1.9 us), the foreign call (0.9 us) and Python bytecode.  Here one C call checks the argument, finds the
// prepared state of the token count, allocates and launches: 4.4 us.
//
// The module holds no state of its own but the addresses of the library's entry points.  It is built against the torch
// that loads it and knows nothing of CUDA beyond the current stream.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>
#include <iterator>

#include "../../include/hygemm.h"

namespace {

decltype(&hg_linear) run_linear = nullptr;
decltype(&hg_linear_silu) run_linear_silu = nullptr;
decltype(&hg_last_error) last_error = nullptr;

PyObject *s_ready, *s_w4, *s_sf4, *s_lo, *s_w8, *s_sf8, *s_hi, *s_low_id, *s_high_id, *s_concurrent, *s_plans, *s_calls;

const char kName[] = "hygemm.ready";

// What calls of one layer with one token count share.  Valid while the layer's six operand tensors still lie where the
// structs say (an attribute may be replaced, and so may the storage behind one) and the schedule ids are the same.
struct Ready {
  PyObject *low_id, *high_id, *problems;              // owned
  void* handle;
  const hg_problem *low, *high;                       // inside `problems`
  int64_t tokens, k, outputs, packed;                 // packed: bytes of the quantised activations
  int fused;                                          // calls quantise inside the GEMM launch: 0 none, 1 all, 2 eager ones
  at::TensorOptions output;
  c10::Device device = c10::Device(c10::kCPU);
};

Ready* ready_of(PyObject* capsule) { return static_cast<Ready*>(PyCapsule_GetPointer(capsule, kName)); }

void destroy(PyObject* capsule) {
  Ready* r = ready_of(capsule);
  if (!r) return;
  for (PyObject* o : {r->low_id, r->high_id, r->problems}) Py_XDECREF(o);
  delete r;
}

// The attributes of a layer.  A call asks for eleven, so they are looked up in the instance's dict directly; one that is
// not there is asked for in the ordinary way.
struct Attributes {
  PyObject *layer, *dict;
  explicit Attributes(PyObject* of) : layer(of), dict(PyObject_GenericGetDict(of, nullptr)) {
    if (!dict) PyErr_Clear();
  }
  ~Attributes() { Py_XDECREF(dict); }
  Attributes(const Attributes&) = delete;
  // A new reference, or null with an error set.
  PyObject* get(PyObject* name) const {
    if (dict) {
      if (PyObject* found = PyDict_GetItemWithError(dict, name)) return Py_NewRef(found);
      if (PyErr_Occurred()) return nullptr;
    }
    return PyObject_GetAttr(layer, name);
  }
};

// True when attribute `name` is `wanted` (the same object, or an equal int).
bool unchanged(const Attributes& layer, PyObject* name, PyObject* wanted) {
  PyObject* now = layer.get(name);
  if (!now) { PyErr_Clear(); return false; }
  bool same = now == wanted;
  if (!same && PyLong_Check(now)) {
    const int equal = PyObject_RichCompareBool(now, wanted, Py_EQ);
    if (equal < 0) PyErr_Clear();
    same = equal == 1;
  }
  Py_DECREF(now);
  return same;
}

// True when attribute `name` is a tensor whose elements start at `data`, `elements` of them (-1: any number).
bool still_at(const Attributes& layer, PyObject* name, const void* data, int64_t elements = -1) {
  PyObject* now = layer.get(name);
  if (!now) { PyErr_Clear(); return false; }
  struct Release { PyObject* o; ~Release() { Py_DECREF(o); } } release{now};   // the tensor's accessors may throw
  if (!THPVariable_Check(now)) return false;
  const at::Tensor& t = THPVariable_Unpack(now);
  return t.const_data_ptr() == data && (elements < 0 || t.numel() == elements);
}

// True for the launch policies that all enqueue the tensor-core launch: False and True, 0 to 3.
bool tensor_core_policy(const Attributes& layer) {
  PyObject* now = layer.get(s_concurrent);
  if (!now) { PyErr_Clear(); return false; }
  bool plain = now == Py_True || now == Py_False;
  if (!plain) {
    PyObject* number = PyNumber_Long(now);
    const long policy = number ? PyLong_AsLong(number) : -1;
    PyErr_Clear();
    Py_XDECREF(number);
    plain = policy >= HG_POLICY_SERIAL && policy < HG_POLICY_GEMV_PAIR1;
  }
  Py_DECREF(now);
  return plain;
}

bool operands_unchanged(const Attributes& layer, const hg_problem& low, const hg_problem& high) {
  return still_at(layer, s_w4, low.weight) && still_at(layer, s_sf4, low.weight_scales) && still_at(layer, s_lo, low.ids, low.rows) &&
         still_at(layer, s_w8, high.weight) && still_at(layer, s_sf8, high.weight_scales) && still_at(layer, s_hi, high.ids, high.rows);
}

// The prepared state of a call, a new reference; null without an error when the call is not a prepared, ordinary one.
PyObject* find(const Attributes& layer, int64_t tokens) {
  PyObject* plans = layer.get(s_plans);
  if (!plans) return nullptr;
  const int planned = PyObject_IsTrue(plans);
  Py_DECREF(plans);
  if (planned) return nullptr;
  PyObject* all = layer.get(s_ready);
  if (!all) return nullptr;
  PyObject* capsule = nullptr;
  PyObject* key = PyLong_FromLongLong(tokens);
  if (key && PyDict_Check(all)) {
    capsule = PyDict_GetItemWithError(all, key);
    Py_XINCREF(capsule);
  }
  Py_XDECREF(key);
  Py_DECREF(all);
  return capsule;
}

bool count_call(const Attributes& layer, int64_t tokens) {
  PyObject* calls = layer.get(s_calls);
  if (!calls) return false;
  bool ok = false;
  PyObject* key = PyLong_FromLongLong(tokens);
  if (key && PyDict_Check(calls)) {
    PyObject* old = PyDict_GetItemWithError(calls, key);
    if (old || !PyErr_Occurred()) {
      PyObject* sum = PyLong_FromLongLong((old ? PyLong_AsLongLong(old) : 0) + 1);
      ok = sum && !PyErr_Occurred() && PyDict_SetItem(calls, key, sum) == 0;
      Py_XDECREF(sum);
    }
  }
  Py_XDECREF(key);
  Py_DECREF(calls);
  return ok;
}

// The interpreter lock given up for a scope, also when it is left by an exception.
struct Unlocked {
  PyThreadState* const state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

PyObject* forward_checked(PyObject* self, const at::Tensor& x, long math) {
  const Attributes layer(self);
  const bool swiglu = math >= 0;
  if (x.dim() != 2) Py_RETURN_NONE;
  const auto type = x.scalar_type();
  if (type != at::kHalf && type != at::kBFloat16) Py_RETURN_NONE;
  const int64_t tokens = x.size(0);
  PyObject* capsule = find(layer, tokens);
  if (!capsule) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  struct Release { PyObject* o; ~Release() { Py_DECREF(o); } } release{capsule};
  const Ready* r = ready_of(capsule);
  if (!r) return nullptr;
  if (x.size(1) != (swiglu ? 2 * r->k : r->k) || x.device() != r->device || !x.is_contiguous() ||
      !unchanged(layer, s_low_id, r->low_id) || !unchanged(layer, s_high_id, r->high_id) || !tensor_core_policy(layer) ||
      !operands_unchanged(layer, *r->low, *r->high))
    Py_RETURN_NONE;
  const int dtype = type == at::kBFloat16 ? HG_DTYPE_BF16 : HG_DTYPE_F16;
  at::Tensor y;
  int status;
  {
    // Without the interpreter lock, as torch's own bindings: an allocator may wait for a thread that wants it (one whose
    // callbacks are Python functions, as of a pool that a serving engine puts to sleep), or for the device.
    const Unlocked unlocked;
    // Fresh tensors per call: under CUDA-graph capture the graph's pool owns them.
    y = at::empty({r->tokens, r->outputs}, r->output);
    const bool in_gemm = !swiglu && (r->fused == 1 || (r->fused == 2 && c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None));
    const int64_t bytes = in_gemm ? 0 : r->packed;
    // Scratch that nobody else sees: the allocator itself, for the same stream and with the same lifetime, without a tensor round it
    // (0.3 us of a call of two launches, of which the host then needs 7.3 to 7.8 us).
    c10::DataPtr workspace;
    if (bytes) {
      const c10::cuda::CUDAGuard guard(r->device);
      workspace = c10::cuda::CUDACachingAllocator::get()->allocate(size_t(bytes));
    }
    const void* in = x.const_data_ptr();
    void* out = y.mutable_data_ptr();
    void* scratch = workspace.get();
    void* stream = c10::cuda::getCurrentCUDAStream(r->device.index()).stream();
    status = swiglu ? run_linear_silu(r->handle, r->low, r->high, in, dtype, int(math), scratch, out, stream)
                    : run_linear(r->handle, r->low, r->high, in, dtype, scratch, out, stream);
  }
  if (status) return PyErr_SetString(PyExc_RuntimeError, last_error()), nullptr;
  if (!count_call(layer, tokens)) return nullptr;
  return THPVariable_Wrap(std::move(y));
}

// forward(layer, x, math): the layer on `x`, of SwiGLU of `x` when math >= 0.  None: not an ordinary call, or the first one.
PyObject* forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) return PyErr_SetString(PyExc_TypeError, "forward(layer, x, math)"), nullptr;
  if (!run_linear || !THPVariable_Check(args[1])) Py_RETURN_NONE;
  const long math = PyLong_AsLong(args[2]);
  if (math == -1 && PyErr_Occurred()) return nullptr;
  try {
    return forward_checked(args[0], THPVariable_Unpack(args[1]), math);
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* type = PyObject_GetAttrString(PyImport_AddModule("torch"), "OutOfMemoryError");
    PyErr_SetString(type ? type : PyExc_RuntimeError, e.what_without_backtrace());
    Py_XDECREF(type);
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// prepare(layer, tokens, handle, low, high, problems, y, packed, fused): the state `forward` looks up.
// `low` and `high` are addresses of the two structs that `problems` keeps alive, `y` is a tensor like the output.
PyObject* prepare(PyObject*, PyObject* args) {
  PyObject *layer, *problems, *y;
  long long tokens, packed;
  int fused;
  unsigned long long handle, low, high;
  if (!PyArg_ParseTuple(args, "OLKKKOOLi", &layer, &tokens, &handle, &low, &high, &problems, &y, &packed, &fused)) return nullptr;
  if (!THPVariable_Check(y)) return PyErr_SetString(PyExc_TypeError, "prepare: y must be a tensor"), nullptr;
  auto* r = new Ready{};
  r->problems = Py_NewRef(problems);
  PyObject* capsule = PyCapsule_New(r, kName, destroy);
  if (!capsule) return nullptr;
  if (!(r->low_id = PyObject_GetAttr(layer, s_low_id)) || !(r->high_id = PyObject_GetAttr(layer, s_high_id))) return Py_DECREF(capsule), nullptr;
  const at::Tensor& like = THPVariable_Unpack(y);
  r->handle = reinterpret_cast<void*>(uintptr_t(handle));
  r->low = reinterpret_cast<const hg_problem*>(uintptr_t(low));
  r->high = reinterpret_cast<const hg_problem*>(uintptr_t(high));
  r->tokens = tokens;
  r->outputs = like.size(1);
  r->k = r->low->k;
  r->packed = packed;
  r->fused = fused;
  r->device = like.device();
  r->output = at::TensorOptions().dtype(like.scalar_type()).device(like.device());
  return capsule;
}

// bind(hg_linear, hg_linear_silu, hg_last_error): addresses in the loaded library.
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long linear, silu, error;
  if (!PyArg_ParseTuple(args, "KKK", &linear, &silu, &error)) return nullptr;
  run_linear = reinterpret_cast<decltype(run_linear)>(uintptr_t(linear));
  run_linear_silu = reinterpret_cast<decltype(run_linear_silu)>(uintptr_t(silu));
  last_error = reinterpret_cast<decltype(last_error)>(uintptr_t(error));
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward)), METH_FASTCALL, nullptr},
    {"prepare", prepare, METH_VARARGS, nullptr},
    {"bind", bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hygemm_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__hygemm_host() {
  PyObject** names[] = {&s_ready, &s_w4, &s_sf4, &s_lo, &s_w8, &s_sf8, &s_hi, &s_low_id, &s_high_id, &s_concurrent, &s_plans, &s_calls};
  const char* text[] = {"_ready", "w4", "sf4", "lo", "w8", "sf8", "hi", "low_id", "high_id", "concurrent", "plans", "calls"};
  for (size_t i = 0; i < std::size(names); ++i)
    if (!(*names[i] = PyUnicode_InternFromString(text[i]))) return nullptr;
  return PyModule_Create(&module);
}
