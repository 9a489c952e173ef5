// The FP8 Linear's single call without Python in between: a call with one row or a few hundred is over on the GPU in 4 - 13 us, and
// checks, allocations, argument conversion and launches take 16 us (one kernel) to 19 (two) from Python, 7 to 9 from here.
//
// A LinearCall belongs to one module and holds what its descriptor was built from.  Calling it returns the output, or None for
// any call that is not exactly of the plain kind (another type or device, a parameter that was replaced or moved, an overridden
// method, a tensor subclass, a mode that watches tensor functions, a layout that needs a copy): the caller then goes its general
// way, which also raises what there is to raise.  Where this extension is absent, every call goes there.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <utility>
#include <vector>

#include "../../include/ksana_b200.h"

namespace {

// A strong reference.
struct Ref {
  PyObject* p = nullptr;
  Ref() = default;
  explicit Ref(PyObject* o) : p(o) { Py_XINCREF(p); }
  Ref(Ref&& o) noexcept : p(o.p) { o.p = nullptr; }
  Ref(const Ref& o) : p(o.p) { Py_XINCREF(p); }
  Ref& operator=(Ref o) noexcept {
    std::swap(p, o.p);
    return *this;
  }
  ~Ref() { Py_XDECREF(p); }
};

// A name in a dict, and what it held when the descriptor was built: an object, and of a tensor its place, type and layout.
struct Entry {
  Ref space, name, object;  // object None: nothing there
  bool tensor = false;
  const void* data = nullptr;
  at::ScalarType type = at::ScalarType::Undefined;
  std::vector<int64_t> sizes, strides;
};

// An exact tensor with memory of its own, not one that a transform wraps.
bool plain_tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  const c10::DispatchKeySet wrapped({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize,
                                     c10::DispatchKey::Python, c10::DispatchKey::Batched});
  return t.defined() && t.has_storage() && t.layout() == at::kStrided && !t.key_set().has_any(wrapped) && !t.is_conj() && !t.is_neg();
}

bool holds(const Entry& e) {
  PyObject* now = PyDict_GetItem(e.space.p, e.name.p);
  if ((now == nullptr ? Py_None : now) != e.object.p) return false;
  if (!e.tensor) return true;
  const at::Tensor& t = THPVariable_Unpack(now);
  return t.has_storage() && t.data_ptr() == e.data && t.scalar_type() == e.type && t.sizes().equals(e.sizes) && t.strides().equals(e.strides);
}

typedef decltype(&ksb_linear_forward) Forward;
typedef decltype(&ksb_linear_workspace) Workspace;

struct State {
  std::vector<Entry> watch;
  Ref parameters;  // the module's _parameters
  Ref quantize;    // the class's own quantize_input
  Ref ops;         // dict of the module that holds STATS
  Ref queued;      // raises for a refused call
  ksb_linear desc{};
  at::ScalarType dtype = at::ScalarType::Undefined;
  c10::Device device{c10::kCPU};
  Forward forward = nullptr;
  Workspace workspace = nullptr;
};

struct LinearCall {
  PyObject_HEAD
  State* s;
};

PyObject *s_quantize, *s_parameters, *s_scale_input, *s_stats, *s_timing;

// The dicts watched hold the module's own, and so this object: the collector has to see through.
int traverse(PyObject* self, visitproc visit, void* arg) {
  if (const State* s = reinterpret_cast<LinearCall*>(self)->s) {
    for (const Entry& e : s->watch) {
      Py_VISIT(e.space.p);
      Py_VISIT(e.name.p);
      Py_VISIT(e.object.p);
    }
    Py_VISIT(s->parameters.p);
    Py_VISIT(s->quantize.p);
    Py_VISIT(s->ops.p);
    Py_VISIT(s->queued.p);
  }
  return 0;
}
int clear(PyObject* self) {
  State* s = reinterpret_cast<LinearCall*>(self)->s;
  reinterpret_cast<LinearCall*>(self)->s = nullptr;
  delete s;
  return 0;
}
void dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  clear(self);
  Py_TYPE(self)->tp_free(self);
}

// Raises TypeError for what it cannot watch: the module then has no LinearCall.
// LinearCall(entries of a Watch, _parameters, descriptor's address, dtype, device index, quantize_input, dict with STATS, queued,
//            address of ksb_linear_forward, address of ksb_linear_workspace)
PyObject* make(PyTypeObject* type, PyObject* args, PyObject*) {
  HANDLE_TH_ERRORS
  PyObject *entries, *parameters, *dtype, *quantize, *ops, *queued;
  unsigned long long desc, forward, workspace;
  int device;
  if (!PyArg_ParseTuple(args, "O!O!KOiOO!OKK", &PyList_Type, &entries, &PyDict_Type, &parameters, &desc, &dtype, &device, &quantize, &PyDict_Type, &ops,
                        &queued, &forward, &workspace))
    return nullptr;
  if (!THPDtype_Check(dtype)) return PyErr_Format(PyExc_TypeError, "dtype expected");
  Ref holder;
  holder.p = type->tp_alloc(type, 0);
  if (!holder.p) return nullptr;
  State* s = reinterpret_cast<LinearCall*>(holder.p)->s = new State;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(entries); ++i) {
    PyObject *space, *name, *object, *layout;
    if (!PyArg_ParseTuple(PyList_GET_ITEM(entries, i), "O!OOO", &PyDict_Type, &space, &name, &object, &layout)) return nullptr;
    Entry e;
    e.space = Ref(space);
    e.name = Ref(name);
    e.object = Ref(object);
    e.tensor = layout != Py_None;
    if (e.tensor) {
      if (!plain_tensor(object)) return PyErr_Format(PyExc_TypeError, "tensor expected");
      const at::Tensor& t = THPVariable_Unpack(object);
      e.data = t.data_ptr();
      e.type = t.scalar_type();
      e.sizes = t.sizes().vec();
      e.strides = t.strides().vec();
    }
    s->watch.push_back(std::move(e));
  }
  s->parameters = Ref(parameters);
  s->quantize = Ref(quantize);
  s->ops = Ref(ops);
  s->queued = Ref(queued);
  s->desc = *reinterpret_cast<const ksb_linear*>(desc);
  s->dtype = reinterpret_cast<THPDtype*>(dtype)->scalar_type;
  s->device = c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device));
  s->forward = reinterpret_cast<Forward>(forward);
  s->workspace = reinterpret_cast<Workspace>(workspace);
  return std::exchange(holder.p, nullptr);
  END_HANDLE_TH_ERRORS
}

// (module, input, epilogue without operands) -> output or None
PyObject* run(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3) return PyErr_Format(PyExc_TypeError, "three arguments expected");
  if (!reinterpret_cast<LinearCall*>(self)->s) Py_RETURN_NONE;
  const State& s = *reinterpret_cast<LinearCall*>(self)->s;
  PyObject *module = args[0], *input = args[1];
  if (!plain_tensor(input) || at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
      torch::jit::tracer::isTracing())
    Py_RETURN_NONE;
  const at::Tensor& x = THPVariable_Unpack(input);
  const int64_t dim = x.dim();
  if (x.scalar_type() != s.dtype || x.device() != s.device || (dim != 2 && dim != 3) || x.size(-1) != s.desc.K || x.stride(-1) != 1) Py_RETURN_NONE;
  if (!PyLong_Check(args[2])) Py_RETURN_NONE;
  const int64_t epilogue = PyLong_AsLongLong(args[2]);
  if (epilogue == -1 && PyErr_Occurred()) PyErr_Clear();
  if (epilogue != KSB_EPI_NONE && epilogue != KSB_EPI_GELU_TANH) Py_RETURN_NONE;
  // rows a constant distance apart, as a view
  int64_t M = x.size(0), ldx = x.stride(0);
  if (dim == 3) {
    const int64_t inner = x.size(1);
    if (inner != 1) {
      if (M != 1 && x.stride(0) != inner * x.stride(1)) Py_RETURN_NONE;
      ldx = x.stride(1);
    }
    M *= inner;
  }
  if (M < 1) Py_RETURN_NONE;
  if (M == 1) ldx = s.desc.K;
  // the module is the one the descriptor describes, and runs its class's own quantiser
  PyObject** dict = _PyObject_GetDictPtr(module);
  if (!dict || !*dict || PyDict_GetItem(*dict, s_parameters) != s.parameters.p || PyDict_GetItem(*dict, s_quantize)) Py_RETURN_NONE;
  PyObject* quantize = PyObject_GetAttr(reinterpret_cast<PyObject*>(Py_TYPE(module)), s_quantize);
  if (!quantize) return nullptr;
  Py_DECREF(quantize);
  if (quantize != s.quantize.p) Py_RETURN_NONE;
  for (const Entry& e : s.watch)
    if (!holds(e)) Py_RETURN_NONE;
  // references of our own: another thread may replace these while the launch has let go of the interpreter
  Ref scale_ref(PyDict_GetItem(*dict, s_scale_input)), stats_ref(PyDict_GetItem(s.ops.p, s_stats));
  if (!scale_ref.p) scale_ref = Ref(PyDict_GetItem(s.parameters.p, s_scale_input));
  PyObject *scale = scale_ref.p, *stats = stats_ref.p;
  if (!scale || !stats) Py_RETURN_NONE;
  const float* in_scale = nullptr;
  if (scale != Py_None) {
    if (!plain_tensor(scale)) Py_RETURN_NONE;
    const at::Tensor& t = THPVariable_Unpack(scale);
    if (t.device() != s.device || t.scalar_type() != at::kFloat || t.numel() != 1) Py_RETURN_NONE;
    in_scale = static_cast<const float*>(t.data_ptr());
  }
  PyObject* timing = PyObject_GetAttr(stats, s_timing);
  if (!timing) return nullptr;
  Py_DECREF(timing);
  if (timing != Py_False) Py_RETURN_NONE;

  const int64_t shape[3] = {x.size(0), dim == 3 ? x.size(1) : s.desc.N, s.desc.N};
  at::Tensor out = at::empty(at::IntArrayRef(shape, dim), at::TensorOptions().dtype(s.dtype).device(s.device));
  at::Tensor ws = at::empty({s.workspace(M, s.desc.K)}, at::TensorOptions().dtype(at::kByte).device(s.device));
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = s.forward(&s.desc, x.data_ptr(), s.dtype == at::kBFloat16 ? KSB_BF16 : KSB_FP16, M, ldx, scale != Py_None, in_scale, out.data_ptr(),
                 static_cast<int>(epilogue), nullptr, 0, nullptr, 0, ws.data_ptr(), stream);
  Py_END_ALLOW_THREADS
  PyObject* r = rc < 0 ? PyObject_CallFunction(s.queued.p, "is", rc, "ksb_linear_forward") : PyObject_CallMethod(stats, "count", "i", rc);
  if (!r) return nullptr;
  Py_DECREF(r);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyMethodDef call_methods[] = {{"run", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(run)), METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyTypeObject call_type = {PyVarObject_HEAD_INIT(nullptr, 0)};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "ksana_b200_host", nullptr, -1, nullptr, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_ksana_b200_host() {
  s_quantize = PyUnicode_InternFromString("quantize_input");
  s_parameters = PyUnicode_InternFromString("_parameters");
  s_scale_input = PyUnicode_InternFromString("scale_input");
  s_stats = PyUnicode_InternFromString("STATS");
  s_timing = PyUnicode_InternFromString("timing");
  call_type.tp_name = "ksana_b200_host.LinearCall";
  call_type.tp_basicsize = sizeof(LinearCall);
  call_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC;
  call_type.tp_traverse = traverse;
  call_type.tp_clear = clear;
  call_type.tp_new = make;
  call_type.tp_dealloc = dealloc;
  call_type.tp_methods = call_methods;
  if (PyType_Ready(&call_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module_def);
  if (!m) return nullptr;
  Py_INCREF(&call_type);
  if (PyModule_AddObject(m, "LinearCall", reinterpret_cast<PyObject*>(&call_type)) < 0) {
    Py_DECREF(&call_type);
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
