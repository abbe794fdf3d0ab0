// Native call path of a program: argument checks, output allocation, slot marshalling and the library call of one
// NativeProgram.run / launch, for calls whose shapes the Python binder (runtime/interface.py) has accepted before.
//
// What the Python binder decides from shapes alone - shape relations, rules, output extents, workspace size, whether the
// call is empty - is taught once per combination of shapes (learn()); everything that depends on the tensors of a call -
// type, device, rank, extents, layout, alignment, overlap - is looked at here on every call.  A call that is anything
// but plain gets NotImplemented back and takes the Python path, which raises what there is to raise.
//
// Bound by the interpreter: one projection of one token (K4096 N14336) took 31.9 us of host time through the Python binder,
// ctypes and the observation record, for a kernel of 12; here it takes the kernel's 12.3.  The two-bit program on 4096 x 4096
// 25.9 -> 6.2 us per call.  The first call of a shape goes through the Python binder, which then calls here: 30 -> 24 us for
// an int8 product, 82 us with a new artifact (84 without this file).  A program keeps sixteen plans and replaces them in
// turn: seventeen shapes by turns find none of them and pay the Python binder every time (21 us a call against 4.5; 27
// without this file).
#define PY_SSIZE_T_CLEAN
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <Python.h>

#include <cstring>
#include <memory>
#include <new>
#include <vector>

namespace {

enum Access { kIn = 0, kOut = 1, kInOut = 2 };
constexpr int kMaxRank = 3, kMaxPlans = 16;

struct View {
  int access;
  at::ScalarType type;
  int rank;
  int64_t alignment;
};

// What the Python binder found for one combination of shapes.
struct Plan {
  std::vector<int64_t> shapes;      // of every view, in declaration order
  std::vector<char> selection;      // the library's switches it was found under
  int64_t workspace;                // bytes asked for; < 0: the program has no workspace
  bool empty;
};

struct Record {                      // the latest call
  std::vector<int64_t> slots;        // without the stream
  int64_t workspace = 0;
  int status = 0;
  std::vector<char> selection;
  bool valid = false;
};

struct Binder {
  PyObject_HEAD
  int (*call)(const int64_t*);
  int slots;                         // of the entry, stream included
  int device;
  const char* selection;
  int64_t selection_bytes;
  PyObject* workspaces;              // the program's dict: stream handle -> tensor
  bool has_workspace;
  std::vector<View>* views;
  std::vector<int64_t>* constants;
  std::vector<std::shared_ptr<const Plan>>* plans;
  std::size_t next;                  // plan to replace when there are kMaxPlans
  Record* last;
};

// Gives the interpreter lock up for its lifetime, also where an exception ends it.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

PyObject* not_plain() { Py_RETURN_NOTIMPLEMENTED; }

// Tensors with a meaning beyond their storage (subclasses aside): transforms, modes, lazy views, other layouts.
bool plain_keys(const at::Tensor& t) {
  static const c10::DispatchKeySet special({
      c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::Functionalize,
      c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchVmapMode, c10::DispatchKey::Batched,
      c10::DispatchKey::VmapMode, c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
      c10::DispatchKey::FuncTorchDynamicLayerBackMode, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative,
      c10::DispatchKey::ZeroTensor, c10::DispatchKey::Fake});
  return !t.key_set().has_any(special) && t.layout() == at::kStrided && t.has_storage() &&
         !t.unsafeGetTensorImpl()->has_symbolic_sizes_strides();
}

bool modes_active() {
  return at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
         c10::impl::tls_local_dispatch_key_set().included_.has_any(c10::DispatchKeySet(
             {c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode,
              c10::DispatchKey::Functionalize, c10::DispatchKey::Python}));
}

// `explicit_outputs`: every view is supplied; `private_workspace`: such a call owns its workspace, which is not made here
PyObject* invoke(Binder* self, PyObject* arguments, bool explicit_outputs, bool private_workspace) {
  const auto& views = *self->views;
  const Py_ssize_t count = PyTuple_GET_SIZE(arguments);
  if (modes_active() || c10::cuda::current_device() != self->device) return not_plain();
  if (private_workspace && self->has_workspace) return not_plain();

  const std::size_t n = views.size();
  const at::Tensor* supplied[16];
  Py_ssize_t next = 0;
  for (std::size_t i = 0; i < n; ++i) {
    supplied[i] = nullptr;
    if (views[i].access == kOut && !explicit_outputs) continue;
    if (next == count) return not_plain();
    PyObject* object = PyTuple_GET_ITEM(arguments, next++);
    if (!THPVariable_CheckExact(object)) return not_plain();
    const at::Tensor& t = THPVariable_Unpack(object);
    if (!t.defined() || t.scalar_type() != views[i].type || t.dim() != views[i].rank || !t.is_cuda() ||
        t.get_device() != self->device || !plain_keys(t) || t.numel() == 0 || !t.is_contiguous())
      return not_plain();
    supplied[i] = &t;
  }
  if (next != count) return not_plain();

  // the plan of these shapes, found under the switches as they are
  std::shared_ptr<const Plan> plan;   // (learn() of another thread may drop it from the list)
  for (const auto& p : *self->plans) {
    const int64_t* extent = p->shapes.data();
    bool same = true;
    for (std::size_t i = 0; i < n && same; extent += views[i].rank, ++i)
      if (supplied[i]) same = std::memcmp(extent, supplied[i]->sizes().data(), views[i].rank * sizeof(int64_t)) == 0;
    if (same) {
      plan = p;
      break;
    }
  }
  if (!plan || std::memcmp(plan->selection.data(), self->selection, self->selection_bytes) != 0) return not_plain();

  const auto stream = c10::cuda::getCurrentCUDAStream(self->device);
  int64_t slots[64];
  int at_slot = 0;
  at::Tensor made[16];
  int64_t begin[16], end[16];
  if (!explicit_outputs) {
    Unlocked unlocked;   // an allocation may reach the driver and take milliseconds
    const int64_t* extent = plan->shapes.data();
    for (std::size_t i = 0; i < n; extent += views[i].rank, ++i)
      if (!supplied[i])
        made[i] = at::empty(at::IntArrayRef(extent, views[i].rank),
                            at::TensorOptions().dtype(views[i].type).device(at::kCUDA, self->device));
  }
  for (std::size_t i = 0; i < n; ++i) {
    const int rank = views[i].rank;
    const at::Tensor& t = supplied[i] ? *supplied[i] : made[i];
    const int64_t pointer = reinterpret_cast<int64_t>(t.data_ptr());
    if (pointer % views[i].alignment != 0 || !t.is_contiguous()) return not_plain();
    begin[i] = pointer;
    end[i] = pointer + t.numel() * int64_t(t.element_size());
    slots[at_slot++] = pointer;
    for (int d = 0; d < rank; ++d) slots[at_slot++] = t.size(d);
    for (int d = 0; d < rank; ++d) slots[at_slot++] = t.stride(d);
  }
  for (std::size_t i = 0; i < n; ++i)
    for (std::size_t j = i + 1; j < n; ++j)
      if ((views[i].access != kIn || views[j].access != kIn) && begin[i] < end[j] && begin[j] < end[i])
        return not_plain();

  if (!plan->empty) {
    at::Tensor workspace;   // kept over the call: another thread may replace the stream's buffer meanwhile
    for (int64_t c : *self->constants) slots[at_slot++] = c;
    int64_t workspace_bytes = 0;
    if (self->has_workspace) {
      int64_t pointer = 0;
      if (plan->workspace > 0) {
        PyObject* key = PyLong_FromUnsignedLongLong(reinterpret_cast<unsigned long long>(stream.stream()));
        if (!key) return nullptr;
        PyObject* held = PyDict_GetItemWithError(self->workspaces, key);
        Py_DECREF(key);
        if (!held) {
          if (PyErr_Occurred()) return nullptr;
          return not_plain();
        }
        if (!THPVariable_CheckExact(held)) return not_plain();
        workspace = THPVariable_Unpack(held);
        if (workspace.numel() < plan->workspace) return not_plain();
        pointer = reinterpret_cast<int64_t>(workspace.data_ptr());
        workspace_bytes = workspace.numel();
      }
      slots[at_slot++] = pointer;
      slots[at_slot++] = workspace_bytes;
    }
    slots[at_slot] = reinterpret_cast<int64_t>(stream.stream());
    if (at_slot + 1 != self->slots) return not_plain();
    std::vector<char> selection(self->selection, self->selection + self->selection_bytes);
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = self->call(slots);
    Py_END_ALLOW_THREADS
    Record& last = *self->last;
    last.slots.assign(slots, slots + at_slot);
    last.workspace = workspace_bytes;
    last.status = status;
    last.selection.swap(selection);
    last.valid = true;
    if (status != 0) return PyLong_FromLong(status);   // the caller raises
  }
  if (explicit_outputs) Py_RETURN_NONE;
  Py_ssize_t outputs = 0;
  for (std::size_t i = 0; i < n; ++i) outputs += views[i].access == kOut;
  if (outputs == 0) Py_RETURN_NONE;
  PyObject* tuple = outputs > 1 ? PyTuple_New(outputs) : nullptr;
  if (outputs > 1 && !tuple) return nullptr;
  Py_ssize_t index = 0;
  for (std::size_t i = 0; i < n; ++i) {
    if (views[i].access != kOut) continue;
    PyObject* wrapped = THPVariable_Wrap(std::move(made[i]));
    if (!tuple || !wrapped) {
      if (!wrapped) Py_XDECREF(tuple);
      return wrapped;
    }
    PyTuple_SET_ITEM(tuple, index++, wrapped);
  }
  return tuple;
}

PyObject* guarded(PyObject* self, PyObject* arguments, bool explicit_outputs, bool private_workspace) {
  if (!PyTuple_Check(arguments)) {
    PyErr_SetString(PyExc_TypeError, "a tuple of arguments is required");
    return nullptr;
  }
  try {
    return invoke(reinterpret_cast<Binder*>(self), arguments, explicit_outputs, private_workspace);
  } catch (const c10::OutOfMemoryError&) {
    return not_plain();   // the Python path allocates again and raises torch's own error
  } catch (const std::bad_alloc&) {
    return PyErr_NoMemory();
  } catch (const std::exception& error) {
    PyErr_SetString(PyExc_RuntimeError, error.what());
    return nullptr;
  }
}
PyObject* binder_run(PyObject* self, PyObject* arguments) { return guarded(self, arguments, false, false); }
PyObject* binder_start(PyObject* self, PyObject* arguments) { return guarded(self, arguments, true, false); }
PyObject* binder_launch(PyObject* self, PyObject* arguments) { return guarded(self, arguments, true, true); }

// learn(shapes of every view as a flat tuple, workspace bytes, empty, selection)
PyObject* binder_learn(PyObject* object, PyObject* arguments) {
  Binder* self = reinterpret_cast<Binder*>(object);
  PyObject* shapes;
  long long workspace;
  int empty;
  const char* selection;
  Py_ssize_t selection_bytes;
  if (!PyArg_ParseTuple(arguments, "O!Lpy#", &PyTuple_Type, &shapes, &workspace, &empty, &selection, &selection_bytes))
    return nullptr;
  std::size_t extents = 0;
  for (const View& v : *self->views) extents += std::size_t(v.rank);
  if (PyTuple_GET_SIZE(shapes) != Py_ssize_t(extents) || selection_bytes != self->selection_bytes) {
    PyErr_SetString(PyExc_ValueError, "the plan does not match the program");
    return nullptr;
  }
  try {
    auto plan = std::make_shared<Plan>();
    for (std::size_t i = 0; i < extents; ++i) {
      const long long extent = PyLong_AsLongLong(PyTuple_GET_ITEM(shapes, Py_ssize_t(i)));
      if (extent == -1 && PyErr_Occurred()) return nullptr;
      plan->shapes.push_back(extent);
    }
    plan->selection.assign(selection, selection + selection_bytes);
    plan->workspace = workspace;
    plan->empty = empty != 0;
    auto& plans = *self->plans;
    for (auto& p : plans)
      if (p->shapes == plan->shapes) {   // found again under other switches
        p = std::move(plan);
        Py_RETURN_NONE;
      }
    if (plans.size() < kMaxPlans) {
      plans.push_back(std::move(plan));
    } else {
      plans[self->next] = std::move(plan);
      self->next = (self->next + 1) % kMaxPlans;
    }
  } catch (const std::bad_alloc&) {
    return PyErr_NoMemory();
  }
  Py_RETURN_NONE;
}

// last() -> (slots without the stream, workspace bytes, status, selection) of the latest native call, or None
PyObject* binder_last(PyObject* object, PyObject*) {
  const Record& last = *reinterpret_cast<Binder*>(object)->last;
  if (!last.valid) Py_RETURN_NONE;
  PyObject* slots = PyTuple_New(Py_ssize_t(last.slots.size()));
  if (!slots) return nullptr;
  for (std::size_t i = 0; i < last.slots.size(); ++i) {
    PyObject* value = PyLong_FromLongLong(last.slots[i]);
    if (!value) {
      Py_DECREF(slots);
      return nullptr;
    }
    PyTuple_SET_ITEM(slots, Py_ssize_t(i), value);
  }
  return Py_BuildValue("(NLiy#)", slots, (long long)last.workspace, last.status, last.selection.data(),
                       Py_ssize_t(last.selection.size()));
}

PyObject* binder_forget(PyObject* object, PyObject*) {
  reinterpret_cast<Binder*>(object)->last->valid = false;
  Py_RETURN_NONE;
}

// Binder(call address, slots, device, selection address, selection bytes, workspaces | None,
//        ((access, dtype, rank, alignment), ...), constants)
PyObject* binder_new(PyTypeObject* type, PyObject* arguments, PyObject*) {
  unsigned long long call, selection;
  int slots, device;
  long long selection_bytes;
  PyObject *workspaces, *views, *constants;
  if (!PyArg_ParseTuple(arguments, "KiiKLOO!O!", &call, &slots, &device, &selection, &selection_bytes, &workspaces,
                        &PyTuple_Type, &views, &PyTuple_Type, &constants))
    return nullptr;
  if (PyTuple_GET_SIZE(views) > 16 || slots > 63 || (workspaces != Py_None && !PyDict_Check(workspaces))) {
    PyErr_SetString(PyExc_ValueError, "unsupported interface");
    return nullptr;
  }
  Binder* self = reinterpret_cast<Binder*>(type->tp_alloc(type, 0));
  if (!self) return nullptr;
  self->call = reinterpret_cast<int (*)(const int64_t*)>(call);
  self->slots = slots;
  self->device = device;
  self->selection = reinterpret_cast<const char*>(selection);
  self->selection_bytes = selection_bytes;
  self->has_workspace = workspaces != Py_None;
  Py_INCREF(workspaces);
  self->workspaces = workspaces;
  try {
    self->views = new std::vector<View>();
    self->constants = new std::vector<int64_t>();
    self->plans = new std::vector<std::shared_ptr<const Plan>>();
    self->last = new Record();
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(views); ++i) {
      View v;
      PyObject* dtype;
      long long alignment;
      if (!PyArg_ParseTuple(PyTuple_GET_ITEM(views, i), "iOiL", &v.access, &dtype, &v.rank, &alignment)) {
        Py_DECREF(self);
        return nullptr;
      }
      if (!THPDtype_Check(dtype) || v.rank < 1 || v.rank > kMaxRank || alignment < 1) {
        Py_DECREF(self);
        PyErr_SetString(PyExc_ValueError, "unsupported view");
        return nullptr;
      }
      v.type = reinterpret_cast<THPDtype*>(dtype)->scalar_type;
      v.alignment = alignment;
      self->views->push_back(v);
    }
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(constants); ++i) {
      const long long value = PyLong_AsLongLong(PyTuple_GET_ITEM(constants, i));
      if (value == -1 && PyErr_Occurred()) {
        Py_DECREF(self);
        return nullptr;
      }
      self->constants->push_back(value);
    }
  } catch (const std::bad_alloc&) {
    Py_DECREF(self);
    return PyErr_NoMemory();
  }
  return reinterpret_cast<PyObject*>(self);
}

void binder_dealloc(PyObject* object) {
  Binder* self = reinterpret_cast<Binder*>(object);
  delete self->views;
  delete self->constants;
  delete self->plans;
  delete self->last;
  Py_XDECREF(self->workspaces);
  PyTypeObject* type = Py_TYPE(object);
  type->tp_free(object);
  Py_DECREF(type);
}

PyMethodDef kMethods[] = {
    {"run", binder_run, METH_O, "run(arguments): outputs, a non-zero status, or NotImplemented"},
    {"start", binder_start, METH_O, "start(all arguments): as launch, on the stream's workspace (the first run of a shape)"},
    {"launch", binder_launch, METH_O, "launch(arguments): None, a non-zero status, or NotImplemented"},
    {"learn", binder_learn, METH_VARARGS, "learn(shapes, workspace, empty, selection)"},
    {"last", binder_last, METH_NOARGS, "the latest native call"},
    {"forget", binder_forget, METH_NOARGS, "drop the record of the latest call"},
    {nullptr, nullptr, 0, nullptr}};

PyType_Slot kSlots[] = {{Py_tp_new, reinterpret_cast<void*>(binder_new)},
                        {Py_tp_dealloc, reinterpret_cast<void*>(binder_dealloc)},
                        {Py_tp_methods, kMethods},
                        {0, nullptr}};
PyType_Spec kSpec = {"intent_b200_binder.Binder", sizeof(Binder), 0, Py_TPFLAGS_DEFAULT, kSlots};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "intent_b200_binder", nullptr, -1, nullptr, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_intent_b200_binder() {
  PyObject* module = PyModule_Create(&kModule);
  if (!module) return nullptr;
  PyObject* type = PyType_FromSpec(&kSpec);
  if (!type || PyModule_AddObject(module, "Binder", type) < 0) {
    Py_XDECREF(type);
    Py_DECREF(module);
    return nullptr;
  }
  return module;
}
