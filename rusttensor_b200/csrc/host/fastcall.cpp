// The calls of the Python front end that a program makes many times a step - applying an op, reading a gradient, letting go of a tensor -
// and those of a trainer's pipelined steps, as a CPython extension over the engine's C API.
//
// A small eager step is bound by the host: of 165 us for an MLP of three layers, most went into ctypes, which converts every
// argument by way of Python objects (4 us an op, 2.5 a gradient, 1.2 a tensor released).  Here a call is a C call with arguments taken
// from the tensors' own fields.  The functions are given by address, so that one extension serves every library that exports the API.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cstdint>

namespace {

using OpFn = int (*)(const char*, const int64_t*, int, const int64_t*, int, const double*, int, int64_t*);
using FreeFn = int (*)(int64_t);
using HasGradFn = int (*)(int64_t, int*);
using GradFn = int (*)(int64_t, int64_t*);

struct Calls {
  PyObject_HEAD
  OpFn op;
  FreeFn release;
  HasGradFn has_grad;
  GradFn grad;
};
struct TensorBase {
  PyObject_HEAD
  PyObject* engine;
  Calls* calls;
  long long handle;
};
extern PyTypeObject CallsType, TensorType;
PyObject* s_calls;  // "_calls"
PyObject* s_raise;  // "_raise"

// The engine's message as the front end's exception.
PyObject* fail(PyObject* engine, int rc) {
  PyObject* code = PyLong_FromLong(rc);
  if (!code) return nullptr;
  PyObject* r = PyObject_CallMethodObjArgs(engine, s_raise, code, nullptr);
  Py_DECREF(code);
  if (r) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, "engine call failed");
  }
  return nullptr;
}

PyObject* make_tensor(PyTypeObject* type, PyObject* engine, Calls* calls, int64_t handle) {
  TensorBase* t = reinterpret_cast<TensorBase*>(type->tp_alloc(type, 0));
  if (!t) {
    calls->release(handle);
    return nullptr;
  }
  Py_INCREF(engine);
  Py_INCREF(calls);
  t->engine = engine;
  t->calls = calls;
  t->handle = handle;
  return reinterpret_cast<PyObject*>(t);
}

// ---- tensors ----
int tensor_init(PyObject* self, PyObject* args, PyObject* kwargs) {
  static const char* names[] = {"engine", "handle", nullptr};
  PyObject* engine;
  long long handle;
  if (!PyArg_ParseTupleAndKeywords(args, kwargs, "OL", const_cast<char**>(names), &engine, &handle)) return -1;
  PyObject* calls = PyObject_GetAttr(engine, s_calls);
  if (!calls) return -1;
  if (!PyObject_TypeCheck(calls, &CallsType)) {
    Py_DECREF(calls);
    PyErr_SetString(PyExc_TypeError, "not an engine");
    return -1;
  }
  TensorBase* t = reinterpret_cast<TensorBase*>(self);
  if (t->calls) {
    Py_DECREF(calls);
    PyErr_SetString(PyExc_RuntimeError, "a tensor is initialised once");
    return -1;
  }
  Py_INCREF(engine);
  t->engine = engine;
  t->calls = reinterpret_cast<Calls*>(calls);
  t->handle = handle;
  return 0;
}
int tensor_traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<TensorBase*>(self)->engine);
  Py_VISIT(reinterpret_cast<PyObject*>(reinterpret_cast<TensorBase*>(self)->calls));
  return 0;
}
int tensor_clear(PyObject*) { return 0; }  // engines do not refer to their tensors
void tensor_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  TensorBase* t = reinterpret_cast<TensorBase*>(self);
  if (t->calls) {
    const FreeFn release = t->calls->release;
    const int64_t handle = t->handle;
    Py_BEGIN_ALLOW_THREADS
    release(handle);
    Py_END_ALLOW_THREADS
  }
  Py_XDECREF(reinterpret_cast<PyObject*>(t->calls));
  Py_XDECREF(t->engine);
  Py_TYPE(self)->tp_free(self);
}
PyObject* tensor_grad(PyObject* self, void*) {
  TensorBase* t = reinterpret_cast<TensorBase*>(self);
  if (!t->calls) {
    PyErr_SetString(PyExc_RuntimeError, "the tensor is not initialised");
    return nullptr;
  }
  int has = 0, rc;
  int64_t out = 0;
  Py_BEGIN_ALLOW_THREADS
  rc = t->calls->has_grad(t->handle, &has);
  if (rc == 0 && has) rc = t->calls->grad(t->handle, &out);
  Py_END_ALLOW_THREADS
  if (rc != 0) return fail(t->engine, rc);
  if (!has) Py_RETURN_NONE;
  return make_tensor(Py_TYPE(self), t->engine, t->calls, out);
}
PyMemberDef tensor_members[] = {
    {"engine", T_OBJECT_EX, offsetof(TensorBase, engine), READONLY, nullptr},
    {"handle", T_LONGLONG, offsetof(TensorBase, handle), READONLY, nullptr},
    {nullptr, 0, 0, 0, nullptr},
};
PyGetSetDef tensor_getset[] = {
    {"grad", tensor_grad, nullptr, "The gradient as a tensor of its own, or None.", nullptr},
    {nullptr, nullptr, nullptr, nullptr, nullptr},
};
PyTypeObject TensorType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- calls ----
int calls_init(PyObject* self, PyObject* args, PyObject*) {
  unsigned long long op, release, has_grad, grad;
  if (!PyArg_ParseTuple(args, "KKKK", &op, &release, &has_grad, &grad)) return -1;
  Calls* c = reinterpret_cast<Calls*>(self);
  c->op = reinterpret_cast<OpFn>(op);
  c->release = reinterpret_cast<FreeFn>(release);
  c->has_grad = reinterpret_cast<HasGradFn>(has_grad);
  c->grad = reinterpret_cast<GradFn>(grad);
  if (c->op && c->release && c->has_grad && c->grad) return 0;
  PyErr_SetString(PyExc_ValueError, "a function's address is null");
  return -1;
}

// A few values on the stack, more on the heap.
template <class T>
struct Values {
  T few[16];
  T* v = few;
  Py_ssize_t n = 0;
  PyObject* seq = nullptr;
  bool open(PyObject* o) {
    seq = PySequence_Fast(o, "expected a sequence");
    if (!seq) return false;
    n = PySequence_Fast_GET_SIZE(seq);
    if (n > 16) {
      v = static_cast<T*>(PyMem_Malloc(sizeof(T) * (size_t)n));
      if (!v) {
        PyErr_NoMemory();
        return false;
      }
    }
    return true;
  }
  PyObject* at(Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(seq, i); }
  ~Values() {
    if (v != few) PyMem_Free(v);
    Py_XDECREF(seq);
  }
};

// op(tensor_type, engine, name, inputs, integers, floats)
PyObject* calls_op(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
  Calls* c = reinterpret_cast<Calls*>(self);
  if (nargs != 6 || !PyType_Check(args[0]) || !PyType_IsSubtype(reinterpret_cast<PyTypeObject*>(args[0]), &TensorType)) {
    PyErr_SetString(PyExc_TypeError, "op(tensor_type, engine, name, inputs, integers, floats)");
    return nullptr;
  }
  const char* name = PyUnicode_AsUTF8(args[2]);
  if (!name) return nullptr;
  Values<int64_t> in, ip;
  Values<double> fp;
  if (!in.open(args[3]) || !ip.open(args[4]) || !fp.open(args[5])) return nullptr;
  for (Py_ssize_t i = 0; i < in.n; ++i) {
    if (!PyObject_TypeCheck(in.at(i), &TensorType)) {
      PyErr_SetString(PyExc_AttributeError, "an input is not a tensor");
      return nullptr;
    }
    in.v[i] = reinterpret_cast<TensorBase*>(in.at(i))->handle;
  }
  for (Py_ssize_t i = 0; i < ip.n; ++i) {
    PyObject* n = PyNumber_Long(ip.at(i));
    if (!n) return nullptr;
    ip.v[i] = PyLong_AsLongLong(n);
    Py_DECREF(n);
    if (ip.v[i] == -1 && PyErr_Occurred()) return nullptr;
  }
  for (Py_ssize_t i = 0; i < fp.n; ++i) {
    fp.v[i] = PyFloat_AsDouble(fp.at(i));
    if (fp.v[i] == -1.0 && PyErr_Occurred()) return nullptr;
  }
  int64_t out = 0;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = c->op(name, in.v, (int)in.n, ip.v, (int)ip.n, fp.v, (int)fp.n, &out);
  Py_END_ALLOW_THREADS
  if (rc != 0) return fail(args[1], rc);
  return make_tensor(reinterpret_cast<PyTypeObject*>(args[0]), args[1], c, out);
}
PyMethodDef calls_methods[] = {
    {"op", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(calls_op)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyTypeObject CallsType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- pipelined steps of a trainer (function address, trainer's handle, ..) ----
bool addresses(PyObject* const* args, Py_ssize_t nargs, Py_ssize_t want, unsigned long long* fn, int64_t* handle) {
  if (nargs != want) {
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");
    return false;
  }
  *fn = PyLong_AsUnsignedLongLong(args[0]);
  *handle = PyLong_AsLongLong(args[1]);
  if (!*fn && !PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "a function's address is null");
  return !PyErr_Occurred();
}
// pointer(fn, handle, index) -> (status, address)
PyObject* module_pointer(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  unsigned long long fn;
  int64_t handle;
  if (!addresses(args, nargs, 3, &fn, &handle)) return nullptr;
  const long index = PyLong_AsLong(args[2]);
  if (index == -1 && PyErr_Occurred()) return nullptr;
  float* out = nullptr;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = reinterpret_cast<int (*)(int64_t, int, float**)>(fn)(handle, (int)index, &out);
  Py_END_ALLOW_THREADS
  return Py_BuildValue("iK", rc, (unsigned long long)(uintptr_t)out);
}
// step(fn, handle) -> (status, loss of the previous step or None)
PyObject* module_step(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  unsigned long long fn;
  int64_t handle;
  if (!addresses(args, nargs, 2, &fn, &handle)) return nullptr;
  float loss = 0.f;
  int has = 0, rc;
  Py_BEGIN_ALLOW_THREADS
  rc = reinterpret_cast<int (*)(int64_t, float*, int*)>(fn)(handle, &loss, &has);
  Py_END_ALLOW_THREADS
  return has ? Py_BuildValue("id", rc, (double)loss) : Py_BuildValue("iO", rc, Py_None);
}
PyMethodDef module_methods[] = {
    {"pointer", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(module_pointer)), METH_FASTCALL, nullptr},
    {"step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(module_step)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall() {
  s_calls = PyUnicode_InternFromString("_calls");
  s_raise = PyUnicode_InternFromString("_raise");
  if (!s_calls || !s_raise) return nullptr;
  TensorType.tp_name = "rusttensor_b200._fastcall.TensorBase";
  TensorType.tp_basicsize = sizeof(TensorBase);
  TensorType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC;
  TensorType.tp_new = PyType_GenericNew;
  TensorType.tp_init = tensor_init;
  TensorType.tp_dealloc = tensor_dealloc;
  TensorType.tp_traverse = tensor_traverse;
  TensorType.tp_clear = tensor_clear;
  TensorType.tp_members = tensor_members;
  TensorType.tp_getset = tensor_getset;
  CallsType.tp_name = "rusttensor_b200._fastcall.Calls";
  CallsType.tp_basicsize = sizeof(Calls);
  CallsType.tp_flags = Py_TPFLAGS_DEFAULT;
  CallsType.tp_new = PyType_GenericNew;
  CallsType.tp_init = calls_init;
  CallsType.tp_methods = calls_methods;
  if (PyType_Ready(&TensorType) < 0 || PyType_Ready(&CallsType) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module);
  if (!m) return nullptr;
  Py_INCREF(&TensorType);
  Py_INCREF(&CallsType);
  if (PyModule_AddObject(m, "TensorBase", reinterpret_cast<PyObject*>(&TensorType)) < 0 ||
      PyModule_AddObject(m, "Calls", reinterpret_cast<PyObject*>(&CallsType)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
