// The calls that a serving loop makes in every step - shape updates, tensor addresses, code generation, launch - as an extension module.
//
// Through ctypes each foreign call costs 0.3 to 1 us beside its own work, and the loops around them as much again: an RMS-norm step
// over seven tensors spent 14 us of 17 in them.  Here such a call goes straight to the C ABI (include/dvm_c.h), whose functions
// frontend.py hands over once at import.  Only the plain cases are handled: whatever is special - keyword arguments, buffers that the
// kernel owns, outputs set by the caller, the first call with a graph, errors - goes to the general method of the same purpose in
// frontend.py.  Where this module cannot be built (no C headers of Python) everything goes there (_capi.py).  Replaces the pybind11 methods of the reference's runner (src/pybind_api.cc:195-271, 1066-1116).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <climits>
#include <cstdint>
#include <cstring>
#include <type_traits>
#include <vector>

#include "dvm.h"
#include "dvm_c.h"

namespace {

constexpr int kMaxRank = 16;
constexpr Py_ssize_t kInline = 16;   // values of an int array kept for comparison

// the C ABI: addresses that frontend.py hands over, of the types that the header gives them
decltype(&dvm_int_array_update) g_int_array_update = nullptr;
decltype(&dvm_normalize) g_normalize = nullptr;
decltype(&dvm_object_shape) g_object_shape = nullptr;
decltype(&dvm_object_dtype) g_object_dtype = nullptr;
decltype(&dvm_codegen) g_codegen = nullptr;
decltype(&dvm_launch) g_launch = nullptr;

// Bytes of an element; 0 for a type this file does not know.
long long ItemSize(int type) {
  switch (type) {
    case dvm::kBool: return 1;
    case dvm::kFloat16:
    case dvm::kBFloat16: return 2;
    case dvm::kFloat32:
    case dvm::kInt32: return 4;
    case dvm::kInt64: return 8;
  }
  return 0;
}

#define DVM_NAMES(X) X(_by_handle) X(_loads) X(_stores) X(_preset) X(_load_offset) X(_relocs) X(_reloc_addr) X(_ws_addr) X(_on_device) X(_k) X(_h) \
  X(_bind_device_any) X(_codegen_any) X(_launch_any) X(_launch_result)
#define DVM_DECLARE(n) PyObject *s##n;
struct {
  DVM_NAMES(DVM_DECLARE)
} g_name;
#undef DVM_DECLARE

// A new reference that is dropped at the end of its block.
struct Ref {
  PyObject *p;
  explicit Ref(PyObject *o) : p(o) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref &) = delete;
  Ref &operator=(const Ref &) = delete;
};

// ---- IntArray: the base of IntArrayRef ------------------------------------------------------------------------
struct IntArray {
  PyObject_HEAD
  dvm_int_array *handle;
  Py_ssize_t n;            // values the native array holds (known up to kInline of them), -1: not known
  int64_t vals[kInline];
};

// tuple(map(int, shape)): into `few` where they fit, else into `many`.  A list or tuple of plain whole numbers is read in place, as nothing
// can change it meanwhile; the conversion of anything else may run code of any kind and goes through the iterator.
bool Values(PyObject *shape, std::vector<int64_t> *many, int64_t *few, const int64_t **out, Py_ssize_t *n) {
  const getiterfunc iter = Py_TYPE(shape)->tp_iter;
  const bool list = PyList_Check(shape) && iter == PyList_Type.tp_iter, tuple = PyTuple_Check(shape) && iter == PyTuple_Type.tp_iter;
  const Py_ssize_t size = list ? PyList_GET_SIZE(shape) : (tuple ? PyTuple_GET_SIZE(shape) : -1);
  bool plain = size >= 0 && size <= kInline;
  for (Py_ssize_t i = 0; plain && i < size; ++i) {
    PyObject *v = list ? PyList_GET_ITEM(shape, i) : PyTuple_GET_ITEM(shape, i);
    plain = PyLong_CheckExact(v);
    if (plain) few[i] = static_cast<int64_t>(PyLong_AsUnsignedLongLongMask(v));   // (what ctypes makes of a number beyond 64 bits)
  }
  *out = few;
  *n = size;
  if (plain) return true;
  Ref it(PyObject_GetIter(shape));
  if (it.p == nullptr) return false;
  for (;;) {
    Ref v(PyIter_Next(it.p));
    if (v.p == nullptr) break;
    Ref whole(PyNumber_Long(v.p));
    if (whole.p == nullptr) return false;
    many->push_back(static_cast<int64_t>(PyLong_AsUnsignedLongLongMask(whole.p)));
  }
  if (PyErr_Occurred()) return false;
  *out = many->data();
  *n = static_cast<Py_ssize_t>(many->size());
  return true;
}

// What the native array now holds.
void Hold(IntArray *a, const int64_t *v, Py_ssize_t n) {
  a->n = n <= kInline ? n : -1;
  if (n > 0 && n <= kInline) std::memcpy(a->vals, v, sizeof(int64_t) * static_cast<size_t>(n));
}

// _attach(handle, values): the native array, and what it holds
PyObject *IntArrayAttach(PyObject *self, PyObject *const *args, Py_ssize_t nargs) {
  IntArray *a = reinterpret_cast<IntArray *>(self);
  if (nargs != 2) {
    PyErr_SetString(PyExc_TypeError, "_attach(handle, values)");
    return nullptr;
  }
  void *h = PyLong_AsVoidPtr(args[0]);
  int64_t few[kInline];
  std::vector<int64_t> many;
  const int64_t *v = nullptr;
  Py_ssize_t n = 0;
  if (PyErr_Occurred() || !Values(args[1], &many, few, &v, &n)) return nullptr;
  a->handle = static_cast<dvm_int_array *>(h);
  Hold(a, v, n);
  Py_RETURN_NONE;
}

PyObject *IntArrayUpdate(PyObject *self, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  IntArray *a = reinterpret_cast<IntArray *>(self);
  const Py_ssize_t kw = kwnames != nullptr ? PyTuple_GET_SIZE(kwnames) : 0;
  if (nargs + kw != 1 || (kw == 1 && PyUnicode_CompareWithASCIIString(PyTuple_GET_ITEM(kwnames, 0), "shape") != 0)) {
    PyErr_SetString(PyExc_TypeError, "update() takes one argument: shape");
    return nullptr;
  }
  if (a->handle == nullptr) {
    PyErr_SetString(PyExc_RuntimeError, "update() of an int array that was not made");
    return nullptr;
  }
  int64_t few[kInline];
  std::vector<int64_t> many;
  const int64_t *v = nullptr;
  Py_ssize_t n = 0;
  if (!Values(args[0], &many, few, &v, &n)) return nullptr;
  if (n == a->n && std::memcmp(v, a->vals, sizeof(int64_t) * static_cast<size_t>(n)) == 0) Py_RETURN_NONE;   // (no call for the same values)
  g_int_array_update(a->handle, v, static_cast<size_t>(n));
  Hold(a, v, n);
  Py_RETURN_NONE;
}

PyMethodDef kIntArrayMethods[] = {
  {"_attach", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(IntArrayAttach)), METH_FASTCALL, nullptr},
  {"update", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(IntArrayUpdate)), METH_FASTCALL | METH_KEYWORDS, "update(shape): new values"},
  {nullptr, nullptr, 0, nullptr}};
PyTypeObject IntArrayType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- ExternalBuf: device memory owned by the caller, bound to a load or store -----------------------------------------
struct ExternalBuf {
  PyObject_HEAD
  unsigned long long ptr;
  long long nbytes;
  bool gone;

  void Set(PyObject *address, PyObject *size) {   // of two whole numbers; a size beyond 63 bits is the largest there is
    int beyond = 0;
    const long long v = PyLong_AsLongLongAndOverflow(size, &beyond);
    ptr = PyLong_AsUnsignedLongLongMask(address);
    nbytes = beyond == 0 ? v : (beyond > 0 ? LLONG_MAX : LLONG_MIN);
    gone = false;
  }
};
int ExternalInit(PyObject *self, PyObject *args, PyObject *) {
  ExternalBuf *b = reinterpret_cast<ExternalBuf *>(self);
  PyObject *p = nullptr, *n = nullptr;
  if (!PyArg_ParseTuple(args, "OO", &p, &n)) return -1;
  Ref ptr(PyNumber_Long(p)), nbytes(ptr.p != nullptr ? PyNumber_Long(n) : nullptr);
  if (nbytes.p == nullptr) return -1;
  b->Set(ptr.p, nbytes.p);
  return 0;
}
PyObject *ExternalFree(PyObject *self, PyObject *) {
  reinterpret_cast<ExternalBuf *>(self)->gone = true;
  Py_RETURN_NONE;
}
PyObject *ExternalPtr(PyObject *self, void *) {
  const ExternalBuf *b = reinterpret_cast<ExternalBuf *>(self);
  if (b->gone) Py_RETURN_NONE;
  return PyLong_FromUnsignedLongLong(b->ptr);
}
PyObject *ExternalBytes(PyObject *self, void *) { return PyLong_FromLongLong(reinterpret_cast<ExternalBuf *>(self)->nbytes); }
PyMethodDef kExternalMethods[] = {{"free", ExternalFree, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyGetSetDef kExternalFields[] = {{"ptr", ExternalPtr, nullptr, nullptr, nullptr},
                                 {"nbytes", ExternalBytes, nullptr, nullptr, nullptr},
                                 {nullptr, nullptr, nullptr, nullptr, nullptr}};
PyTypeObject ExternalBufType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- KernelCalls: a base of PyKernel ---------------------------------------------------------------------------------
PyObject *General(PyObject *self, PyObject *name, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  Ref method(PyObject_GetAttr(self, name));
  return method.p == nullptr ? nullptr : PyObject_Vectorcall(method.p, args, static_cast<size_t>(nargs), kwnames);
}
void *Handle(PyObject *o, PyObject *name) {   // an attribute that is an address; null (and no error set) when it is none
  Ref v(PyObject_GetAttr(o, name));
  void *p = v.p != nullptr && PyLong_Check(v.p) ? PyLong_AsVoidPtr(v.p) : nullptr;
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return nullptr;
  }
  return p;
}

// bind_device(obj, ptr, nbytes) of an object whose memory has been the caller's before
bool BindFast(PyObject *self, PyObject *const *args) {
  if (!PyLong_Check(args[1]) || !PyLong_Check(args[2])) return false;
  Ref table(PyObject_GetAttr(self, g_name.s_by_handle)), loads(PyObject_GetAttr(self, g_name.s_loads)), stores(PyObject_GetAttr(self, g_name.s_stores));
  Ref h(PyObject_GetAttr(args[0], g_name.s_h));
  if (table.p == nullptr || loads.p == nullptr || stores.p == nullptr || h.p == nullptr) return false;
  if (!PyDict_Check(table.p) || !PyList_Check(loads.p) || !PyList_Check(stores.p)) return false;
  if (PyDict_GET_SIZE(table.p) != PyList_GET_SIZE(loads.p) + PyList_GET_SIZE(stores.p)) return false;
  PyObject *rec = PyDict_GetItemWithError(table.p, h.p);   // (borrowed)
  if (rec == nullptr || !PyList_Check(rec) || PyList_GET_SIZE(rec) < 2 || Py_TYPE(PyList_GET_ITEM(rec, 1)) != &ExternalBufType) return false;
  reinterpret_cast<ExternalBuf *>(PyList_GET_ITEM(rec, 1))->Set(args[1], args[2]);
  return true;
}
PyObject *BindDevice(PyObject *self, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  if (kwnames == nullptr && nargs == 3) {
    if (BindFast(self, args)) Py_RETURN_NONE;
    PyErr_Clear();
  }
  return General(self, g_name.s_bind_device_any, args, nargs, kwnames);
}

// codegen() of a graph that has been generated before, all of its tensors in memory of the caller that is large enough.
// 1: done, 0: not such a case (nothing has been bound), -1: failed
int CodegenFast(PyObject *self) {
  Ref dev(PyObject_GetAttr(self, g_name.s_on_device)), preset(PyObject_GetAttr(self, g_name.s_preset)), offset(PyObject_GetAttr(self, g_name.s_load_offset));
  Ref loads(PyObject_GetAttr(self, g_name.s_loads)), stores(PyObject_GetAttr(self, g_name.s_stores)), relocs(PyObject_GetAttr(self, g_name.s_relocs));
  if (dev.p != Py_True || preset.p == nullptr || offset.p == nullptr || loads.p == nullptr || stores.p == nullptr || relocs.p == nullptr) return 0;
  if (!PyDict_Check(preset.p) || PyDict_GET_SIZE(preset.p) != 0 || !PyDict_Check(offset.p) || PyDict_GET_SIZE(offset.p) != 0) return 0;
  if (!PyList_Check(loads.p) || !PyList_Check(stores.p) || !PyTuple_Check(relocs.p) || PyTuple_GET_SIZE(relocs.p) < 2) return 0;
  const Py_ssize_t n_stores = PyList_GET_SIZE(stores.p), count = n_stores + PyList_GET_SIZE(loads.p);
  if (PyLong_AsSsize_t(PyTuple_GET_ITEM(relocs.p, 1)) != count) return 0;
  dvm_kernel *const k = static_cast<dvm_kernel *>(Handle(self, g_name.s_k));
  const dvm_ws_alloc_fn ws = reinterpret_cast<dvm_ws_alloc_fn>(Handle(self, g_name.s_ws_addr));
  dvm_reloc *const arr = static_cast<dvm_reloc *>(Handle(self, g_name.s_reloc_addr));
  if (k == nullptr || ws == nullptr || arr == nullptr) return 0;
  auto record = [&](Py_ssize_t i) { return i < n_stores ? PyList_GET_ITEM(stores.p, i) : PyList_GET_ITEM(loads.p, i - n_stores); };
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject *rec = record(i);
    if (!PyList_Check(rec) || PyList_GET_SIZE(rec) < (i < n_stores ? 5 : 2) || Py_TYPE(PyList_GET_ITEM(rec, 1)) != &ExternalBufType) return 0;
    if (reinterpret_cast<ExternalBuf *>(PyList_GET_ITEM(rec, 1))->gone || (i < n_stores && PyList_GET_ITEM(rec, 3) == Py_None)) return 0;
  }
  if (g_normalize(k) != 0) return 0;   // (the general method reports it)
  for (Py_ssize_t i = 0; i < count; ++i) {
    PyObject *rec = record(i);
    const ExternalBuf *b = reinterpret_cast<ExternalBuf *>(PyList_GET_ITEM(rec, 1));
    if (i < n_stores) {
      const dvm_object *h = static_cast<const dvm_object *>(Handle(PyList_GET_ITEM(rec, 0), g_name.s_h));
      int64_t dims[kMaxRank];
      const int rank = h != nullptr ? g_object_shape(h, dims, kMaxRank) : -1;
      long long nbytes = h != nullptr ? ItemSize(g_object_dtype(h)) : 0;
      if (rank < 0 || rank > kMaxRank || nbytes == 0) return 0;
      Ref shape(PyList_New(rank));
      if (shape.p == nullptr) return -1;
      for (int d = 0; d < rank; ++d) {
        if (__builtin_mul_overflow(nbytes, dims[d], &nbytes)) return 0;
        PyObject *v = PyLong_FromLongLong(dims[d]);
        if (v == nullptr) return -1;
        PyList_SET_ITEM(shape.p, d, v);
      }
      if (b->nbytes < nbytes) return 0;   // (the general method replaces the buffer)
      Py_INCREF(Py_None);
      PyList_SetItem(rec, 2, Py_None);
      PyList_SetItem(rec, 4, shape.p);
      shape.p = nullptr;
    }
    arr[i].addr = reinterpret_cast<void *>(static_cast<uintptr_t>(b->ptr));
  }
  int rc = 0;
  Py_BEGIN_ALLOW_THREADS
  rc = g_codegen(k, arr, static_cast<size_t>(count), ws, nullptr);
  Py_END_ALLOW_THREADS
  return rc == 0 ? 1 : 0;   // (a failure shows itself again in the general method, which reports it)
}
PyObject *Codegen(PyObject *self, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  if (kwnames == nullptr && (nargs == 0 || (nargs == 1 && args[0] == Py_None))) {
    const int done = CodegenFast(self);
    if (done > 0) Py_RETURN_NONE;
    if (done < 0) return nullptr;
    PyErr_Clear();
  }
  return General(self, g_name.s_codegen_any, args, nargs, kwnames);
}

PyObject *Launch(PyObject *self, PyObject *const *args, Py_ssize_t nargs, PyObject *kwnames) {
  if (kwnames == nullptr && (nargs == 0 || (nargs == 1 && (args[0] == Py_None || PyLong_CheckExact(args[0]))))) {
    dvm_kernel *const k = static_cast<dvm_kernel *>(Handle(self, g_name.s_k));
    void *stream = nargs == 1 && args[0] != Py_None ? reinterpret_cast<void *>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(args[0]))) : nullptr;
    if (k != nullptr && !PyErr_Occurred()) {
      int rc = 0;
      Py_BEGIN_ALLOW_THREADS
      rc = g_launch(k, stream);
      Py_END_ALLOW_THREADS
      if (rc == 0) Py_RETURN_NONE;
      Ref code(PyLong_FromLong(rc));
      return code.p == nullptr ? nullptr : General(self, g_name.s_launch_result, &code.p, 1, nullptr);
    }
    PyErr_Clear();
  }
  return General(self, g_name.s_launch_any, args, nargs, kwnames);
}

PyMethodDef kKernelMethods[] = {
  {"bind_device", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(BindDevice)), METH_FASTCALL | METH_KEYWORDS,
   "bind_device(obj, ptr, nbytes): use caller-owned device memory for a load or store"},
  {"codegen", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(Codegen)), METH_FASTCALL | METH_KEYWORDS,
   "codegen(pass_names=None): plan for the current shapes and bind the addresses"},
  {"launch", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(Launch)), METH_FASTCALL | METH_KEYWORDS,
   "launch(stream=None): enqueue without synchronising"},
  {nullptr, nullptr, 0, nullptr}};
PyTypeObject KernelCallsType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// setup(addresses): the C ABI, by name
PyObject *Setup(PyObject *, PyObject *table) {
  auto get = [&](const char *name, auto *to) {
    PyObject *v = PyDict_Check(table) ? PyDict_GetItemString(table, name) : nullptr;
    *to = reinterpret_cast<std::remove_pointer_t<decltype(to)>>(v != nullptr ? PyLong_AsVoidPtr(v) : nullptr);
    return *to != nullptr;
  };
  if (!get("dvm_int_array_update", &g_int_array_update) || !get("dvm_normalize", &g_normalize) || !get("dvm_object_shape", &g_object_shape) ||
      !get("dvm_object_dtype", &g_object_dtype) || !get("dvm_codegen", &g_codegen) || !get("dvm_launch", &g_launch)) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "setup() wants the addresses of the C ABI");
    return nullptr;
  }
  Py_RETURN_NONE;
}
PyMethodDef kModuleMethods[] = {{"setup", Setup, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, kModuleMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) {
#define DVM_INTERN(n) \
  if ((g_name.s##n = PyUnicode_InternFromString(#n)) == nullptr) return nullptr;
  DVM_NAMES(DVM_INTERN)
#undef DVM_INTERN
  auto type = [](PyTypeObject *t, const char *name, Py_ssize_t size, PyMethodDef *methods, bool base) {
    t->tp_name = name;
    t->tp_basicsize = size;
    t->tp_flags = Py_TPFLAGS_DEFAULT | (base ? Py_TPFLAGS_BASETYPE : 0);
    t->tp_methods = methods;
    t->tp_new = PyType_GenericNew;
  };
  type(&IntArrayType, "dvm_b200._calls.IntArray", sizeof(IntArray), kIntArrayMethods, true);
  type(&ExternalBufType, "dvm_b200._calls.ExternalBuf", sizeof(ExternalBuf), kExternalMethods, false);
  ExternalBufType.tp_init = ExternalInit;
  ExternalBufType.tp_getset = kExternalFields;
  type(&KernelCallsType, "dvm_b200._calls.KernelCalls", sizeof(PyObject), kKernelMethods, true);
  Ref m(PyModule_Create(&kModule));
  if (m.p == nullptr) return nullptr;
  PyTypeObject *const types[] = {&IntArrayType, &ExternalBufType, &KernelCallsType};
  const char *const names[] = {"IntArray", "ExternalBuf", "KernelCalls"};
  for (int i = 0; i < 3; ++i) {
    if (PyType_Ready(types[i]) < 0 || PyModule_AddObjectRef(m.p, names[i], reinterpret_cast<PyObject *>(types[i])) < 0) return nullptr;
  }
  PyObject *module = m.p;
  m.p = nullptr;
  return module;
}
