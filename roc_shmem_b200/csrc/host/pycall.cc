// pycall.cc — CPython callables over the extern "C" entry points of the native libraries.
//
// ctypes builds an argument object, a conversion and a libffi call frame for every argument of every call: 1.5 to 3 us
// for the 6 to 20 integers and addresses that the entry points here take, which is as long as a kernel launch and
// shows wherever a program issues many small operations.  `Native(address, nargs, kind, pointers)` is a vectorcall object
// that converts its arguments straight to machine words and calls the function: about 0.15 us.
//
// Only integer and pointer arguments are supported, and they take what ctypes takes for them: an integer argument anything
// with __index__ (a numpy integer, a one-element tensor) but not None; an address (bit i of `pointers`) an int or None.  Every argument is passed as one 64-bit word: under the System V
// x86-64 and the AArch64 Linux calling conventions an int or pointer argument occupies one full register or stack
// slot, of which the callee reads the width it declares (the same convention libffi relies on).
// Like ctypes' CDLL, the interpreter lock is released around the call: blocking entry points wait for other threads.
// The reference has no Python layer, hence no counterpart.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cstdint>
#include <utility>

namespace {

constexpr int kMaxArgs = 24;

enum Kind { RET_STATUS = 0, RET_WORD = 1, RET_VOID = 2 };   // int, pointer / 64-bit unsigned, nothing

struct Native {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  uintptr_t addr;
  int nargs;
  int kind;
  uint32_t pointers;             // bit i: argument i is an address
};

template <size_t> using Word = uint64_t;
using Thunk = uint64_t (*)(uintptr_t, const uint64_t*);

template <size_t... I>
uint64_t invoke(uintptr_t addr, const uint64_t* a, std::index_sequence<I...>) {
  (void)a;
  return reinterpret_cast<uint64_t (*)(Word<I>...)>(addr)(a[I]...);
}
template <size_t N> uint64_t thunk(uintptr_t addr, const uint64_t* a) { return invoke(addr, a, std::make_index_sequence<N>{}); }

template <size_t... N> constexpr void fill(Thunk* t, std::index_sequence<N...>) { ((t[N] = thunk<N>), ...); }
struct Table {
  Thunk t[kMaxArgs + 1];
  constexpr Table() : t{} { fill(t, std::make_index_sequence<kMaxArgs + 1>{}); }
};
constexpr Table kThunks;

PyObject* native_call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  const Native* self = reinterpret_cast<Native*>(callable);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != self->nargs || (kwnames && PyTuple_GET_SIZE(kwnames))) {
    PyErr_Format(PyExc_TypeError, "native function takes %d positional arguments, %zd given", self->nargs, n);
    return nullptr;
  }
  uint64_t a[kMaxArgs];
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* o = args[i];
    if (PyLong_Check(o)) {
      a[i] = PyLong_AsUnsignedLongLongMask(o);       // negative integers keep their two's complement bits
    } else if (self->pointers >> i & 1) {
      if (o != Py_None) {
        PyErr_Format(PyExc_TypeError, "native function: argument %zd is a %s, not an address or None", i, Py_TYPE(o)->tp_name);
        return nullptr;
      }
      a[i] = 0;
      continue;
    } else {
      PyObject* n_obj = PyNumber_Index(o);
      if (!n_obj) return nullptr;
      a[i] = PyLong_AsUnsignedLongLongMask(n_obj);
      Py_DECREF(n_obj);
    }
    if (a[i] == (uint64_t)-1 && PyErr_Occurred()) return nullptr;
  }
  uint64_t r;
  const Thunk t = kThunks.t[n];
  Py_BEGIN_ALLOW_THREADS
  r = t(self->addr, a);
  Py_END_ALLOW_THREADS
  switch (self->kind) {
    case RET_STATUS: return PyLong_FromLong((long)(int32_t)(uint32_t)r);
    case RET_WORD: return PyLong_FromUnsignedLongLong(r);
    default: Py_RETURN_NONE;
  }
}

PyObject* native_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long addr = 0;
  int nargs = 0, kind = 0;
  unsigned int pointers = 0;
  if (!PyArg_ParseTuple(args, "KiiI", &addr, &nargs, &kind, &pointers)) return nullptr;
  if (addr == 0 || nargs < 0 || nargs > kMaxArgs || kind < RET_STATUS || kind > RET_VOID) {
    PyErr_SetString(PyExc_ValueError, "Native(address, nargs, kind, pointers): bad address, argument count or result kind");
    return nullptr;
  }
  Native* self = reinterpret_cast<Native*>(type->tp_alloc(type, 0));
  if (!self) return nullptr;
  self->vectorcall = native_call;
  self->addr = (uintptr_t)addr;
  self->nargs = nargs;
  self->kind = kind;
  self->pointers = pointers;
  return reinterpret_cast<PyObject*>(self);
}

PyMemberDef native_members[] = {
    {"__vectorcalloffset__", T_PYSSIZET, offsetof(Native, vectorcall), READONLY, nullptr},
    {nullptr, 0, 0, 0, nullptr},
};
PyType_Slot native_slots[] = {
    {Py_tp_new, reinterpret_cast<void*>(native_new)},
    {Py_tp_call, reinterpret_cast<void*>(PyVectorcall_Call)},
    {Py_tp_members, native_members},
    {Py_tp_doc, const_cast<char*>("Native(address, nargs, kind, pointers): an extern \"C\" function of integers and addresses")},
    {0, nullptr},
};
PyType_Spec native_spec = {"bshmem_pycall.Native", sizeof(Native), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL, native_slots};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "bshmem_pycall", "Direct calls of the native libraries.", -1, nullptr, nullptr,
                          nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_bshmem_pycall(void) {
  PyObject* m = PyModule_Create(&module_def);
  if (!m) return nullptr;
  PyObject* t = PyType_FromSpec(&native_spec);
  if (!t || PyModule_AddObject(m, "Native", t) < 0) {
    Py_XDECREF(t);
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
