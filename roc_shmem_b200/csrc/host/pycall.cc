// pycall.cc — CPython callables over the extern "C" entry points of the native libraries.
//
// ctypes builds an argument object, a conversion and a libffi call frame for every argument of every call: 1.5 to 3 us
// for the 6 to 20 integers and addresses that the entry points here take, which is as long as a kernel launch and
// shows wherever a program issues many small operations.  `Native(address, nargs, kind, pointers)` is a vectorcall object
// that converts its arguments straight to machine words and calls the function: about 0.15 us.
//
// `Mover` is the same for the messages of a context, put(dest, src, pe, nbi=...): it takes the tensors themselves and reads their addresses
// and sizes through DLPack's C exchange table.  What the attribute look-ups of a Python method and its frame add to that was three
// quarters of a small message's 0.6 us: a window of 64 non-blocking puts of 64 bytes took 41 us, so 25.  Calls of any other form go to the
// method of the context's type; so do all while that is another one than it was (tracing puts a method with ranges there).
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

// ---- messages of a context -------------------------------------------------------------------------------------
// DLPack (public standard, ABI version 1): a tensor as its producer describes it, and the table of its C functions.
struct DlTensor {
  void* data;
  struct { int32_t type, id; } device;
  int32_t ndim;
  struct { uint8_t code, bits; uint16_t lanes; } dtype;
  int64_t* shape;
  int64_t* strides;
  uint64_t byte_offset;
};
struct DlExchange {
  struct { uint32_t major, minor; } version;
  void* older;
  void* allocate;
  void* owned_from;
  void* to;
  int (*describe)(void* object, DlTensor* out);      // borrows; may be null
  void* work_stream;
};
constexpr int kDlCuda = 2;

struct Mover {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  uintptr_t addr;                // int (handle, context, dest, src, bytes, pe, nbi)
  uint64_t handle;
  int context, device, local;    // local: which argument is this PE's own buffer and says how much is moved, 0 = dest, 1 = src
  int (*describe)(void*, DlTensor*);
  PyObject* tensor;              // the type whose instances `describe` takes
  PyObject *owner, *name;        // the context, and the method of its type for every other call
  PyObject* plain;               // that method as this one stands for it
  PyObject* check;               // raises for a status
};
PyObject* g_nbi = nullptr;       // the interned keyword

bool move_at_once(const Mover* m, PyObject* const* args, Py_ssize_t n, PyObject* kwnames, uint64_t* a) {
  if (n != 3 || Py_TYPE(args[0]) != (PyTypeObject*)m->tensor || Py_TYPE(args[1]) != (PyTypeObject*)m->tensor || !PyLong_CheckExact(args[2])) return false;
  a[6] = 0;
  if (kwnames && PyTuple_GET_SIZE(kwnames)) {
    if (PyTuple_GET_SIZE(kwnames) != 1 || PyTuple_GET_ITEM(kwnames, 0) != g_nbi) return false;
    if (args[3] == Py_True) a[6] = 1;
    else if (args[3] != Py_False) return false;
  }
  DlTensor t[2];
  for (int i = 0; i < 2; ++i)
    if (m->describe(args[i], &t[i]) != 0) {
      PyErr_Clear();
      return false;
    }
  const DlTensor& l = t[m->local];
  if (!t[0].data || !t[1].data) return false;        // tensors that a transformation made up have none
  if (l.device.type != kDlCuda || l.device.id != m->device || (l.dtype.bits & 7)) return false;
  uint64_t bytes = (uint64_t)(l.dtype.bits >> 3) * l.dtype.lanes;
  for (int i = 0; i < l.ndim; ++i) bytes *= (uint64_t)l.shape[i];
  const long pe = PyLong_AsLong(args[2]);
  if (pe == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  if (bytes == 0 || pe != (int)pe) return false;
  a[0] = m->handle;
  a[1] = (uint64_t)(int64_t)m->context;
  a[2] = (uint64_t)t[0].data + t[0].byte_offset;
  a[3] = (uint64_t)t[1].data + t[1].byte_offset;
  a[4] = bytes;
  a[5] = (uint64_t)(int64_t)pe;
  return true;
}
PyObject* mover_call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  const Mover* m = reinterpret_cast<Mover*>(callable);
  uint64_t a[7];
  PyTypeObject* type = Py_TYPE(m->owner);
  PyObject* method = _PyType_Lookup(type, m->name);            // borrowed
  if (!method) return PyErr_Format(PyExc_AttributeError, "%U", m->name);
  if (method != m->plain || !move_at_once(m, args, PyVectorcall_NARGS(nargsf), kwnames, a)) {
    const descrgetfunc bind = Py_TYPE(method)->tp_descr_get;
    Py_INCREF(method);
    PyObject* bound = bind ? bind(method, m->owner, reinterpret_cast<PyObject*>(type)) : Py_NewRef(method);
    Py_DECREF(method);
    if (!bound) return nullptr;
    PyObject* result = PyObject_Vectorcall(bound, args, nargsf, kwnames);
    Py_DECREF(bound);
    return result;
  }
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = (int32_t)(uint32_t)thunk<7>(m->addr, a);
  Py_END_ALLOW_THREADS
  if (status == 0) Py_RETURN_NONE;
  return PyObject_CallFunction(m->check, "i", status);
}
PyObject* mover_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long addr = 0, handle = 0;
  int context = 0, device = 0, local = 0;
  PyObject *tensor, *capsule, *owner, *name, *plain, *check;
  if (!PyArg_ParseTuple(args, "KKiiiOOOUOO", &addr, &handle, &context, &device, &local, &tensor, &capsule, &owner, &name, &plain, &check)) return nullptr;
  const auto* x = static_cast<const DlExchange*>(PyCapsule_GetPointer(capsule, "dlpack_exchange_api"));
  if (!x) return nullptr;
  if (!addr || !PyType_Check(tensor) || (local != 0 && local != 1) || x->version.major != 1 || !x->describe) {
    PyErr_SetString(PyExc_ValueError, "Mover: bad address, tensor type or operand, or an exchange table of another version");
    return nullptr;
  }
  Mover* m = reinterpret_cast<Mover*>(type->tp_alloc(type, 0));
  if (!m) return nullptr;
  m->vectorcall = mover_call;
  m->addr = (uintptr_t)addr;
  m->handle = handle;
  m->context = context;
  m->device = device;
  m->local = local;
  m->describe = x->describe;
  m->tensor = Py_NewRef(tensor);
  m->owner = Py_NewRef(owner);
  m->name = Py_NewRef(name);
  PyUnicode_InternInPlace(&m->name);
  m->plain = Py_NewRef(plain);
  m->check = Py_NewRef(check);
  return reinterpret_cast<PyObject*>(m);
}
int mover_traverse(PyObject* o, visitproc visit, void* arg) {
  Mover* m = reinterpret_cast<Mover*>(o);
  Py_VISIT(Py_TYPE(o));
  Py_VISIT(m->tensor);
  Py_VISIT(m->owner);
  Py_VISIT(m->plain);
  Py_VISIT(m->check);
  return 0;
}
int mover_clear(PyObject* o) {
  Mover* m = reinterpret_cast<Mover*>(o);
  Py_CLEAR(m->tensor);
  Py_CLEAR(m->owner);
  Py_CLEAR(m->name);
  Py_CLEAR(m->plain);
  Py_CLEAR(m->check);
  return 0;
}
void mover_dealloc(PyObject* o) {
  PyTypeObject* type = Py_TYPE(o);
  PyObject_GC_UnTrack(o);
  mover_clear(o);
  type->tp_free(o);
  Py_DECREF(type);
}
PyMemberDef mover_members[] = {
    {"__vectorcalloffset__", T_PYSSIZET, offsetof(Mover, vectorcall), READONLY, nullptr},
    {"context", T_INT, offsetof(Mover, context), 0, nullptr},
    {nullptr, 0, 0, 0, nullptr},
};
PyType_Slot mover_slots[] = {
    {Py_tp_new, reinterpret_cast<void*>(mover_new)},
    {Py_tp_call, reinterpret_cast<void*>(PyVectorcall_Call)},
    {Py_tp_traverse, reinterpret_cast<void*>(mover_traverse)},
    {Py_tp_clear, reinterpret_cast<void*>(mover_clear)},
    {Py_tp_dealloc, reinterpret_cast<void*>(mover_dealloc)},
    {Py_tp_members, mover_members},
    {Py_tp_doc, const_cast<char*>("Mover(address, handle, context, device, local, tensor type, exchange table, owner, name, plain method, "
                                  "status check): put or get of a context, called as its method of that name is")},
    {0, nullptr},
};
PyType_Spec mover_spec = {"bshmem_pycall.Mover", sizeof(Mover), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_HAVE_GC, mover_slots};

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
  g_nbi = PyUnicode_InternFromString("nbi");
  t = PyType_FromSpec(&mover_spec);
  if (!g_nbi || !t || PyModule_AddObject(m, "Mover", t) < 0) {
    Py_XDECREF(t);
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
