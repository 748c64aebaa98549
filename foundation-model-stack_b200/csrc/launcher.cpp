// Calls from Python into the kernels' C entries.
//
// A step launched call by call makes some five to a hundred launches of 10 to 30 arguments each, most of them tensors' addresses.
// With every address checked and fetched in Python and every argument converted by ctypes a launch took 6 to 10 us of the host,
// more than many of the kernels take.  Here an entry takes the tensors themselves, makes the same checks (on a CUDA device,
// contiguous) and the call.  Measured (with one allocation instead of two for the splits' scratch): an attention layer's decode
// step, four launches, 59 -> 38 us; a latent one's, eight, 111 -> 76; a delta rule layer's prompt and four steps 410 -> 331.
//
// The arguments go by the platform's C calling convention, in which integers and pointers on one side and floats on the other
// are counted separately: the first of each in registers, further integers in eight-byte places on the stack, in order.  So one
// call with all integers in order and all floats in order reaches an entry whose parameters mix them, as long as the
// floats fit their eight registers (checked when an entry is made; the kernels' entries have six at most).
#include <Python.h>

#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <cstring>
#include <exception>

namespace {

#if defined(__x86_64__)
#define REGISTERS(a) a[0], a[1], a[2], a[3], a[4], a[5]
#define REGISTER_TYPES u64, u64, u64, u64, u64, u64
constexpr int IN_REGISTERS = 6;
#elif defined(__aarch64__) && defined(__linux__)
#define REGISTERS(a) a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]
#define REGISTER_TYPES u64, u64, u64, u64, u64, u64, u64, u64
constexpr int IN_REGISTERS = 8;
#else
#error "the calling convention of this platform is not described here"
#endif

typedef uint64_t u64;
constexpr int ON_STACK = 40, MOST = IN_REGISTERS + ON_STACK, FLOATS = 8;
#define EIGHT(a, i) a[i], a[i + 1], a[i + 2], a[i + 3], a[i + 4], a[i + 5], a[i + 6], a[i + 7]
#define EIGHT_TYPES u64, u64, u64, u64, u64, u64, u64, u64
typedef int (*entry_fn)(REGISTER_TYPES, float, float, float, float, float, float, float, float, EIGHT_TYPES, EIGHT_TYPES, EIGHT_TYPES,
                        EIGHT_TYPES, EIGHT_TYPES);

struct Entry {
  PyObject_HEAD vectorcallfunc call;
  entry_fn fn;
  PyObject* error;  // raised for a tensor that a kernel cannot take
  int n;            // parameters
  char kind[MOST + FLOATS];
};

// The address of a tensor's data, or 0 with an exception set
bool address(const Entry* self, PyObject* arg, u64* out) {
  try {
    const at::Tensor& t = THPVariable_Unpack(arg);
    if (!t.is_cuda()) {
      PyErr_SetString(self->error, "a tensor on the CPU reached a CUDA kernel; this library has no CPU path");
      return false;
    }
    if (!t.is_contiguous()) {
      PyErr_SetString(self->error, "a non-contiguous tensor reached a CUDA kernel");
      return false;
    }
    *out = reinterpret_cast<u64>(t.data_ptr());
    return true;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return false;
  }
}

PyObject* entry_call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  const Entry* self = reinterpret_cast<const Entry*>(callable);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != self->n || (kwnames && PyTuple_GET_SIZE(kwnames))) return PyErr_Format(PyExc_TypeError, "this entry takes %d arguments, not %zd", self->n, n);
  u64 whole[MOST] = {};
  float real[FLOATS] = {};
  int w = 0, r = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* a = args[i];
    const char kind = self->kind[i];
    if (kind == 'f') {
      const double x = PyFloat_AsDouble(a);
      if (x == -1.0 && PyErr_Occurred()) return nullptr;
      real[r++] = static_cast<float>(x);
    } else if (PyLong_Check(a)) {
      const u64 x = PyLong_AsUnsignedLongLongMask(a);
      if (x == ~0ull && PyErr_Occurred()) return nullptr;
      whole[w++] = x;
    } else if (kind == 'p' && a == Py_None) {
      whole[w++] = 0;
    } else if (kind == 'p' && THPVariable_Check(a)) {
      if (!address(self, a, &whole[w++])) return nullptr;
    } else if (kind == 'i' && PyIndex_Check(a)) {  // numpy's whole numbers and the like, as ctypes takes them
      PyObject* index = PyNumber_Index(a);
      if (!index) return nullptr;
      const u64 x = PyLong_AsUnsignedLongLongMask(index);
      Py_DECREF(index);
      if (x == ~0ull && PyErr_Occurred()) return nullptr;
      whole[w++] = x;
    } else {
      return PyErr_Format(PyExc_TypeError, "argument %zd: '%s' where a %s is taken", i + 1, Py_TYPE(a)->tp_name,
                          kind == 'p' ? "tensor, an address or None" : "whole number");
    }
  }
  const u64* s = whole + IN_REGISTERS;
  int rc;
  Py_BEGIN_ALLOW_THREADS  // a launch waits where the device's queue is full
  rc = self->fn(REGISTERS(whole), real[0], real[1], real[2], real[3], real[4], real[5], real[6], real[7], EIGHT(s, 0), EIGHT(s, 8),
                EIGHT(s, 16), EIGHT(s, 24), EIGHT(s, 32));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

void entry_dealloc(PyObject* o) {
  Py_XDECREF(reinterpret_cast<Entry*>(o)->error);
  Py_TYPE(o)->tp_free(o);
}

PyTypeObject entry_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// entry(address, kinds, error): kinds has a letter a parameter, p a pointer, i a whole number, f a float
PyObject* make_entry(PyObject*, PyObject* args) {
  unsigned long long fn;
  const char* kinds;
  PyObject* error;
  if (!PyArg_ParseTuple(args, "KsO", &fn, &kinds, &error)) return nullptr;
  int whole = 0, real = 0;
  const size_t n = strlen(kinds);
  for (size_t i = 0; i < n; ++i) {
    if (kinds[i] == 'f') ++real;
    else if (kinds[i] == 'p' || kinds[i] == 'i') ++whole;
    else return PyErr_Format(PyExc_ValueError, "kinds of parameters are p, i and f, not %c", kinds[i]);
  }
  if (whole > MOST || real > FLOATS) return PyErr_Format(PyExc_ValueError, "at most %d whole numbers and %d floats", MOST, FLOATS);
  Entry* e = PyObject_New(Entry, &entry_type);
  if (!e) return nullptr;
  e->call = entry_call;
  e->fn = reinterpret_cast<entry_fn>(static_cast<uintptr_t>(fn));
  Py_INCREF(error);
  e->error = error;
  e->n = static_cast<int>(n);
  memcpy(e->kind, kinds, n);
  return reinterpret_cast<PyObject*>(e);
}

PyMethodDef methods[] = {{"entry", make_entry, METH_VARARGS, "entry(address, kinds, error): a C entry as a callable"}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "launcher", nullptr, -1, methods};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_launcher() {
  entry_type.tp_name = "launcher.Entry";
  entry_type.tp_basicsize = sizeof(Entry);
  entry_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  entry_type.tp_vectorcall_offset = offsetof(Entry, call);
  entry_type.tp_call = PyVectorcall_Call;
  entry_type.tp_dealloc = entry_dealloc;
  if (PyType_Ready(&entry_type) < 0) return nullptr;
  return PyModule_Create(&module);
}
