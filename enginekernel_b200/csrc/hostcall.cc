// Calls a kernel launcher's C entry point from Python: arguments converted in one loop, the interpreter lock released,
// the entry point's int returned.  ctypes spends 2.8 us of the host on a call of 26 arguments, this 0.5; a short prompt's
// layer makes four to eight of them while the device waits.
//
// One call serves every signature: the System V ABI of x86-64 hands integers and pointers over in six registers and then
// eight-byte stack places, in their order, and up to eight floats in registers of their own, whatever their order among
// each other.  A function with fewer parameters leaves the rest of both alone.  Other signatures (and other machines) are
// refused by bind() and stay with ctypes.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>

namespace {

constexpr int kRegs = 6, kStack = 42, kInts = kRegs + kStack, kFloats = 8;

#define W6(a) a[0], a[1], a[2], a[3], a[4], a[5]
#define W8(a) a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]
#define T6 uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t
typedef int (*Entry)(T6, float, float, float, float, float, float, float, float, T6, T6, T6, T6, T6, T6, T6);

PyObject* data_ptr;                   // the method's name

struct Launcher {
  PyObject_HEAD
  vectorcallfunc call;
  void* entry;
  int n;
  char kinds[kInts + kFloats];      // 'p' address, tensor or None, 'i' integer, 'f' float
};

PyObject* launch(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* names) {
  Launcher* l = (Launcher*)self;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != l->n || (names && PyTuple_GET_SIZE(names))) {
    PyErr_Format(PyExc_TypeError, "this entry point takes %d arguments, not %zd", l->n, n);
    return nullptr;
  }
  uint64_t ints[kInts] = {};
  float floats[kFloats] = {};
  int ni = 0, nf = 0;
  for (int i = 0; i < l->n; ++i) {
    PyObject* a = args[i];
    if (l->kinds[i] == 'f') {
      const double v = PyFloat_AsDouble(a);
      if (v == -1.0 && PyErr_Occurred()) return nullptr;
      floats[nf++] = (float)v;
    } else if (PyLong_Check(a)) {
      ints[ni++] = (uint64_t)PyLong_AsUnsignedLongLongMask(a);
    } else if (a == Py_None && l->kinds[i] == 'p') {
      ints[ni++] = 0;
    } else if (l->kinds[i] == 'p') {            // a tensor
      PyObject* at = PyObject_CallMethodNoArgs(a, data_ptr);
      if (!at) return nullptr;
      ints[ni++] = (uint64_t)PyLong_AsUnsignedLongLongMask(at);
      Py_DECREF(at);
      if (PyErr_Occurred()) return nullptr;
    } else {
      PyErr_Format(PyExc_TypeError, "argument %d: an integer, not %.100s", i + 1, Py_TYPE(a)->tp_name);
      return nullptr;
    }
  }
  const Entry entry = (Entry)l->entry;
  const uint64_t* s = ints + kRegs;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = entry(W6(ints), W8(floats), W6(s), W6((s + 6)), W6((s + 12)), W6((s + 18)), W6((s + 24)), W6((s + 30)), W6((s + 36)));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

PyTypeObject launcher_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// bind(address, kinds): a callable, or None for a signature this cannot call
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long address;
  const char* kinds;
  Py_ssize_t n;
  if (!PyArg_ParseTuple(args, "Ks#", &address, &kinds, &n)) return nullptr;
#if defined(__x86_64__) && !defined(_WIN32)
  int floats = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (kinds[i] != 'p' && kinds[i] != 'i' && kinds[i] != 'f') Py_RETURN_NONE;
    floats += kinds[i] == 'f';
  }
  if (floats > kFloats || n - floats > kInts) Py_RETURN_NONE;
  Launcher* l = PyObject_New(Launcher, &launcher_type);
  if (!l) return nullptr;
  l->call = launch;
  l->entry = (void*)(uintptr_t)address;
  l->n = (int)n;
  for (Py_ssize_t i = 0; i < n; ++i) l->kinds[i] = kinds[i];
  return (PyObject*)l;
#else
  Py_RETURN_NONE;
#endif
}

PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "ek_hostcall", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_ek_hostcall() {
  launcher_type.tp_name = "ek_hostcall.Launcher";
  launcher_type.tp_basicsize = sizeof(Launcher);
  launcher_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  launcher_type.tp_vectorcall_offset = offsetof(Launcher, call);
  launcher_type.tp_call = PyVectorcall_Call;
  launcher_type.tp_dealloc = [](PyObject* o) { PyObject_Free(o); };
  data_ptr = PyUnicode_InternFromString("data_ptr");
  if (!data_ptr || PyType_Ready(&launcher_type) < 0) return nullptr;
  return PyModule_Create(&module);
}
