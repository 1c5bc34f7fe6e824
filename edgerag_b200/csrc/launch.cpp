// The way from Python to the extern "C" entry points of the kernels' libraries, in place of ctypes: tensors are passed as they are,
// and the checks that every entry point makes of a tensor (device, element type, layout) run here.
//
// A call of an entry point with 24 arguments costs 2.2 us in ctypes' conversions alone, before which every tensor is asked for its
// pointer and checked in Python; a decode layer of four launches took 59 us of host time, of nine (latent attention) 111.  From here 33
// and 82, most of them the driver's launches.
//
// An entry point takes pointers, integers and floats.  Both calling conventions that CUDA hosts use here (System V x86-64, AAPCS64) give
// integers and floats registers of their own and the stack to the integers that are left, in order, 8 bytes each.  So one function type with
// room for every entry point's integers (as 64 bits) and floats passes any mixture of them; what an entry point does not take is ignored.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstddef>
#include <cstdint>

#ifndef Py_T_LONG                   // (its name before Python 3.12)
#include <structmember.h>
#define Py_T_LONG T_LONG
#endif

#if !defined(__linux__) || !(defined(__x86_64__) || defined(__aarch64__))
#error "written for the calling conventions of x86-64 and aarch64 Linux"
#endif

namespace {

constexpr int kMaxInts = 36, kMaxFloats = 8, kMaxArgs = kMaxInts + kMaxFloats;

using Word = int64_t;
using Entry = int (*)(Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word,
                      Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, Word, float, float, float,
                      float, float, float, float, float);

PyObject* g_counts = nullptr;       // {"own": launches of this package's kernels, "library": the library's}
PyObject* g_error = nullptr;        // KernelError
PyObject* g_need = nullptr;         // the check in Python, which words the complaint
PyObject *g_own = nullptr, *g_library = nullptr;

struct Launcher {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  Entry entry;
  const char* (*last_error)();
  long own;                         // kernels of this package that a call launches
  int n;
  char kinds[kMaxArgs];             // 'p' pointer, 'i' integer, 'f' float
};

// Converts the arguments and calls; false with an exception set where one does not fit.
bool run(Launcher* self, PyObject* const* args, Py_ssize_t n, int* rc) {
  if (n != self->n) {
    PyErr_Format(PyExc_TypeError, "an entry point takes %d arguments, %zd given", self->n, n);
    return false;
  }
  Word w[kMaxInts] = {};
  float f[kMaxFloats] = {};
  int ni = 0, nf = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* a = args[i];
    if (self->kinds[i] == 'f') {
      const double v = PyFloat_AsDouble(a);
      if (v == -1.0 && PyErr_Occurred()) return false;
      f[nf++] = (float)v;
    } else if (self->kinds[i] == 'p' && a == Py_None) {
      w[ni++] = 0;
    } else if (self->kinds[i] == 'p' && THPVariable_Check(a)) {
      try {
        w[ni++] = (Word)(uintptr_t)THPVariable_Unpack(a).data_ptr();
      } catch (python_error& e) {                              // (a tensor class of Python's own)
        e.restore();
        return false;
      } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return false;
      }
    } else if (PyLong_Check(a)) {
      w[ni++] = (Word)PyLong_AsUnsignedLongLongMask(a);
    } else {
      PyErr_Format(PyExc_TypeError, "argument %zd of an entry point: %s", i + 1, Py_TYPE(a)->tp_name);
      return false;
    }
  }
  if (PyErr_Occurred()) return false;
  Py_BEGIN_ALLOW_THREADS
  *rc = self->entry(w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], w[9], w[10], w[11], w[12], w[13], w[14], w[15], w[16], w[17], w[18],
                    w[19], w[20], w[21], w[22], w[23], w[24], w[25], w[26], w[27], w[28], w[29], w[30], w[31], w[32], w[33], w[34], w[35],
                    f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]);
  Py_END_ALLOW_THREADS
  return true;
}

// launcher(...): the entry point's result.
PyObject* launcher_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  if (kwnames && PyTuple_GET_SIZE(kwnames)) {
    PyErr_SetString(PyExc_TypeError, "an entry point takes no keywords");
    return nullptr;
  }
  int rc = 0;
  return run(reinterpret_cast<Launcher*>(self), args, PyVectorcall_NARGS(nargsf), &rc) ? PyLong_FromLong(rc) : nullptr;
}

PyTypeObject launcher_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// launcher(address, address of its library's erb_last_error, kinds, kernels that a call launches)
PyObject* make_launcher(PyObject*, PyObject* args) {
  unsigned long long entry, error;
  const char* kinds;
  Py_ssize_t n;
  long own;
  if (!PyArg_ParseTuple(args, "KKs#l", &entry, &error, &kinds, &n, &own)) return nullptr;
  int ni = 0, nf = 0;
  for (Py_ssize_t i = 0; i < n; ++i) (kinds[i] == 'f' ? nf : ni)++;
  if (ni > kMaxInts || nf > kMaxFloats) {
    PyErr_Format(PyExc_ValueError, "an entry point of %d integers and %d floats (at most %d and %d)", ni, nf, kMaxInts, kMaxFloats);
    return nullptr;
  }
  Launcher* self = PyObject_New(Launcher, &launcher_type);
  if (!self) return nullptr;
  self->vectorcall = launcher_call;
  self->entry = reinterpret_cast<Entry>(entry);
  self->last_error = reinterpret_cast<const char* (*)()>(error);
  self->own = own;
  self->n = (int)n;
  for (Py_ssize_t i = 0; i < n; ++i) self->kinds[i] = kinds[i];
  return reinterpret_cast<PyObject*>(self);
}

bool count(PyObject* key, long n) {
  PyObject* old = PyDict_GetItemWithError(g_counts, key);
  if (!old) return false;
  PyObject* now = PyLong_FromLong(PyLong_AsLong(old) + n);
  const bool ok = now && PyDict_SetItem(g_counts, key, now) == 0;
  Py_XDECREF(now);
  return ok;
}

// call(launcher, ...): counts the launch; a result other than 0 raises KernelError with the library's words.
PyObject* checked_call(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n < 1 || !Py_IS_TYPE(args[0], &launcher_type)) {
    PyErr_SetString(PyExc_TypeError, "call: the first argument is an entry point");
    return nullptr;
  }
  Launcher* fn = reinterpret_cast<Launcher*>(args[0]);
  int rc = 0;
  if (!run(fn, args + 1, n - 1, &rc)) return nullptr;
  if (!count(fn->own ? g_own : g_library, fn->own ? fn->own : 1)) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, "launch counts");
    return nullptr;
  }
  if (rc) {
    PyErr_SetString(g_error, fn->last_error());
    return nullptr;
  }
  Py_RETURN_NONE;
}

// need(tensor, name, dtype=None, contiguous=True): nothing where the tensor is as it has to be; everything else is the Python check's.
PyObject* need(PyObject*, PyObject* const* args, Py_ssize_t n, PyObject* kwnames) {
  PyObject *dtype = n > 2 ? args[2] : Py_None, *contiguous = n > 3 ? args[3] : Py_True;
  const Py_ssize_t n_kw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  bool known = n >= 2 && n <= 4;
  for (Py_ssize_t i = 0; i < n_kw; ++i) {
    PyObject* key = PyTuple_GET_ITEM(kwnames, i);
    if (PyUnicode_CompareWithASCIIString(key, "dtype") == 0) dtype = args[n + i];
    else if (PyUnicode_CompareWithASCIIString(key, "contiguous") == 0) contiguous = args[n + i];
    else known = false;
  }
  if (known && args[0] == Py_None) Py_RETURN_NONE;
  if (known && THPVariable_Check(args[0]) && (contiguous == Py_True || contiguous == Py_False) && (dtype == Py_None || THPDtype_Check(dtype))) {
    const at::Tensor& t = THPVariable_Unpack(args[0]);
    try {
      if (t.is_cuda() && (dtype == Py_None || t.scalar_type() == reinterpret_cast<THPDtype*>(dtype)->scalar_type) &&
          (contiguous == Py_False || t.is_contiguous()))
        Py_RETURN_NONE;
    } catch (const std::exception&) {                          // (layouts and tensor classes that do not say: asked there, they raise)
    }
  }
  return PyObject_Vectorcall(g_need, args, (size_t)n, kwnames);
}

// bind(counts, KernelError, the check in Python)
PyObject* bind(PyObject*, PyObject* args) {
  PyObject *counts, *error, *check;
  if (!PyArg_ParseTuple(args, "O!OO", &PyDict_Type, &counts, &error, &check)) return nullptr;
  Py_XSETREF(g_counts, Py_NewRef(counts));
  Py_XSETREF(g_error, Py_NewRef(error));
  Py_XSETREF(g_need, Py_NewRef(check));
  Py_RETURN_NONE;
}

PyMemberDef launcher_members[] = {{"_erb_own", Py_T_LONG, offsetof(Launcher, own), 0, nullptr}, {nullptr, 0, 0, 0, nullptr}};

PyMethodDef methods[] = {
    {"launcher", make_launcher, METH_VARARGS, nullptr},
    {"bind", bind, METH_VARARGS, nullptr},
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(checked_call)), METH_FASTCALL, nullptr},
    {"need", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(need)), METH_FASTCALL | METH_KEYWORDS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

// The module is made in two phases: it then belongs to whoever loads it, and takes no name in sys.modules.
int start(PyObject*) {
  if (g_own) return 0;              // (loaded before)
  launcher_type.tp_name = "edgerag_b200.launcher";
  launcher_type.tp_basicsize = sizeof(Launcher);
  launcher_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  launcher_type.tp_vectorcall_offset = offsetof(Launcher, vectorcall);
  launcher_type.tp_call = PyVectorcall_Call;
  launcher_type.tp_members = launcher_members;
  launcher_type.tp_dealloc = [](PyObject* self) { PyObject_Free(self); };
  if (PyType_Ready(&launcher_type) < 0) return -1;
  g_library = PyUnicode_InternFromString("library");
  if (!g_library || !(g_own = PyUnicode_InternFromString("own"))) return -1;
  return 0;
}

PyModuleDef_Slot slots[] = {{Py_mod_exec, reinterpret_cast<void*>(start)}, {0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "edgerag_b200._launch", nullptr, 0, methods, slots, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__launch() { return PyModuleDef_Init(&module); }
