/* A call into libb200parallm.so from Python without ctypes' conversions: a small call spends 3 of its 7 us in them.
 *
 * bind(address, signature, fallback) -> callable.  signature: one letter per argument, "p" pointer (None is NULL), "i" integer of up to 64 bits, "f" float.
 * The System V x86-64 calling convention passes integers and floats in register files of their own, and what overflows the six integer
 * registers in order on the stack, so a call with all integers first and all floats (eight at most) behind them puts every argument where the
 * callee, whose prototype mixes them, looks for it; arguments it does not have are ignored.  Every function bound here returns an int.
 * Arguments of other types (ctypes objects, byref) or another number of them go to `fallback`, the ctypes function. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <stdint.h>
#include <stddef.h>
#include <string.h>

#if !defined(__x86_64__) || !defined(__linux__)
#error "the argument order relies on the System V x86-64 calling convention"
#endif

#define MAX_INT 32
#define MAX_FLOAT 8
#define MAX_ARGS (MAX_INT + MAX_FLOAT)

typedef struct {
  PyObject_HEAD
  vectorcallfunc call;
  void* fn;
  PyObject* fallback;
  Py_ssize_t n;
  char sig[MAX_ARGS];
} Bound;

typedef uint64_t u;
typedef int (*Target)(u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, u, float, float, float, float, float,
                      float, float, float);

static PyObject* bound_call(PyObject* o, PyObject* const* args, size_t nargsf, PyObject* kw) {
  Bound* b = (Bound*)o;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  u a[MAX_INT] = {0};
  float f[MAX_FLOAT] = {0};
  int ni = 0, nf = 0, rc;
  if (n != b->n || (kw && PyTuple_GET_SIZE(kw))) return PyObject_Vectorcall(b->fallback, args, nargsf, kw);
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* x = args[i];
    if (b->sig[i] == 'f') {
      if (!PyFloat_Check(x)) return PyObject_Vectorcall(b->fallback, args, nargsf, kw);
      f[nf++] = (float)PyFloat_AS_DOUBLE(x);
    } else if (PyLong_Check(x)) {
      a[ni] = PyLong_AsUnsignedLongLongMask(x);                 /* (ctypes wraps larger numbers the same way) */
      if (a[ni++] == (u)-1 && PyErr_Occurred()) return NULL;
    } else if (b->sig[i] == 'p' && x == Py_None) {
      a[ni++] = 0;
    } else {
      return PyObject_Vectorcall(b->fallback, args, nargsf, kw);
    }
  }
  Py_BEGIN_ALLOW_THREADS
  rc = ((Target)b->fn)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16], a[17], a[18],
                       a[19], a[20], a[21], a[22], a[23], a[24], a[25], a[26], a[27], a[28], a[29], a[30], a[31], f[0], f[1], f[2], f[3], f[4],
                       f[5], f[6], f[7]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static void bound_dealloc(PyObject* o) {
  Py_XDECREF(((Bound*)o)->fallback);
  Py_TYPE(o)->tp_free(o);
}

static PyTypeObject BoundType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "mlx_parallm_b200._fastcall.Bound",
    .tp_basicsize = sizeof(Bound),
    .tp_dealloc = bound_dealloc,
    .tp_call = PyVectorcall_Call,
    .tp_vectorcall_offset = offsetof(Bound, call),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
};

static PyObject* bind(PyObject* self, PyObject* args) {
  unsigned long long address;
  const char* sig;
  Py_ssize_t n, ints = 0, floats = 0;
  PyObject* fallback;
  (void)self;
  if (!PyArg_ParseTuple(args, "Ks#O", &address, &sig, &n, &fallback)) return NULL;
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (!strchr("pif", sig[i])) return PyErr_Format(PyExc_ValueError, "unknown argument type in signature %s", sig);
    if (sig[i] == 'f') ++floats; else ++ints;
  }
  if (ints > MAX_INT || floats > MAX_FLOAT) return PyErr_Format(PyExc_ValueError, "too many arguments: %s", sig);
  Bound* b = PyObject_New(Bound, &BoundType);
  if (!b) return NULL;
  b->call = bound_call;
  b->fn = (void*)(uintptr_t)address;
  b->fallback = Py_NewRef(fallback);
  b->n = n;
  memcpy(b->sig, sig, (size_t)n);
  return (PyObject*)b;
}

static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "bind(address, signature, fallback) -> callable"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void) {
  if (PyType_Ready(&BoundType) < 0) return NULL;
  return PyModule_Create(&module);
}
