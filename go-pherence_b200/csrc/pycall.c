/* Calls into the C ABI from Python without ctypes' per-argument objects: Function(address, signature) is a callable
 * that turns its arguments into machine words and calls the address.  A small product is a launch of some 2 us of
 * host time; ctypes added 1.1 to 1.5 us to it (2.8 for a call with arrays), this adds 0.1.
 * Signature letters: p address (number, None, bytes, or an object with a number as .value), n / i numbers, f float.
 * System V x86-64: integer words go to the integer registers and the stack in their order, floats to the vector
 * registers in theirs, so one call with all words and two floats serves every signature. */
#if !defined(__x86_64__) || defined(__ILP32__) || defined(_WIN32)
#error "written for the System V x86-64 calling convention; the package does without this module elsewhere"
#endif
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#define MAX_WORDS 18
#define MAX_FLOATS 2

typedef struct {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  void* address;
  int nargs;
  char sig[MAX_WORDS + MAX_FLOATS + 1];
} Function;

typedef int (*Target)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                      uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, float, float);

/* 0 done, -1 with an exception set */
static int word_of(PyObject* o, char kind, uint64_t* out) {
  if (PyLong_Check(o)) {
    *out = PyLong_AsUnsignedLongLongMask(o);
    return *out == (uint64_t)-1 && PyErr_Occurred() ? -1 : 0;
  }
  if (kind == 'p') {
    if (o == Py_None) {
      *out = 0;
      return 0;
    }
    if (PyBytes_Check(o)) {
      *out = (uint64_t)(uintptr_t)PyBytes_AS_STRING(o);
      return 0;
    }
  } else if (PyIndex_Check(o)) {
    PyObject* v = PyNumber_Index(o);
    if (!v) return -1;
    *out = PyLong_AsUnsignedLongLongMask(v);
    Py_DECREF(v);
    return 0;
  }
  PyObject* v = PyObject_GetAttrString(o, "value"); /* the simple ctypes types */
  if (v) {
    const int none = v == Py_None, number = PyLong_Check(v);
    if (number) *out = PyLong_AsUnsignedLongLongMask(v);
    else *out = 0;
    Py_DECREF(v);
    if (number || (none && kind == 'p')) return 0;
  } else {
    PyErr_Clear();
    Py_buffer view; /* arrays, ctypes arrays among them */
    if (kind == 'p' && PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) == 0) {
      *out = (uint64_t)(uintptr_t)view.buf;
      PyBuffer_Release(&view);
      return 0;
    }
    PyErr_Clear();
  }
  PyErr_Format(PyExc_TypeError, "%s wanted", kind == 'p' ? "an address (number, None, bytes, buffer)" : "a number");
  return -1;
}

static PyObject* function_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kw) {
  Function* f = (Function*)self;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != f->nargs || (kw && PyTuple_GET_SIZE(kw))) {
    PyErr_Format(PyExc_TypeError, "%d arguments wanted", f->nargs);
    return NULL;
  }
  uint64_t w[MAX_WORDS] = {0};
  float x[MAX_FLOATS] = {0};
  int nw = 0, nx = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (f->sig[i] == 'f') {
      double d = PyFloat_AsDouble(args[i]);
      if (d == -1.0 && PyErr_Occurred()) {
        PyObject* v;
        PyErr_Clear();
        v = PyObject_GetAttrString(args[i], "value");
        if (!v) return NULL;
        d = PyFloat_AsDouble(v);
        Py_DECREF(v);
        if (d == -1.0 && PyErr_Occurred()) return NULL;
      }
      x[nx++] = (float)d;
    } else if (word_of(args[i], f->sig[i], &w[nw++]) != 0) {
      return NULL;
    }
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = ((Target)f->address)(w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], w[9], w[10], w[11], w[12], w[13], w[14], w[15], w[16],
                            w[17], x[0], x[1]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyObject* function_new(PyTypeObject* type, PyObject* args, PyObject* kw) {
  unsigned long long address;
  const char* sig;
  (void)kw;
  if (!PyArg_ParseTuple(args, "Ks", &address, &sig)) return NULL;
  int nw = 0, nx = 0;
  for (const char* c = sig; *c; ++c) {
    if (*c == 'f') ++nx;
    else if (strchr("pni", *c)) ++nw;
    else nw = MAX_WORDS + 1;
  }
  if (nw > MAX_WORDS || nx > MAX_FLOATS || !address) {
    PyErr_SetString(PyExc_ValueError, "a null address or a signature this cannot call");
    return NULL;
  }
  Function* f = (Function*)type->tp_alloc(type, 0);
  if (!f) return NULL;
  f->vectorcall = function_call;
  f->address = (void*)(uintptr_t)address;
  f->nargs = nw + nx;
  strcpy(f->sig, sig);
  return (PyObject*)f;
}

static PyTypeObject FunctionType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "goph_pycall.Function",
    .tp_basicsize = sizeof(Function),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_vectorcall_offset = offsetof(Function, vectorcall),
    .tp_call = PyVectorcall_Call,
    .tp_new = function_new,
    .tp_doc = "Function(address, signature)",
};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "goph_pycall", NULL, -1, NULL, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit_goph_pycall(void) {
  if (PyType_Ready(&FunctionType) < 0) return NULL;
  PyObject* m = PyModule_Create(&module);
  if (!m) return NULL;
  Py_INCREF(&FunctionType);
  if (PyModule_AddObject(m, "Function", (PyObject*)&FunctionType) < 0) {
    Py_DECREF(&FunctionType);
    Py_DECREF(m);
    return NULL;
  }
  return m;
}
