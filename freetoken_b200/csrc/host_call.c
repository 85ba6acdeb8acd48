// The host side of a kernel launch: what stands between an op's Python face and its extern "C" launcher.
//
// A Launcher holds the address of a launcher's packed form (common.cuh, FT_PACKED) and the kinds of its arguments, and is
// called with tensors, numbers and None as the face has them.  It takes the tensors' addresses, adds the current stream,
// calls the launcher without the interpreter lock and turns a code other than 0 into the package's KernelError.  need()
// checks a tensor as every face does first.  Through ctypes a launch of twenty arguments cost 3 us for their conversion and
// as much again for the addresses, checks, stream and counter in Python; a step that carries a prompt is some sixty of them.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <limits.h>
#include <stddef.h>
#include <string.h>

typedef union {
  void* p;
  long long i;
  double f;
} Arg;

#define MOST_ARGS 48

typedef struct {
  PyObject_HEAD
  vectorcallfunc call;
  int (*packed)(const Arg*);
  int n, kernels;
  char kinds[MOST_ARGS];
  char name[64];
} Launcher;

static PyObject *tensor_type, *get_device, *get_stream, *kernel_error, *error_names;
static PyObject *s_data_ptr, *s_is_cuda, *s_dtype, *s_is_contiguous;
static long long launches;
static _Thread_local int promised_ahead;      // handed on behind the arguments (common.cuh)

static int address_of(PyObject* o, void** out) {
  if (o == Py_None) {
    *out = NULL;
    return 0;
  }
  if (PyLong_Check(o)) {
    *out = PyLong_AsVoidPtr(o);
    return PyErr_Occurred() ? -1 : 0;
  }
  if (PyObject_TypeCheck(o, (PyTypeObject*)tensor_type)) {
    PyObject* r = PyObject_CallMethodNoArgs(o, s_data_ptr);
    if (!r) return -1;
    *out = PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    return PyErr_Occurred() ? -1 : 0;
  }
  // a ctypes array (a tensor map, a list of slots): the caller's reference keeps it for the length of the call
  Py_buffer view;
  if (PyObject_GetBuffer(o, &view, PyBUF_SIMPLE)) return -1;
  *out = view.buf;
  PyBuffer_Release(&view);
  return 0;
}

static PyObject* launcher_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Launcher* l = (Launcher*)self;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != l->n || (kwnames && PyTuple_GET_SIZE(kwnames)))
    return PyErr_Format(PyExc_TypeError, "%s takes %d arguments, not %zd", l->name, l->n, n);
  Arg a[MOST_ARGS + 2];
  for (int k = 0; k < l->n; ++k) {
    PyObject* o = args[k];
    switch (l->kinds[k]) {
      case 'p':
        if (address_of(o, &a[k].p)) return NULL;
        break;
      case 'f':
        a[k].f = PyFloat_AsDouble(o);
        if (a[k].f == -1.0 && PyErr_Occurred()) return NULL;
        break;
      default:
        a[k].i = l->kinds[k] == 'q' ? (long long)PyLong_AsUnsignedLongLongMask(o) : PyLong_AsLongLong(o);
        if (a[k].i == -1 && PyErr_Occurred()) return NULL;
        if (l->kinds[k] == 'i' && (a[k].i > INT_MAX || a[k].i < INT_MIN))
          return PyErr_Format(kernel_error, "%s: argument %d does not fit 32 bits", l->name, k);
    }
  }
  // the stream is asked for each time: callers switch streams between launches
  PyObject* device = PyObject_CallNoArgs(get_device);
  if (!device) return NULL;
  PyObject* stream = PyObject_CallOneArg(get_stream, device);
  Py_DECREF(device);
  if (!stream) return NULL;
  a[l->n].p = PyLong_AsVoidPtr(stream);
  a[l->n + 1].i = promised_ahead;
  Py_DECREF(stream);
  if (PyErr_Occurred()) return NULL;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = l->packed(a);
  Py_END_ALLOW_THREADS
  launches += l->kernels;
  if (rc) {
    PyObject* key = PyLong_FromLong(rc);
    PyObject* what = key ? PyDict_GetItemWithError(error_names, key) : NULL;
    Py_XDECREF(key);
    if (PyErr_Occurred()) return NULL;
    const char* name = strncmp(l->name, "ft_", 3) ? l->name : l->name + 3;
    if (what) return PyErr_Format(kernel_error, "%s: %U", name, what);
    return PyErr_Format(kernel_error, "%s: CUDA error %d", name, rc);
  }
  Py_RETURN_NONE;
}

static PyObject* launcher_new(PyTypeObject* type, PyObject* args, PyObject* kw) {
  unsigned long long address;
  const char *kinds, *name;
  int kernels;
  if (kw && PyDict_GET_SIZE(kw)) return PyErr_Format(PyExc_TypeError, "Launcher takes no keywords");
  if (!PyArg_ParseTuple(args, "Kssi", &address, &kinds, &name, &kernels)) return NULL;
  Launcher* l = (Launcher*)type->tp_alloc(type, 0);
  if (!l) return NULL;
  l->call = launcher_call;
  l->packed = (int (*)(const Arg*))(size_t)address;
  l->kernels = kernels;
  strncpy(l->name, name, sizeof(l->name) - 1);
  for (; *kinds; ++kinds) {
    if (*kinds == ' ') continue;
    if (l->n == MOST_ARGS || !strchr("piqf", *kinds)) {
      Py_DECREF(l);
      return PyErr_Format(PyExc_ValueError, "%s: argument kinds are up to %d of p, i, q and f", name, MOST_ARGS);
    }
    l->kinds[l->n++] = *kinds;
  }
  return (PyObject*)l;
}

static PyTypeObject launcher_type = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "ft_host.Launcher",
    .tp_basicsize = sizeof(Launcher),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_vectorcall_offset = offsetof(Launcher, call),
    .tp_call = PyVectorcall_Call,
    .tp_new = launcher_new,
};

// need(tensor, name, dtype=None, contiguous=True)
static PyObject* need(PyObject* self, PyObject* const* args, Py_ssize_t n, PyObject* kwnames) {
  PyObject *t = NULL, *name = NULL, *dtype = Py_None, *contiguous = Py_True;
  if (n > 0) t = args[0];
  if (n > 1) name = args[1];
  if (n > 2) dtype = args[2];
  if (n > 3) contiguous = args[3];
  for (Py_ssize_t k = 0; kwnames && k < PyTuple_GET_SIZE(kwnames); ++k) {
    PyObject* key = PyTuple_GET_ITEM(kwnames, k);
    if (PyUnicode_CompareWithASCIIString(key, "dtype") == 0) dtype = args[n + k];
    else if (PyUnicode_CompareWithASCIIString(key, "contiguous") == 0) contiguous = args[n + k];
    else return PyErr_Format(PyExc_TypeError, "need() has no argument %U", key);
  }
  if (n < 2 || n > 4) return PyErr_Format(PyExc_TypeError, "need() takes a tensor, its name, a dtype and whether it is contiguous");
  PyObject* v = PyObject_GetAttr(t, s_is_cuda);
  if (!v) return NULL;
  Py_DECREF(v);
  if (v != Py_True) return PyErr_Format(kernel_error, "%U must be a CUDA tensor", name);
  if (dtype != Py_None) {
    v = PyObject_GetAttr(t, s_dtype);
    if (!v) return NULL;
    if (v != dtype) {
      PyErr_Format(kernel_error, "%U must be %S, is %S", name, dtype, v);
      Py_DECREF(v);
      return NULL;
    }
    Py_DECREF(v);
  }
  const int wants = PyObject_IsTrue(contiguous);
  if (wants < 0) return NULL;
  if (wants) {
    v = PyObject_CallMethodNoArgs(t, s_is_contiguous);
    if (!v) return NULL;
    Py_DECREF(v);
    if (v != Py_True) return PyErr_Format(kernel_error, "%U must be contiguous", name);
  }
  Py_RETURN_NONE;
}

static PyObject* count(PyObject* self, PyObject* unused) { return PyLong_FromLongLong(launches); }

// ahead(promise) -> what was promised before; this thread's launches from here on
static PyObject* ahead(PyObject* self, PyObject* promise) {
  const int now = PyObject_IsTrue(promise), before = promised_ahead;
  if (now < 0) return NULL;
  promised_ahead = now;
  return PyBool_FromLong(before);
}

// setup(tensor type, current device, current raw stream of a device, error type, {code: what it means})
static PyObject* setup(PyObject* self, PyObject* args) {
  PyObject* o[5];
  if (!PyArg_ParseTuple(args, "OOOOO", &o[0], &o[1], &o[2], &o[3], &o[4])) return NULL;
  PyObject** to[5] = {&tensor_type, &get_device, &get_stream, &kernel_error, &error_names};
  for (int k = 0; k < 5; ++k) {
    Py_INCREF(o[k]);
    Py_XSETREF(*to[k], o[k]);
  }
  Py_RETURN_NONE;
}

static PyMethodDef methods[] = {
    {"need", (PyCFunction)(void (*)(void))need, METH_FASTCALL | METH_KEYWORDS, "a CUDA tensor of that type, contiguous"},
    {"ahead", ahead, METH_O, "whether this thread's launches may read weights, tables and metadata ahead of their wait"},
    {"count", count, METH_NOARGS, "kernels launched so far"},
    {"setup", setup, METH_VARARGS, "what the module asks Python for"},
    {NULL, NULL, 0, NULL},
};

static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "ft_host", NULL, -1, methods};

PyMODINIT_FUNC PyInit_ft_host(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_is_cuda = PyUnicode_InternFromString("is_cuda");
  s_dtype = PyUnicode_InternFromString("dtype");
  s_is_contiguous = PyUnicode_InternFromString("is_contiguous");
  if (!s_data_ptr || !s_is_cuda || !s_dtype || !s_is_contiguous || PyType_Ready(&launcher_type) < 0) return NULL;
  PyObject* m = PyModule_Create(&module);
  if (!m) return NULL;
  if (PyModule_AddObjectRef(m, "Launcher", (PyObject*)&launcher_type) < 0) {
    Py_DECREF(m);
    return NULL;
  }
  return m;
}
