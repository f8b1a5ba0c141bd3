// Calls of this package's hot entry points from Python, outside ctypes: a small all-reduce spent 1.7 of its 5.3 us on describing two tensors
// and converting seven arguments. Knows neither torch nor a library: tensors are asked for what the wrappers ask them for, entry points come in as
// addresses. The interpreter's lock is released while they run, as ctypes does. Without this module the wrappers go through ctypes.
#define PY_SSIZE_T_CLEAN
#define Py_LIMITED_API 0x030a0000
#include <Python.h>
#include <stdint.h>

static PyObject *sDataPtr, *sNumel, *sIsContiguous, *sDtype, *sIsCuda, *sDevice, *sIndex, *sCudaStream, *sValue;

typedef struct {
  uint64_t ptr, count;
  int type, cuda;   // type -1: no buffer
} Buffer;

// A result as an unsigned word; takes the reference. -1: an exception is set.
static int wordOf(PyObject* v, uint64_t* out) {
  if (!v) return -1;
  if (!PyLong_Check(v)) {
    PyErr_Format(PyExc_TypeError, "an integer is required, not %R", (PyObject*)Py_TYPE(v));
    Py_DECREF(v);
    return -1;
  }
  *out = PyLong_AsUnsignedLongLongMask(v);
  Py_DECREF(v);
  return PyErr_Occurred() ? -1 : 0;
}

// Handles: an integer, None, or what carries one as `value` (ctypes).
static int handleOf(PyObject* v, uint64_t* out) {
  *out = 0;
  if (v == Py_None) return 0;
  if (PyLong_Check(v)) {
    Py_INCREF(v);
    return wordOf(v, out);
  }
  PyObject* inner = PyObject_GetAttr(v, sValue);
  if (inner == Py_None) {
    Py_DECREF(inner);
    return 0;
  }
  return wordOf(inner, out);
}

// 0, -1 with an exception, or 1: not a tensor, which the wrapper describes itself.
static int describe(PyObject* buf, PyObject* types, Buffer* b) {
  b->ptr = b->count = 0;
  b->type = -1;
  b->cuda = 0;
  if (buf == Py_None) return 0;
  PyObject* contiguous = PyObject_CallMethodObjArgs(buf, sIsContiguous, NULL);
  if (!contiguous) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError) || PyObject_HasAttr(buf, sDataPtr)) return -1;
    PyErr_Clear();
    return 1;
  }
  const int ok = PyObject_IsTrue(contiguous);
  Py_DECREF(contiguous);
  if (ok < 0) return -1;
  if (!ok) {
    PyErr_SetString(PyExc_ValueError, "tensors must be contiguous");
    return -1;
  }
  if (wordOf(PyObject_CallMethodObjArgs(buf, sDataPtr, NULL), &b->ptr) || wordOf(PyObject_CallMethodObjArgs(buf, sNumel, NULL), &b->count)) return -1;
  PyObject* dtype = PyObject_GetAttr(buf, sDtype);
  if (!dtype) return -1;
  PyObject* code = PyDict_GetItemWithError(types, dtype);   // borrowed
  if (!code) {
    if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, dtype);
    Py_DECREF(dtype);
    return -1;
  }
  Py_DECREF(dtype);
  b->type = (int)PyLong_AsLong(code);
  PyObject* cuda = PyObject_GetAttr(buf, sIsCuda);
  if (!cuda) return -1;
  b->cuda = PyObject_IsTrue(cuda);
  Py_DECREF(cuda);
  return b->cuda < 0 || PyErr_Occurred() ? -1 : 0;
}

// The given stream (an integer or an object with its handle), or the current one of the buffer's device.
static int streamOf(PyObject* stream, PyObject* buf, const Buffer* b, PyObject* current, uint64_t* out) {
  *out = 0;
  if (stream != Py_None) {
    if (PyLong_Check(stream)) {
      Py_INCREF(stream);
      return wordOf(stream, out);
    }
    PyObject* handle = PyObject_GetAttr(stream, sCudaStream);
    const int got = handle ? handleOf(handle, out) : -1;
    Py_XDECREF(handle);
    return got;
  }
  if (!b->cuda) return 0;
  PyObject* device = PyObject_GetAttr(buf, sDevice);
  if (!device) return -1;
  PyObject* index = PyObject_GetAttr(device, sIndex);
  Py_DECREF(device);
  if (!index) return -1;
  PyObject* handle = PyObject_CallFunctionObjArgs(current, index, NULL);
  Py_DECREF(index);
  return wordOf(handle, out);
}

// collective(address, types, current, send, recv, lead, divisor, extra, comm, stream): address(send, recv, count, type, [extra,] comm, stream)
// with the count (over divisor) and type of recv if lead has bit 0, else of send, on the stream given or the current one of recv's device if lead
// has bit 1, else of send's. Bit 2: the entry point takes `extra` (an operator, a root). Without the bit it does if an extra is given. types: codes by
// dtype; current: handle of a device's current stream. NotImplemented for what ctypes has to see: buffers that are no tensors, an `extra` or a divisor
// that is no int (ctypes takes whatever stands for one, and refuses the rest).
static PyObject* collective(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  (void)self;
  if (n != 10) return PyErr_Format(PyExc_TypeError, "collective takes 10 arguments, not %zd", n);
  uint64_t fn, comm, stream, extra = 0, divisor;
  Buffer b[2];
  for (int i = 0; i < 2; ++i) {
    const int got = describe(a[3 + i], a[1], &b[i]);
    if (got < 0) return NULL;
    if (got) {
      Py_INCREF(Py_NotImplemented);
      return Py_NotImplemented;
    }
  }
  const long bits = PyLong_AsLong(a[5]);
  const int lead = bits & 1, at = bits >> 1 & 1, takesExtra = bits & 4 || a[7] != Py_None;
  if (((takesExtra && !PyLong_Check(a[7])) || !PyLong_Check(a[6])) && !PyErr_Occurred()) {
    Py_INCREF(Py_NotImplemented);
    return Py_NotImplemented;
  }
  if (PyErr_Occurred() || handleOf(a[0], &fn) || handleOf(a[6], &divisor) || handleOf(a[7], &extra) || handleOf(a[8], &comm)) return NULL;
  if (streamOf(a[9], a[3 + at], &b[at], a[2], &stream)) return NULL;
  if (!fn || !divisor || b[lead].type < 0) {
    PyErr_SetString(PyExc_TypeError, "collective: no entry point or no buffer");
    return NULL;
  }
  const size_t count = (size_t)(b[lead].count / divisor);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  if (!takesExtra)
    rc = ((int (*)(void*, void*, size_t, int, void*, void*))(uintptr_t)fn)((void*)(uintptr_t)b[0].ptr, (void*)(uintptr_t)b[1].ptr, count, b[lead].type,
                                                                           (void*)(uintptr_t)comm, (void*)(uintptr_t)stream);
  else
    rc = ((int (*)(void*, void*, size_t, int, int, void*, void*))(uintptr_t)fn)((void*)(uintptr_t)b[0].ptr, (void*)(uintptr_t)b[1].ptr, count, b[lead].type,
                                                                                (int)extra, (void*)(uintptr_t)comm, (void*)(uintptr_t)stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// invoke(address, ...): an entry point whose parameters are integers and pointers. None is a null pointer wherever it stands: an integer of the
// caller's comes here only as an int. A tuple (a shape) stands for four of them: the number of
// dimensions and, for two or three dimensions, their sizes (zeros behind the last). System V x86-64: words are what such
// parameters travel as, and words beyond the callee's last parameter are not looked at.
enum { kWords = 32 };
static PyObject* invoke(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  (void)self;
  uint64_t fn, w[kWords] = {0};
  if (n < 1 || handleOf(a[0], &fn)) return PyErr_Occurred() ? NULL : PyErr_Format(PyExc_TypeError, "invoke takes an address");
  if (!fn) return PyErr_Format(PyExc_TypeError, "invoke: no entry point");
  int used = 0;
  for (Py_ssize_t i = 1; i < n; ++i) {
    const int tuple = PyTuple_Check(a[i]);
    if (used + (tuple ? 4 : 1) > kWords) return PyErr_Format(PyExc_TypeError, "invoke: more than %d words", (int)kWords);
    if (!tuple) {
      if (handleOf(a[i], &w[used++])) return NULL;
      continue;
    }
    const Py_ssize_t dims = PyTuple_Size(a[i]);
    w[used] = (uint64_t)dims;
    for (Py_ssize_t d = 0; (dims == 2 || dims == 3) && d < dims; ++d)
      if (handleOf(PyTuple_GetItem(a[i], d), &w[used + 1 + d])) return NULL;
    used += 4;
  }
#define W(i) w[i], w[i + 1], w[i + 2], w[i + 3], w[i + 4], w[i + 5], w[i + 6], w[i + 7]
#define P8 uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t
  int rc;
  Py_BEGIN_ALLOW_THREADS
  if (used <= 8) rc = ((int (*)(P8))(uintptr_t)fn)(W(0));
  else if (used <= 16) rc = ((int (*)(P8, P8))(uintptr_t)fn)(W(0), W(8));
  else rc = ((int (*)(P8, P8, P8, P8))(uintptr_t)fn)(W(0), W(8), W(16), W(24));
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {
    {"collective", (PyCFunction)(void (*)(void))collective, METH_FASTCALL, "rc of a collective on two tensors, or NotImplemented"},
    {"invoke", (PyCFunction)(void (*)(void))invoke, METH_FASTCALL, "rc of an entry point with integer and pointer parameters"},
    {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void) {
#if !defined(__x86_64__)
  PyErr_SetString(PyExc_ImportError, "words travel as System V x86-64 passes them");
  return NULL;
#endif
  const struct { PyObject** at; const char* name; } names[] = {{&sDataPtr, "data_ptr"}, {&sNumel, "numel"}, {&sIsContiguous, "is_contiguous"}, {&sDtype, "dtype"},
      {&sIsCuda, "is_cuda"}, {&sDevice, "device"}, {&sIndex, "index"}, {&sCudaStream, "cuda_stream"}, {&sValue, "value"}};
  for (size_t i = 0; i < sizeof(names) / sizeof(names[0]); ++i)
    if (!(*names[i].at = PyUnicode_InternFromString(names[i].name))) return NULL;
  return PyModule_Create(&module);
}
