/* Calls from Python into the C ABI without ctypes' argument machinery, for the entry points a program calls per layer.
 *
 * bind(kind, address) returns a callable over the C function at that address; kind is the shape of its argument list:
 *   "oft"   (m, n, k, group_size, reconn_sz, A, ldA, B, ldB, R, ldR, C, ldC, stream)
 *   "gemm"  (m, n, k, A, ldA, B, ldB, C, ldC, stream)
 *   "ex"    (transA, transB, in_type, out_type, m, n, k, alpha, A, ldA, B, ldB, beta, C, ldC, stream)
 * Operands are tensors (anything with data_ptr()), addresses or None, streams have cuda_stream or are addresses or None.  The
 * callable returns the status code, or None without having called anything when an argument is something else: the
 * caller then takes the ctypes path, which accepts or refuses it as ever.  The GIL is released around the call.
 *
 * Host time of one call is what the smallest products take: through ctypes 2.5 us (10 arguments) to 3.2 us (14) with the
 * Python around it, here 0.6 to 0.7 (same host core); the library adds 2.9 us, of which the launch is 2.4.  200 x 328 x 136
 * half 9.9 -> 7.8 us a call in a loop, 512 x 1024 x 1024 OFT 10.4 -> 8.6, where the GPU takes over.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

typedef int (*oft_fn)(int, int, int, int, int, const void*, int, const void*, int, const void*, int, void*, int, void*);
typedef int (*gemm_fn)(int, int, int, const void*, int, const void*, int, void*, int, void*);
typedef int (*ex_fn)(char, char, int, int, int, int, int, float, const void*, int, const void*, int, float, void*, int, void*);

static PyObject *s_data_ptr, *s_cuda_stream;

/* All three return 0 when the argument is not theirs to take (no exception is left set). */
static int get_int(PyObject* o, int* out) {
  if (!PyLong_Check(o)) return 0;
  *out = (int)PyLong_AsUnsignedLongMask(o); /* wraps, as ctypes' c_int does */
  return 1;
}

static int address(PyObject* o, void** out) {
  int overflow_free;
  unsigned long long v;
  if (!PyLong_Check(o)) return 0;
  v = PyLong_AsUnsignedLongLong(o);
  overflow_free = !(v == (unsigned long long)-1 && PyErr_Occurred());
  if (!overflow_free) {
    PyErr_Clear();
    return 0;
  }
  *out = (void*)(uintptr_t)v;
  return 1;
}

static int get_ptr(PyObject* o, void** out) {
  PyObject* r;
  int ok;
  if (o == Py_None) {
    *out = NULL;
    return 1;
  }
  if (PyLong_Check(o)) return address(o, out);
  r = PyObject_CallMethodNoArgs(o, s_data_ptr);
  if (!r) {
    PyErr_Clear();
    return 0;
  }
  ok = address(r, out);
  Py_DECREF(r);
  return ok;
}

static int get_stream(PyObject* o, void** out) {
  PyObject* r;
  int ok;
  if (o == Py_None) {
    *out = NULL;
    return 1;
  }
  if (PyLong_Check(o)) return address(o, out);
  r = PyObject_GetAttr(o, s_cuda_stream);
  if (!r) {
    PyErr_Clear();
    return 0;
  }
  ok = address(r, out);
  Py_DECREF(r);
  return ok;
}

static int get_char(PyObject* o, char* out) {
  Py_ssize_t len;
  const char* s;
  if (!PyUnicode_Check(o)) return 0;
  s = PyUnicode_AsUTF8AndSize(o, &len);
  if (!s) PyErr_Clear();
  if (!s || len != 1) return 0;
  *out = s[0];
  return 1;
}

static int get_float(PyObject* o, float* out) {
  if (!PyFloat_CheckExact(o)) return 0;
  *out = (float)PyFloat_AS_DOUBLE(o);
  return 1;
}

static PyObject* call_oft(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  int d[5], ld[4], i, rc;
  void *p[4], *stream;
  const oft_fn fn = (oft_fn)PyCapsule_GetPointer(self, NULL);
  if (!fn) return NULL;
  if (n != 14) Py_RETURN_NONE;
  for (i = 0; i < 5; ++i)
    if (!get_int(a[i], &d[i])) Py_RETURN_NONE;
  for (i = 0; i < 4; ++i)
    if (!get_ptr(a[5 + 2 * i], &p[i]) || !get_int(a[6 + 2 * i], &ld[i])) Py_RETURN_NONE;
  if (!get_stream(a[13], &stream)) Py_RETURN_NONE;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(d[0], d[1], d[2], d[3], d[4], p[0], ld[0], p[1], ld[1], p[2], ld[2], p[3], ld[3], stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyObject* call_gemm(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  int d[3], ld[3], i, rc;
  void *p[3], *stream;
  const gemm_fn fn = (gemm_fn)PyCapsule_GetPointer(self, NULL);
  if (!fn) return NULL;
  if (n != 10) Py_RETURN_NONE;
  for (i = 0; i < 3; ++i)
    if (!get_int(a[i], &d[i])) Py_RETURN_NONE;
  for (i = 0; i < 3; ++i)
    if (!get_ptr(a[3 + 2 * i], &p[i]) || !get_int(a[4 + 2 * i], &ld[i])) Py_RETURN_NONE;
  if (!get_stream(a[9], &stream)) Py_RETURN_NONE;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(d[0], d[1], d[2], p[0], ld[0], p[1], ld[1], p[2], ld[2], stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyObject* call_ex(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  char t[2];
  float alpha, beta;
  int d[5], ld[3], i, rc;
  void *p[3], *stream;
  const ex_fn fn = (ex_fn)PyCapsule_GetPointer(self, NULL);
  if (!fn) return NULL;
  if (n != 16 || !get_char(a[0], &t[0]) || !get_char(a[1], &t[1])) Py_RETURN_NONE;
  for (i = 0; i < 5; ++i)
    if (!get_int(a[2 + i], &d[i])) Py_RETURN_NONE;
  if (!get_float(a[7], &alpha) || !get_float(a[12], &beta)) Py_RETURN_NONE;
  if (!get_ptr(a[8], &p[0]) || !get_int(a[9], &ld[0]) || !get_ptr(a[10], &p[1]) || !get_int(a[11], &ld[1]) || !get_ptr(a[13], &p[2]) || !get_int(a[14], &ld[2]))
    Py_RETURN_NONE;
  if (!get_stream(a[15], &stream)) Py_RETURN_NONE;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(t[0], t[1], d[0], d[1], d[2], d[3], d[4], alpha, p[0], ld[0], p[1], ld[1], beta, p[2], ld[2], stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyMethodDef def_oft = {"oft", (PyCFunction)(void (*)(void))call_oft, METH_FASTCALL, NULL};
static PyMethodDef def_gemm = {"gemm", (PyCFunction)(void (*)(void))call_gemm, METH_FASTCALL, NULL};
static PyMethodDef def_ex = {"ex", (PyCFunction)(void (*)(void))call_ex, METH_FASTCALL, NULL};

static PyObject* bind(PyObject* self, PyObject* args) {
  const char* kind;
  unsigned long long at;
  PyMethodDef* def;
  PyObject *capsule, *fn;
  (void)self;
  if (!PyArg_ParseTuple(args, "sK", &kind, &at)) return NULL;
  def = !strcmp(kind, "oft") ? &def_oft : !strcmp(kind, "gemm") ? &def_gemm : !strcmp(kind, "ex") ? &def_ex : NULL;
  if (!def || !at) {
    PyErr_SetString(PyExc_ValueError, "unknown kind or null address");
    return NULL;
  }
  capsule = PyCapsule_New((void*)(uintptr_t)at, NULL, NULL);
  if (!capsule) return NULL;
  fn = PyCFunction_New(def, capsule);
  Py_DECREF(capsule);
  return fn;
}

static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "bind(kind, address) -> callable over the C function at address"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__call(void) {
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  s_cuda_stream = PyUnicode_InternFromString("cuda_stream");
  if (!s_data_ptr || !s_cuda_stream) return NULL;
  return PyModule_Create(&module);
}
