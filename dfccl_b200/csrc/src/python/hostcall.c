/* Calls of C entry points whose arguments are all integers, addresses or None, from Python: what ctypes does with its argument
 * types costs 0.5 to 1 us a call, and a submission, a stream-ordered collective or a small product is a call every few
 * microseconds.  A function is named by its address; the interpreter's lock is released around it, as ctypes does. */
#define Py_LIMITED_API 0x030a0000
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

#define MAX_ARGS 14
typedef int (*Entry)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t);

/* call(address, arguments...) -> the int it returns.  (Both calling conventions this builds for, x86-64 System V and AArch64,
 * pass integer arguments alike whatever their width, and leave surplus ones to the caller.)  Anything that is not an integer or
 * None is a TypeError before the call is made. */
static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  uint64_t v[MAX_ARGS + 1] = {0};
  if (n < 1 || n > MAX_ARGS + 1) { PyErr_SetString(PyExc_TypeError, "an address and at most 14 arguments"); return NULL; }
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (args[i] == Py_None) continue;
    v[i] = PyLong_AsUnsignedLongLongMask(args[i]);
    if (v[i] == (uint64_t)-1 && PyErr_Occurred()) return NULL;
  }
  if (v[0] == 0) { PyErr_SetString(PyExc_TypeError, "no address"); return NULL; }
  int r;
  Py_BEGIN_ALLOW_THREADS
  r = ((Entry)(uintptr_t)v[0])(v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12], v[13], v[14]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(r);
}

static PyMethodDef methods[] = {{"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, "call(address, arguments...) -> int"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "dfccl_hostcall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit_dfccl_hostcall(void) { return PyModule_Create(&module); }
