/* call(address, *args): a kernel library's launcher, called without ctypes, whose conversion of thirty arguments takes the host as
 * long as the launch itself.
 *
 * Launchers take integers of 32 and 64 bits, pointers and floats.  On x86-64 (System V) every integer and pointer has a place of
 * 64 bits, in six registers and then on the stack in their order, and the first eight floats have registers of their own wherever
 * they stand, so one function type serves all of them.  Elsewhere build.py calls them with ctypes.
 *
 * An argument: an int (its low 64 bits), a bool, a float, None (null), or an object whose `value` is one of these (ctypes). */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#if !defined(__x86_64__) || defined(_WIN32)
#error "the places of a call's arguments are those of the System V ABI for x86-64"
#endif

#define INTS 58
#define FLOATS 8
typedef long long L;
typedef int (*launcher)(L, L, L, L, L, L, float, float, float, float, float, float, float, float, L, L, L, L, L, L, L, L, L, L, L, L, L, L,
                        L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L, L);

/* one argument into its place; 0, or -1 with an exception */
static int put(PyObject *o, L *ints, int *n, float *floats, int *f) {
  if (PyFloat_Check(o)) {
    if (*f == FLOATS) {
      PyErr_SetString(PyExc_TypeError, "a launcher takes at most 8 floats");
      return -1;
    }
    floats[(*f)++] = (float)PyFloat_AS_DOUBLE(o);
    return 0;
  }
  if (*n == INTS) {
    PyErr_SetString(PyExc_TypeError, "a launcher takes at most 58 integers and pointers");
    return -1;
  }
  if (o == Py_None) {
    ints[(*n)++] = 0;
    return 0;
  }
  if (PyLong_Check(o)) {
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
    if (v == (unsigned long long)-1 && PyErr_Occurred()) return -1;
    ints[(*n)++] = (L)v;
    return 0;
  }
  PyObject *value = PyObject_GetAttrString(o, "value");
  if (value == NULL) {
    if (PyErr_ExceptionMatches(PyExc_AttributeError))
      PyErr_Format(PyExc_TypeError, "a launcher takes integers, floats and None, not %.100s", Py_TYPE(o)->tp_name);
    return -1;
  }
  int rc = -1;
  if (value == Py_None || PyLong_Check(value) || PyFloat_Check(value)) rc = put(value, ints, n, floats, f);
  else PyErr_Format(PyExc_TypeError, "a launcher takes integers, floats and None, not %.100s", Py_TYPE(o)->tp_name);
  Py_DECREF(value);
  return rc;
}

static PyObject *call(PyObject *self, PyObject *const *args, Py_ssize_t count) {
  L i[INTS] = {0};
  float f[FLOATS] = {0};
  int n = 0, m = 0;
  if (count < 1) {
    PyErr_SetString(PyExc_TypeError, "call(address, *args)");
    return NULL;
  }
  void *address = PyLong_AsVoidPtr(args[0]);
  if (address == NULL) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "a null address");
    return NULL;
  }
  for (Py_ssize_t k = 1; k < count; ++k)
    if (put(args[k], i, &n, f, &m) != 0) return NULL;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = ((launcher)address)(i[0], i[1], i[2], i[3], i[4], i[5], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], i[6], i[7], i[8], i[9],
                           i[10], i[11], i[12], i[13], i[14], i[15], i[16], i[17], i[18], i[19], i[20], i[21], i[22], i[23], i[24],
                           i[25], i[26], i[27], i[28], i[29], i[30], i[31], i[32], i[33], i[34], i[35], i[36], i[37], i[38], i[39],
                           i[40], i[41], i[42], i[43], i[44], i[45], i[46], i[47], i[48], i[49], i[50], i[51], i[52], i[53], i[54],
                           i[55], i[56], i[57]);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {{"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, "call(address, *args) -> int"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ll_launch", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__ll_launch(void) { return PyModule_Create(&module); }
