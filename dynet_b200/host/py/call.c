/* CPython extension behind dynet_b200.capi: calls an entry point of libdyb200.so with the arguments of a node call.
 *
 * A node call on small tensors is 2 us of kernel launch; through ctypes (argument converters, byref objects, an array type
 * instantiated per call) the binding added 3 - 4 us to it.  Here the arguments are read straight from the objects, each by the kind that
 * the entry point wants at its place:
 *   i  an integer                                   v  an address: an integer, a c_void_p or None
 *   t  a tensor structure, T  one or None           x  a list or tuple of them (a C array; None or empty: NULL)
 *   s  the structure of the entry's types tuple     a  any structure, or None (node attributes)
 *   n  only None
 * Every parameter of these entry points is a pointer or an integer, i.e. one integer register or 8-byte stack slot of the
 * System V x86-64 calling convention, so one call with all slots filled serves them all.  An argument of another kind, or another
 * number of them, makes call() return NotImplemented, and the binding takes the ctypes route, which converts it or raises.  The GIL is released around the call, as ctypes does. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#define MAX_ARGS 24
#define MAX_STRUCTS 128

static PyObject *struct_type, *tensor_type, *voidp_type;
static Py_ssize_t tensor_size;

static PyObject* setup(PyObject* self, PyObject* args) {
  PyObject *s, *t, *p;
  Py_ssize_t n;
  if (!PyArg_ParseTuple(args, "OOOn", &s, &t, &p, &n)) return NULL;
  if (n > 64) { PyErr_SetString(PyExc_ValueError, "tensor structure too large"); return NULL; }
  Py_INCREF(s); Py_INCREF(t); Py_INCREF(p);
  struct_type = s; tensor_type = t; voidp_type = p; tensor_size = n;
  Py_RETURN_NONE;
}

typedef int (*entry)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                     uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t);

/* call((address, kinds, types), *arguments): kinds has one letter per parameter of the entry point, types the structure of an 's' one. */
static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  uint64_t v[MAX_ARGS];
  char arena[MAX_STRUCTS * 64] __attribute__((aligned(16)));
  Py_ssize_t used = 0;
  Py_buffer held[MAX_ARGS];
  int nheld = 0, known = 1, rc = 0;
  if (n < 1 || n - 1 > MAX_ARGS || !struct_type || !PyTuple_Check(args[0]) || PyTuple_GET_SIZE(args[0]) != 3) Py_RETURN_NOTIMPLEMENTED;
  PyObject *address = PyTuple_GET_ITEM(args[0], 0), *kinds = PyTuple_GET_ITEM(args[0], 1), *types = PyTuple_GET_ITEM(args[0], 2);
  if (!PyLong_Check(address) || !PyBytes_Check(kinds) || PyBytes_GET_SIZE(kinds) != n - 1 || !PyTuple_Check(types) || PyTuple_GET_SIZE(types) != n - 1)
    Py_RETURN_NOTIMPLEMENTED;
  memset(v, 0, sizeof(v));
  for (Py_ssize_t k = 1; k < n && known; ++k) {
    PyObject *a = args[k], *type = (PyObject*)Py_TYPE(a);
    const char kind = PyBytes_AS_STRING(kinds)[k - 1];
    uint64_t* out = &v[k - 1];
    int by_address = 0;
    switch (kind) {
      case 'i':
        if (PyLong_Check(a)) *out = PyLong_AsUnsignedLongLongMask(a); else known = 0;
        break;
      case 'v':
        if (PyLong_Check(a)) *out = PyLong_AsUnsignedLongLongMask(a);
        else if (type == voidp_type) by_address = 1;
        else known = a == Py_None;
        break;
      case 'n':
        known = a == Py_None;
        break;
      case 'T':
        if (a == Py_None) break;   /* fall through */
      case 't':
        by_address = known = type == tensor_type;
        break;
      case 's':
        by_address = known = type == PyTuple_GET_ITEM(types, k - 1);
        break;
      case 'a':
        if (a == Py_None) break;
        by_address = known = PyObject_IsInstance(a, struct_type) == 1;
        break;
      case 'x': {
        if (a == Py_None) break;
        if (!PyList_Check(a) && !PyTuple_Check(a)) { known = 0; break; }
        const Py_ssize_t len = PySequence_Fast_GET_SIZE(a);
        PyObject** items = PySequence_Fast_ITEMS(a);
        if ((used + len) * tensor_size > (Py_ssize_t)sizeof(arena)) { known = 0; break; }
        *out = len ? (uint64_t)(uintptr_t)(arena + used * tensor_size) : 0;
        for (Py_ssize_t i = 0; i < len && known; ++i, ++used) {
          Py_buffer b;
          if ((PyObject*)Py_TYPE(items[i]) != tensor_type || PyObject_GetBuffer(items[i], &b, PyBUF_SIMPLE) != 0) { known = 0; break; }
          if (b.len == tensor_size) memcpy(arena + used * tensor_size, b.buf, (size_t)tensor_size); else known = 0;
          PyBuffer_Release(&b);
        }
        break;
      }
      default: known = 0;
    }
    if (known && by_address) {
      if (PyObject_GetBuffer(a, &held[nheld], PyBUF_SIMPLE) != 0) { known = 0; break; }
      if (kind == 'v') memcpy(out, held[nheld].buf, sizeof(uint64_t));
      else *out = (uint64_t)(uintptr_t)held[nheld].buf;
      ++nheld;
    }
  }
  if (known && !PyErr_Occurred()) {
    const entry f = (entry)(uintptr_t)PyLong_AsUnsignedLongLongMask(address);
    Py_BEGIN_ALLOW_THREADS
    rc = f(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10], v[11], v[12], v[13], v[14], v[15], v[16], v[17], v[18], v[19], v[20], v[21],
           v[22], v[23]);
    Py_END_ALLOW_THREADS
  }
  for (int k = 0; k < nheld; ++k) PyBuffer_Release(&held[k]);
  if (PyErr_Occurred()) { PyErr_Clear(); known = 0; }
  if (!known) Py_RETURN_NOTIMPLEMENTED;
  return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {{"setup", setup, METH_VARARGS, "setup(Structure, tensor type, c_void_p, size of a tensor)"},
                                {"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, "call((address, kinds, types), *arguments) -> status or NotImplemented"},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__call(void) { return PyModule_Create(&module); }
