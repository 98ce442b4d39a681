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
 * number of them, makes call() return NotImplemented, and the binding takes the ctypes route, which converts it or raises.  The GIL is released around the call, as ctypes does.
 *
 * Context.fwd and .bwd are replaced by method(), the same in C: the entry point looked up, the list measured and the status checked without a Python frame.  And a
 * structure's address is read from the object (an instance keeps it behind its header, which setup() checks on one; else through the buffer protocol, 50 ns
 * each and up to seven per call).  A node call on 100 x 16 values, of which the launch is 1.9 us: 2.53 - 2.64 us with the function in Python, 2.48 - 2.61 like this
 * (bursts of 24 and of 200 calls, 1 to 3 % on every one of three runs). */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#define MAX_ARGS 24
#define MAX_STRUCTS 128

static PyObject *struct_type, *tensor_type, *voidp_type;
static Py_ssize_t tensor_size;
static int direct;   /* the address of a ctypes instance's memory lies right behind its object header */

static char* instance_memory(PyObject* a) { return *(char**)((char*)a + sizeof(PyObject)); }

/* setup(Structure, tensor type, c_void_p, size of a tensor, a tensor, its ctypes.addressof) */
static PyObject* setup(PyObject* self, PyObject* args) {
  PyObject *s, *t, *p, *sample;
  Py_ssize_t n;
  unsigned long long at;
  if (!PyArg_ParseTuple(args, "OOOnOK", &s, &t, &p, &n, &sample, &at)) return NULL;
  if (n > 64) { PyErr_SetString(PyExc_ValueError, "tensor structure too large"); return NULL; }
  Py_INCREF(s); Py_INCREF(t); Py_INCREF(p);
  struct_type = s; tensor_type = t; voidp_type = p; tensor_size = n;
  direct = (PyObject*)Py_TYPE(sample) == t && Py_TYPE(sample)->tp_basicsize >= (Py_ssize_t)(sizeof(PyObject) + sizeof(char*)) &&
           (uint64_t)(uintptr_t)instance_memory(sample) == at;
  Py_RETURN_NONE;
}

typedef int (*entry)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                     uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t);

/* Calls the entry point of `e` = (address, kinds, types): kinds has one letter per parameter, types the structure of an 's' one.  items: the `count` arguments; NULL
 * stands for the integer `len`.  1: called, *status is its result; 0: an argument of another kind. */
static int run(PyObject* e, PyObject* const* items, Py_ssize_t count, uint64_t len, int* status) {
  uint64_t v[MAX_ARGS];
  char arena[MAX_STRUCTS * 64] __attribute__((aligned(16)));
  Py_ssize_t used = 0;
  Py_buffer held[MAX_ARGS];
  int nheld = 0, known = 1, rc = 0;
  if (count > MAX_ARGS || !struct_type || !PyTuple_Check(e) || PyTuple_GET_SIZE(e) != 3) return 0;
  PyObject *address = PyTuple_GET_ITEM(e, 0), *kinds = PyTuple_GET_ITEM(e, 1), *types = PyTuple_GET_ITEM(e, 2);
  if (!PyLong_Check(address) || !PyBytes_Check(kinds) || PyBytes_GET_SIZE(kinds) != count || !PyTuple_Check(types) || PyTuple_GET_SIZE(types) != count) return 0;
  memset(v, 0, sizeof(v));
  for (Py_ssize_t k = 0; k < count && known; ++k) {
    PyObject* a = items[k];
    const char kind = PyBytes_AS_STRING(kinds)[k];
    uint64_t* out = &v[k];
    int by_address = 0;
    if (!a) {
      if (kind == 'i') *out = len; else known = 0;
      continue;
    }
    PyObject* type = (PyObject*)Py_TYPE(a);
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
        by_address = known = type == PyTuple_GET_ITEM(types, k);
        break;
      case 'a':
        if (a == Py_None) break;
        by_address = known = PyType_IsSubtype(Py_TYPE(a), (PyTypeObject*)struct_type);
        break;
      case 'x': {
        if (a == Py_None) break;
        if (!PyList_Check(a) && !PyTuple_Check(a)) { known = 0; break; }
        const Py_ssize_t n = PySequence_Fast_GET_SIZE(a);
        PyObject** list = PySequence_Fast_ITEMS(a);
        if ((used + n) * tensor_size > (Py_ssize_t)sizeof(arena)) { known = 0; break; }
        *out = n ? (uint64_t)(uintptr_t)(arena + used * tensor_size) : 0;
        for (Py_ssize_t i = 0; i < n && known; ++i, ++used) {
          Py_buffer b;
          if ((PyObject*)Py_TYPE(list[i]) != tensor_type) { known = 0; break; }
          if (direct) { memcpy(arena + used * tensor_size, instance_memory(list[i]), (size_t)tensor_size); continue; }
          if (PyObject_GetBuffer(list[i], &b, PyBUF_SIMPLE) != 0) { known = 0; break; }
          if (b.len == tensor_size) memcpy(arena + used * tensor_size, b.buf, (size_t)tensor_size); else known = 0;
          PyBuffer_Release(&b);
        }
        break;
      }
      default: known = 0;
    }
    if (known && by_address) {
      const char* at;
      if (direct) at = instance_memory(a);
      else {
        if (PyObject_GetBuffer(a, &held[nheld], PyBUF_SIMPLE) != 0) { known = 0; break; }
        at = held[nheld++].buf;
      }
      if (kind == 'v') memcpy(out, at, sizeof(uint64_t));
      else *out = (uint64_t)(uintptr_t)at;
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
  *status = rc;
  return known;
}

/* call((address, kinds, types), *arguments) */
static PyObject* call(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  int rc;
  if (n < 1 || !run(args[0], args + 1, n - 1, 0, &rc)) Py_RETURN_NOTIMPLEMENTED;
  return PyLong_FromLong(rc);
}

/* method(function, name of the entries' dictionary, number of parameters, names of the handle and of the check): `function` is the method in Python, of the parameters
 * self, node, xs, ...; what run() does not take goes to it. */
typedef struct {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  PyObject *function, *entries, *handle, *check;
  Py_ssize_t params;
} Method;

static PyObject* method_call(PyObject* callable, PyObject* const* args, size_t nargsf, PyObject* names) {
  Method* m = (Method*)callable;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (!names && n >= 4 && n <= m->params && PyUnicode_CheckExact(args[1])) {
    PyObject *self = args[0], *xs = args[2], *entries = PyObject_GetAttr(self, m->entries), *handle = entries ? PyObject_GetAttr(self, m->handle) : NULL;
    int called = 0, rc = 0;
    if (handle && PyDict_CheckExact(entries)) {
      PyObject* e = PyDict_GetItemWithError(entries, args[1]);
      const int list = PyList_CheckExact(xs) || PyTuple_CheckExact(xs);
      if (e && (list || xs == Py_None)) {
        PyObject* items[MAX_ARGS];
        Py_ssize_t k = 0;
        Py_INCREF(e);
        items[k++] = xs;
        items[k++] = NULL;
        for (Py_ssize_t i = 3; i < m->params; ++i) items[k++] = i < n ? args[i] : Py_None;
        items[k++] = handle;
        called = run(e, items, k, list ? (uint64_t)PySequence_Fast_GET_SIZE(xs) : 0, &rc);
        Py_DECREF(e);
      }
    }
    Py_XDECREF(entries);
    Py_XDECREF(handle);
    PyErr_Clear();
    if (called) {
      if (rc == 0) Py_RETURN_NONE;
      PyObject *status = PyLong_FromLong(rc), *out = status ? PyObject_CallMethodOneArg(self, m->check, status) : NULL;
      Py_XDECREF(status);
      if (!out) return NULL;
      Py_DECREF(out);
      Py_RETURN_NONE;
    }
  }
  return PyObject_Vectorcall(m->function, args, nargsf, names);
}

static PyObject* method_get(PyObject* self, PyObject* obj, PyObject* type) {
  if (!obj || obj == Py_None) return Py_NewRef(self);
  return PyMethod_New(self, obj);
}
static PyObject* method_getattro(PyObject* self, PyObject* name) {   /* (its documentation, its name: the function's) */
  PyObject* v = PyObject_GenericGetAttr(self, name);
  if (v || !PyErr_ExceptionMatches(PyExc_AttributeError)) return v;
  PyErr_Clear();
  return PyObject_GetAttr(((Method*)self)->function, name);
}
static int method_traverse(PyObject* self, visitproc visit, void* arg) {
  Method* m = (Method*)self;
  Py_VISIT(m->function); Py_VISIT(m->entries); Py_VISIT(m->handle); Py_VISIT(m->check);
  return 0;
}
static int method_clear(PyObject* self) {
  Method* m = (Method*)self;
  Py_CLEAR(m->function); Py_CLEAR(m->entries); Py_CLEAR(m->handle); Py_CLEAR(m->check);
  return 0;
}
static void method_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  method_clear(self);
  PyObject_GC_Del(self);
}
static PyTypeObject MethodType = {
  PyVarObject_HEAD_INIT(NULL, 0)
  .tp_name = "dynet_b200._call.method", .tp_basicsize = sizeof(Method), .tp_dealloc = method_dealloc, .tp_vectorcall_offset = offsetof(Method, vectorcall),
  .tp_call = PyVectorcall_Call, .tp_getattro = method_getattro,
  .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL | Py_TPFLAGS_METHOD_DESCRIPTOR, .tp_traverse = method_traverse, .tp_clear = method_clear,
  .tp_descr_get = method_get,
};

static PyObject* method(PyObject* self, PyObject* args) {
  PyObject *f, *entries, *handle, *check;
  Py_ssize_t params;
  if (!PyArg_ParseTuple(args, "OUnUU", &f, &entries, &params, &handle, &check)) return NULL;
  if (params < 4 || params + 2 > MAX_ARGS) { PyErr_SetString(PyExc_ValueError, "number of parameters"); return NULL; }
  Method* m = PyObject_GC_New(Method, &MethodType);
  if (!m) return NULL;
  m->vectorcall = method_call;
  m->params = params;
  m->function = Py_NewRef(f); m->entries = Py_NewRef(entries); m->handle = Py_NewRef(handle); m->check = Py_NewRef(check);
  PyObject_GC_Track((PyObject*)m);
  return (PyObject*)m;
}

static PyMethodDef methods[] = {{"setup", setup, METH_VARARGS, "setup(Structure, tensor type, c_void_p, size of a tensor, a tensor, its address)"},
                                {"call", (PyCFunction)(void (*)(void))call, METH_FASTCALL, "call((address, kinds, types), *arguments) -> status or NotImplemented"},
                                {"method", method, METH_VARARGS, "method(function, entries' name, parameters, handle's name, check's name)"},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__call(void) {
  if (PyType_Ready(&MethodType) < 0) return NULL;
  return PyModule_Create(&module);
}
