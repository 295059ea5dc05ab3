/* fastcall.c - the entry points of the C ABI as Python callables without ctypes in between.
 *
 * A decode step whose row count changes from call to call issues its launches one by one, and with short kernels the time per
 * call is what bounds it: through a Python function and ctypes a call of six arguments took 4.1 us, 1.7 of them before the
 * launch; from here 3.0 and 0.4 (eight layers of projections at four rows, 40 calls: 185 -> 125 us). build.py writes fastcall_calls.inc, one function per parameter list of the
 * header, from the header itself.
 *
 * A Call takes what the Python function takes: tensors (their device address), integers, floats, None as a null pointer; the current
 * CUDA stream is appended. Whatever it does not know - other types, values out of range, another number of arguments,
 * tensor subclasses - goes to the Python function unchanged. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <limits.h>
#include <pthread.h>
#include <structmember.h>

typedef struct {
  PyObject_HEAD
  vectorcallfunc call;
  void* fn;
  PyObject* slow;      /* the Python function */
  PyObject* fail;      /* called with a return code other than 0; raises */
  PyObject* name;
} Call;

static PyObject *tensor_type, *parameter_type, *first_stream, *raw_stream, *get_device, *s_data_ptr;
/* The first call asks the Python function for the stream (it initialises CUDA); a forked child starts over. */
static volatile int cuda_up;
static void forked(void) { cuda_up = 0; }

static int as_u64(PyObject* o, unsigned long long* v) {
  *v = PyLong_AsUnsignedLongLong(o);
  if (*v == (unsigned long long)-1 && PyErr_Occurred()) { PyErr_Clear(); return 0; }
  return 1;
}
/* 1: taken, 0: not for this path, -1: an exception is set */
static int as_pointer(PyObject* o, void** p) {
  unsigned long long v = 0;
  if (o == Py_None) { *p = NULL; return 1; }
  if ((PyObject*)Py_TYPE(o) == tensor_type || (PyObject*)Py_TYPE(o) == parameter_type) {
    PyObject* a = PyObject_CallMethodNoArgs(o, s_data_ptr);
    int ok;
    if (a == NULL) return -1;
    ok = PyLong_Check(a) && as_u64(a, &v);
    Py_DECREF(a);
    if (!ok) return 0;
  } else if (!PyLong_CheckExact(o) || !as_u64(o, &v)) {
    return 0;
  }
  *p = (void*)(uintptr_t)v;
  return 1;
}
static int as_integer(PyObject* o, long long lo, long long hi, long long* v) {
  int over = 0;
  if (!PyLong_CheckExact(o) && !PyBool_Check(o)) return 0;
  *v = PyLong_AsLongLongAndOverflow(o, &over);
  return over == 0 && *v >= lo && *v <= hi;
}
static int as_double(PyObject* o, double* v) {
  if (!PyFloat_CheckExact(o)) return 0;
  *v = PyFloat_AS_DOUBLE(o);
  return 1;
}
static int as_stream(void** s) {
  PyObject *d = NULL, *r = NULL;
  int ok;
  if (cuda_up) {
    d = PyObject_CallNoArgs(get_device);
    if (d != NULL) r = PyObject_CallOneArg(raw_stream, d);
    Py_XDECREF(d);
  } else {
    r = PyObject_CallNoArgs(first_stream);
  }
  if (r == NULL) return -1;
  *s = PyLong_AsVoidPtr(r);
  ok = !PyErr_Occurred();
  Py_DECREF(r);
  if (ok) cuda_up = 1;
  return ok ? 1 : -1;
}

#define TAKE(expr)                                 \
  do {                                             \
    const int got = (expr);                        \
    if (got < 0) return NULL;                      \
    if (got == 0) return PyObject_Vectorcall(c->slow, a, nargsf, kw); \
  } while (0)

static PyObject* finish(Call* c, int rc) {
  if (rc == 0) Py_RETURN_NONE;
  return PyObject_CallFunction(c->fail, "i", rc);
}

#include "fastcall_calls.inc"

static int call_traverse(PyObject* self, visitproc visit, void* arg) {
  Call* c = (Call*)self;
  Py_VISIT(c->slow);
  Py_VISIT(c->fail);
  Py_VISIT(c->name);
  return 0;
}
static int call_clear(PyObject* self) {
  Call* c = (Call*)self;
  Py_CLEAR(c->slow);
  Py_CLEAR(c->fail);
  Py_CLEAR(c->name);
  return 0;
}
static void call_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  call_clear(self);
  Py_TYPE(self)->tp_free(self);
}
static PyMemberDef call_members[] = {{"__name__", T_OBJECT, offsetof(Call, name), READONLY, NULL},
                                     {"__wrapped__", T_OBJECT, offsetof(Call, slow), READONLY, NULL},
                                     {NULL, 0, 0, 0, NULL}};
static PyTypeObject CallType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "sager_b200._fastcall.Call",
    .tp_basicsize = sizeof(Call),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_vectorcall_offset = offsetof(Call, call),
    .tp_call = PyVectorcall_Call,
    .tp_dealloc = call_dealloc,
    .tp_traverse = call_traverse,
    .tp_clear = call_clear,
    .tp_members = call_members,
};

/* bind(kinds, address, slow, fail, name): the entry point at `address`; None when no function takes such a parameter list. */
static PyObject* py_bind(PyObject* self, PyObject* args) {
  const char* kinds;
  unsigned long long address;
  PyObject *slow, *fail, *name;
  Call* c;
  vectorcallfunc f;
  (void)self;
  if (!PyArg_ParseTuple(args, "sKOOU", &kinds, &address, &slow, &fail, &name)) return NULL;
  f = call_of(kinds);
  if (f == NULL) Py_RETURN_NONE;
  c = PyObject_GC_New(Call, &CallType);
  if (c == NULL) return NULL;
  c->call = f;
  c->fn = (void*)(uintptr_t)address;
  c->slow = Py_NewRef(slow);
  c->fail = Py_NewRef(fail);
  c->name = Py_NewRef(name);
  PyObject_GC_Track((PyObject*)c);
  return (PyObject*)c;
}
/* setup(Tensor, Parameter, first_stream, raw_stream, get_device) */
static PyObject* py_setup(PyObject* self, PyObject* args) {
  PyObject *t, *p, *f, *r, *d;
  (void)self;
  if (!PyArg_ParseTuple(args, "OOOOO", &t, &p, &f, &r, &d)) return NULL;
  Py_XSETREF(tensor_type, Py_NewRef(t));
  Py_XSETREF(parameter_type, Py_NewRef(p));
  Py_XSETREF(first_stream, Py_NewRef(f));
  Py_XSETREF(raw_stream, Py_NewRef(r));
  Py_XSETREF(get_device, Py_NewRef(d));
  Py_RETURN_NONE;
}
static PyMethodDef methods[] = {{"bind", py_bind, METH_VARARGS, NULL}, {"setup", py_setup, METH_VARARGS, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__fastcall(void) {
  if (PyType_Ready(&CallType) < 0) return NULL;
  s_data_ptr = PyUnicode_InternFromString("data_ptr");
  if (s_data_ptr == NULL || pthread_atfork(NULL, NULL, forked) != 0) return NULL;
  return PyModule_Create(&module);
}
