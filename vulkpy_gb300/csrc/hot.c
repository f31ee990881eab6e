/* CPython binding of the calls that every array operation makes (allocate,
 * launch, free).  The rest of the library is called through ctypes, which
 * costs 0.4 to 0.6 us a call; an operation on a small array makes three such
 * calls around 2 us of launch.  Each function takes the arguments of the
 * vkc_ function of its name, device handle first (an int); device pointers are
 * Buf objects, ints or None.  A status other than VKC_OK raises through the
 * Python function given to bind.  The interpreter lock is released around
 * every library call, as ctypes does.
 *
 * The module is not linked with the library: bind takes the functions'
 * addresses from the one that ctypes has loaded (VULKPY_GB300_LIB may name
 * another file than the one beside this module), so a process has one copy
 * of the library's state. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include "../../include/vulkpy_gb300.h"

/* The functions of the library that are called here. */
#define FUNCTIONS(X)                                                                                              \
  X(alloc) X(free) X(unary) X(binary) X(binary_scalar) X(broadcast_binary) X(clamp) X(reduce_all) X(reduce_axis) \
  X(arg_reduce_all) X(arg_reduce_axis) X(gather) X(gather_axis) X(matmul)
static struct {
#define X(name) __typeof__(&vkc_##name) name;
  FUNCTIONS(X)
#undef X
} lib;

static PyObject* g_check = NULL; /* check(status): raises; NULL until bind */
static PyObject *g_capture, *g_streams, *g_release;

static PyObject* unbound(void) { return PyErr_Format(PyExc_RuntimeError, "no library bound"); }

static PyObject* finish(int st) {
  if (st == VKC_OK) Py_RETURN_NONE;
  PyObject* r = PyObject_CallFunction(g_check, "i", st);
  if (r) {
    Py_DECREF(r);
    PyErr_Format(PyExc_RuntimeError, "library status %d", st);
  } else if (!PyErr_Occurred()) {
    PyErr_Format(PyExc_RuntimeError, "library status %d", st);
  }
  return NULL;
}

/* ---- Buf: one device allocation, freed stream-ordered when collected ---- */
typedef struct {
  PyObject_HEAD
  PyObject* dev;     /* the Python device object (capture, streams, release()) */
  void* h;           /* its handle */
  void* ptr;
  Py_ssize_t nbytes;
  PyObject* graph;   /* the graph whose capture allocated it, or None */
  PyObject* h2d_job; /* raw handle of a pending pinned upload, or None */
} Buf;

static PyTypeObject BufType;

static Buf* buf_alloc(PyObject* dev, void* h, Py_ssize_t nbytes, PyObject* graph) {
  Buf* b = PyObject_GC_New(Buf, &BufType);
  if (!b) return NULL;
  b->dev = Py_NewRef(dev);
  b->h = h;
  b->ptr = NULL;
  b->nbytes = nbytes;
  b->graph = Py_NewRef(graph);
  b->h2d_job = Py_NewRef(Py_None);
  PyObject_GC_Track((PyObject*)b);
  return b;
}

/* alloc(dev, handle, nbytes, graph) -> Buf on the device's current stream */
static PyObject* hot_alloc(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 4) return PyErr_Format(PyExc_TypeError, "alloc takes 4 arguments");
  if (!g_check) return unbound();
  void* h = PyLong_AsVoidPtr(a[1]);
  const Py_ssize_t nbytes = PyLong_AsSsize_t(a[2]);
  if (PyErr_Occurred()) return NULL;
  if (nbytes < 0) return PyErr_Format(PyExc_ValueError, "negative size");
  Buf* b = buf_alloc(a[0], h, nbytes, a[3]);
  if (!b) return NULL;
  int st;
  void* p = NULL;
  Py_BEGIN_ALLOW_THREADS
  st = lib.alloc((vkc_device_t)h, (size_t)nbytes, &p);
  Py_END_ALLOW_THREADS
  if (st != VKC_OK) {
    Py_DECREF(b);
    return finish(st);
  }
  b->ptr = p;
  return (PyObject*)b;
}

/* adopt(dev, handle, ptr, nbytes, graph, h2d_job) -> Buf owning ptr */
static PyObject* hot_adopt(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) return PyErr_Format(PyExc_TypeError, "adopt takes 6 arguments");
  if (!g_check) return unbound();
  void* h = PyLong_AsVoidPtr(a[1]);
  void* p = a[2] == Py_None ? NULL : PyLong_AsVoidPtr(a[2]);
  const Py_ssize_t nbytes = PyLong_AsSsize_t(a[3]);
  if (PyErr_Occurred()) return NULL;
  Buf* b = buf_alloc(a[0], h, nbytes, a[4]);
  if (!b) return NULL;
  b->ptr = p;
  Py_SETREF(b->h2d_job, Py_NewRef(a[5]));
  return (PyObject*)b;
}

static int buf_traverse(Buf* b, visitproc visit, void* arg) {
  Py_VISIT(b->dev);
  Py_VISIT(b->graph);
  Py_VISIT(b->h2d_job);
  return 0;
}

/* Free the memory: at once when no capture and no branch is open and it is
 * no graph's, else by the device object's rules. */
static void buf_release(Buf* b) {
  if (!b->ptr || !b->dev) return;
  void* p = b->ptr;
  b->ptr = NULL;
  PyObject *et, *ev, *tb;
  PyErr_Fetch(&et, &ev, &tb);
  int plain = 0;
  if (b->graph == Py_None) {
    PyObject* cap = PyObject_GetAttr(b->dev, g_capture);
    PyObject* streams = cap == Py_None ? PyObject_GetAttr(b->dev, g_streams) : NULL;
    plain = streams && PyList_CheckExact(streams) && PyList_GET_SIZE(streams) == 1;
    Py_XDECREF(cap);
    Py_XDECREF(streams);
  }
  if (plain) {
    Py_BEGIN_ALLOW_THREADS
    lib.free((vkc_device_t)b->h, p);
    Py_END_ALLOW_THREADS
  } else {
    PyErr_Clear();
    PyObject* ip = PyLong_FromVoidPtr(p);
    PyObject* r = ip ? PyObject_CallMethodObjArgs(b->dev, g_release, ip, b->graph, NULL) : NULL;
    Py_XDECREF(ip);
    Py_XDECREF(r);
  }
  PyErr_Restore(et, ev, tb); /* an error here is the interpreter's shutdown */
}

/* Before the collector clears what the release needs (the device object). */
static void buf_finalize(PyObject* self) { buf_release((Buf*)self); }

static int buf_clear(Buf* b) {
  Py_CLEAR(b->dev);
  Py_CLEAR(b->graph);
  Py_CLEAR(b->h2d_job);
  return 0;
}

static void buf_dealloc(Buf* b) {
  if (PyObject_CallFinalizerFromDealloc((PyObject*)b) < 0) return;
  PyObject_GC_UnTrack(b);
  buf_clear(b);
  PyObject_GC_Del(b);
}

static PyObject* buf_get_ptr(Buf* b, void* unused) {
  if (!b->ptr) Py_RETURN_NONE;
  return PyLong_FromVoidPtr(b->ptr);
}

static PyGetSetDef buf_getset[] = {{"ptr", (getter)buf_get_ptr, NULL, "device address, or None", NULL}, {NULL}};
static PyMemberDef buf_members[] = {
    {"dev", T_OBJECT, offsetof(Buf, dev), READONLY, NULL},
    {"nbytes", T_PYSSIZET, offsetof(Buf, nbytes), READONLY, NULL},
    {"graph", T_OBJECT, offsetof(Buf, graph), READONLY, NULL},
    {"h2d_job", T_OBJECT, offsetof(Buf, h2d_job), 0, NULL},
    {NULL}};

static PyTypeObject BufType = {
    PyVarObject_HEAD_INIT(NULL, 0).tp_name = "vulkpy_gb300._hot.Buf",
    .tp_basicsize = sizeof(Buf),
    .tp_dealloc = (destructor)buf_dealloc,
    .tp_finalize = buf_finalize,
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC,
    .tp_doc = "Device allocation, freed stream-ordered when collected.",
    .tp_traverse = (traverseproc)buf_traverse,
    .tp_clear = (inquiry)buf_clear,
    .tp_members = buf_members,
    .tp_getset = buf_getset,
};

/* ---- arguments ---- */
static void* ptr_of(PyObject* o) {
  if (Py_TYPE(o) == &BufType) return ((Buf*)o)->ptr;
  if (o == Py_None) return NULL;
  return PyLong_AsVoidPtr(o);
}
#define DEV ((vkc_device_t)PyLong_AsVoidPtr(a[0]))
#define INT(i) ((int)PyLong_AsLong(a[i]))
#define SIZE(i) (PyLong_AsSize_t(a[i]))
#define I64(i) ((int64_t)PyLong_AsLongLong(a[i]))
#define FLT(i) ((float)PyFloat_AsDouble(a[i]))
#define PTR(i) (ptr_of(a[i]))

/* name(args...): the converted arguments first, with the lock held; then the call */
#define HOT(name, count, decl, call)                                              \
  static PyObject* hot_##name(PyObject* self, PyObject* const* a, Py_ssize_t n) { \
    if (n != count) return PyErr_Format(PyExc_TypeError, #name " takes %d arguments", count); \
    if (!g_check) return unbound();                                               \
    vkc_device_t dev = DEV;                                                       \
    decl;                                                                         \
    if (PyErr_Occurred()) return NULL;                                            \
    int st;                                                                       \
    Py_BEGIN_ALLOW_THREADS                                                        \
    st = call;                                                                    \
    Py_END_ALLOW_THREADS                                                          \
    return finish(st);                                                            \
  }

HOT(unary, 5, int op = INT(1); void* x = PTR(2); void* y = PTR(3); size_t m = SIZE(4), lib.unary(dev, op, x, y, m))
HOT(binary, 6, int op = INT(1); void* x = PTR(2); void* y = PTR(3); void* z = PTR(4); size_t m = SIZE(5),
    lib.binary(dev, op, x, y, z, m))
HOT(binary_scalar, 6, int op = INT(1); void* x = PTR(2); float s = FLT(3); void* z = PTR(4); size_t m = SIZE(5),
    lib.binary_scalar(dev, op, x, s, z, m))
HOT(broadcast_binary, 9,
    int op = INT(1); void* x = PTR(2); void* sx = PTR(3); void* y = PTR(4); void* sy = PTR(5); void* z = PTR(6);
    void* sz = PTR(7); int nd = INT(8), lib.broadcast_binary(dev, op, x, sx, y, sy, z, sz, nd))
HOT(clamp, 8, void* x = PTR(1); void* lo = PTR(2); void* hi = PTR(3); float l = FLT(4); float u = FLT(5);
    void* z = PTR(6); size_t m = SIZE(7), lib.clamp(dev, x, lo, hi, l, u, z, m))
HOT(reduce_all, 7, int op = INT(1); int prec = INT(2); void* x = PTR(3); size_t m = SIZE(4); void* z = PTR(5);
    float s = FLT(6), lib.reduce_all(dev, op, prec, x, m, z, s))
HOT(reduce_axis, 9, int op = INT(1); void* x = PTR(2); size_t p = SIZE(3); size_t m = SIZE(4); size_t q = SIZE(5);
    void* z = PTR(6); int re = INT(7); float s = FLT(8), lib.reduce_axis(dev, op, x, p, m, q, z, re, s))
HOT(arg_reduce_all, 5, int op = INT(1); void* x = PTR(2); size_t m = SIZE(3); void* z = PTR(4),
    lib.arg_reduce_all(dev, op, x, m, z))
HOT(arg_reduce_axis, 7, int op = INT(1); void* x = PTR(2); size_t p = SIZE(3); size_t m = SIZE(4);
    size_t q = SIZE(5); void* z = PTR(6), lib.arg_reduce_axis(dev, op, x, p, m, q, z))
HOT(gather, 6, void* x = PTR(1); size_t m = SIZE(2); void* i = PTR(3); size_t k = SIZE(4); void* z = PTR(5),
    lib.gather(dev, x, m, i, k, z))
HOT(gather_axis, 8, void* x = PTR(1); size_t p = SIZE(2); size_t m = SIZE(3); size_t q = SIZE(4); void* i = PTR(5);
    size_t k = SIZE(6); void* z = PTR(7), lib.gather_axis(dev, x, p, m, q, i, k, z))
HOT(matmul, 8, int prec = INT(1); void* x = PTR(2); void* y = PTR(3); void* z = PTR(4); int64_t m = I64(5);
    int64_t k = I64(6); int64_t q = I64(7), lib.matmul(dev, prec, x, y, z, m, k, q))

/* bind(address, check): address(name) is that of the library's vkc_<name> */
static PyObject* hot_bind(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) return PyErr_Format(PyExc_TypeError, "bind takes 2 arguments");
  __typeof__(lib) l;
#define X(name)                                                  \
  {                                                              \
    PyObject* r = PyObject_CallFunction(a[0], "s", "vkc_" #name); \
    void* p = r ? PyLong_AsVoidPtr(r) : NULL;                    \
    Py_XDECREF(r);                                               \
    if (PyErr_Occurred()) return NULL;                           \
    if (!p) return PyErr_Format(PyExc_ValueError, "vkc_" #name " is NULL"); \
    l.name = (__typeof__(l.name))p;                              \
  }
  FUNCTIONS(X)
#undef X
  lib = l;
  Py_XSETREF(g_check, Py_NewRef(a[1]));
  Py_RETURN_NONE;
}

#define M(name) {#name, (PyCFunction)(void (*)(void))hot_##name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {M(alloc), M(adopt), M(unary), M(binary), M(binary_scalar), M(broadcast_binary),
                                M(clamp), M(reduce_all), M(reduce_axis), M(arg_reduce_all), M(arg_reduce_axis),
                                M(gather), M(gather_axis), M(matmul),
                                M(bind),
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hot", "Binding of the per-operation calls.", -1, methods};

PyMODINIT_FUNC PyInit__hot(void) {
  g_capture = PyUnicode_InternFromString("capture");
  g_streams = PyUnicode_InternFromString("streams");
  g_release = PyUnicode_InternFromString("release");
  if (!g_capture || !g_streams || !g_release || PyType_Ready(&BufType) < 0) return NULL;
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddObjectRef(m, "Buf", (PyObject*)&BufType) < 0) Py_CLEAR(m);
  return m;
}
