/* Direct calls of the library's hot entry points from Python.
 *
 * A product of one row takes the GPU about 4 us; converting its six arguments through ctypes alone takes more than one.
 * These functions take plain integers (addresses, sizes, enum values) in METH_FASTCALL form and return the status.  The
 * entry points' addresses come from the ctypes binding (bind), so nothing is linked here. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

typedef int (*mul_mat_fn)(const void*, const void*, int, void*, int, void*);
typedef int (*topk_fn)(const void*, int, int, int, int, const void*, int, float, float, void*, void*, void*);
typedef int (*ffn_fn)(const void*, const void*, const void*, const void*, const void*, int, int, void*, int, void*);

static mul_mat_fn p_mul_mat;
static topk_fn p_topk;
static ffn_fn p_ffn;

static void* address(PyObject* o) { return o == Py_None ? NULL : (void*)(uintptr_t)PyLong_AsUnsignedLongLong(o); }
static int number(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v != (int)v) PyErr_SetString(PyExc_OverflowError, "argument does not fit a C int");
    return (int)v;
}
static int arity(Py_ssize_t got, Py_ssize_t want) {
    if (got == want) return 1;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
    return 0;
}

static PyObject* bind(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    (void)self;
    if (!arity(n, 3)) return NULL;
    p_mul_mat = (mul_mat_fn)address(a[0]);
    p_topk = (topk_fn)address(a[1]);
    p_ffn = (ffn_fn)address(a[2]);
    if (PyErr_Occurred()) return NULL;
    Py_RETURN_NONE;
}
/* weight, x, m, y, y_dtype, stream */
static PyObject* mul_mat(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    (void)self;
    if (!arity(n, 6)) return NULL;
    const void *w = address(a[0]), *x = address(a[1]);
    const int m = number(a[2]);
    void* y = address(a[3]);
    const int dt = number(a[4]);
    void* s = address(a[5]);
    if (PyErr_Occurred()) return NULL;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = p_mul_mat(w, x, m, y, dt, s);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
/* logits, tokens, experts, k, mode, bias, normalize, norm_floor, scale, ids, weights, stream */
static PyObject* moe_topk(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    (void)self;
    if (!arity(n, 12)) return NULL;
    const void* z = address(a[0]);
    const int t = number(a[1]), e = number(a[2]), k = number(a[3]), mode = number(a[4]);
    const void* bias = address(a[5]);
    const int norm = number(a[6]);
    const float norm_floor = (float)PyFloat_AsDouble(a[7]), scale = (float)PyFloat_AsDouble(a[8]);
    void *ids = address(a[9]), *w = address(a[10]), *s = address(a[11]);
    if (PyErr_Occurred()) return NULL;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = p_topk(z, t, e, k, mode, bias, norm, norm_floor, scale, ids, w, s);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
/* gate_up, down, x, ids, weights, tokens, routes, y, y_dtype, stream */
static PyObject* moe_ffn(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    (void)self;
    if (!arity(n, 10)) return NULL;
    const void *g = address(a[0]), *d = address(a[1]), *x = address(a[2]), *ids = address(a[3]), *w = address(a[4]);
    const int t = number(a[5]), r = number(a[6]);
    void* y = address(a[7]);
    const int dt = number(a[8]);
    void* s = address(a[9]);
    if (PyErr_Occurred()) return NULL;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = p_ffn(g, d, x, ids, w, t, r, y, dt, s);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {{"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, "addresses of mfqb_mul_mat, mfqb_moe_topk, mfqb_moe_ffn"},
                                {"mul_mat", (PyCFunction)(void (*)(void))mul_mat, METH_FASTCALL, "mfqb_mul_mat"},
                                {"moe_topk", (PyCFunction)(void (*)(void))moe_topk, METH_FASTCALL, "mfqb_moe_topk"},
                                {"moe_ffn", (PyCFunction)(void (*)(void))moe_ffn, METH_FASTCALL, "mfqb_moe_ffn"},
                                {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast", "Direct calls of the library's hot entry points.", -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__fast(void) { return PyModule_Create(&module); }
