/* CPython entry points of the kernel-level calls that take a few microseconds of device work. The arguments are those of the C ABI
 * (include/hipster_b200.h): integers for numbers and addresses, None for an absent buffer, the stream last. ctypes spends a microsecond
 * on converting nine such arguments, these functions a tenth of it. The library is not linked: bind() takes the addresses of its functions,
 * so that the module calls the library that the package has loaded. The interpreter lock is released around each call, as ctypes does. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

typedef struct { const char* name; void* fn; } Bound;
enum { QUANTIZE, GEMV, ARGMAX, ACCEPT, ATTN, N_BOUND };
static Bound bound[N_BOUND] = {{"hp_quantize_x_q8", NULL}, {"hp_gemv_q4k_q8", NULL}, {"hp_argmax", NULL}, {"hp_accept_greedy", NULL}, {"hp_attn_decode", NULL}};

static void* as_ptr(PyObject* o) { return o == Py_None ? NULL : (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(o); }
static int as_int(PyObject* o) { return (int)PyLong_AsUnsignedLongLongMask(o); }

/* argument count and binding; afterwards PyErr_Occurred() tells whether a conversion failed */
static int usable(int which, Py_ssize_t n, Py_ssize_t want) {
    if (n != want) { PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, %zd were given", bound[which].name, want, n); return 0; }
    if (!bound[which].fn) { PyErr_Format(PyExc_RuntimeError, "%s is not bound", bound[which].name); return 0; }
    return 1;
}
#define CALL(expr) do { int rc_; if (PyErr_Occurred()) return NULL; Py_BEGIN_ALLOW_THREADS rc_ = (expr); Py_END_ALLOW_THREADS return PyLong_FromLong(rc_); } while (0)

static PyObject* py_quantize(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    if (!usable(QUANTIZE, n, 7)) return NULL;
    void *x = as_ptr(a[0]), *q = as_ptr(a[4]), *sc = as_ptr(a[5]), *s = as_ptr(a[6]);
    const int ldx = as_int(a[1]), R = as_int(a[2]), K = as_int(a[3]);
    CALL(((int (*)(const float*, int, int, int, void*, void*, void*))bound[QUANTIZE].fn)(x, ldx, R, K, q, sc, s));
}
static PyObject* py_gemv(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    if (!usable(GEMV, n, 9)) return NULL;
    void *w = as_ptr(a[0]), *q = as_ptr(a[1]), *sc = as_ptr(a[2]), *y = as_ptr(a[3]), *s = as_ptr(a[8]);
    const int N = as_int(a[4]), K = as_int(a[5]), R = as_int(a[6]), ldy = as_int(a[7]);
    CALL(((int (*)(const void*, const void*, const void*, float*, int, int, int, int, void*))bound[GEMV].fn)(w, q, sc, y, N, K, R, ldy, s));
}
static PyObject* py_argmax(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    if (!usable(ARGMAX, n, 8)) return NULL;
    void *x = as_ptr(a[0]), *ids = as_ptr(a[4]), *vals = as_ptr(a[5]), *scratch = as_ptr(a[6]), *s = as_ptr(a[7]);
    const int R = as_int(a[1]), cols = as_int(a[2]), ld = as_int(a[3]);
    CALL(((int (*)(const float*, int, int, int, int*, float*, void*, void*))bound[ARGMAX].fn)(x, R, cols, ld, ids, vals, scratch, s));
}
static PyObject* py_accept(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    if (!usable(ACCEPT, n, 5)) return NULL;
    void *ids = as_ptr(a[0]), *drafts = as_ptr(a[1]), *out = as_ptr(a[3]), *s = as_ptr(a[4]);
    const int nd = as_int(a[2]);
    CALL(((int (*)(const int*, const int*, int, int*, void*))bound[ACCEPT].fn)(ids, drafts, nd, out, s));
}
static PyObject* py_attn(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    if (!usable(ATTN, n, 19)) return NULL;
    void *qkv = as_ptr(a[0]), *qn = as_ptr(a[7]), *kn = as_ptr(a[8]), *rope = as_ptr(a[9]), *kc = as_ptr(a[10]), *vc = as_ptr(a[11]), *out = as_ptr(a[13]), *q = as_ptr(a[14]), *sc = as_ptr(a[15]),
         *ws = as_ptr(a[17]), *s = as_ptr(a[18]);
    const int ld = as_int(a[1]), R = as_int(a[2]), pos0 = as_int(a[3]), nh = as_int(a[4]), nkv = as_int(a[5]), nrot = as_int(a[6]), ctx = as_int(a[12]);
    const float eps = (float)PyFloat_AsDouble(a[16]);
    CALL(((int (*)(float*, int, int, int, int, int, int, const void*, const void*, const float*, void*, void*, int, float*, void*, void*, float, void*, void*))bound[ATTN].fn)(
        qkv, ld, R, pos0, nh, nkv, nrot, qn, kn, rope, kc, vc, ctx, out, q, sc, eps, ws, s));
}
/* bind(name, address) */
static PyObject* py_bind(PyObject* self, PyObject* args) {
    const char* name; PyObject* addr;
    if (!PyArg_ParseTuple(args, "sO", &name, &addr)) return NULL;
    for (int i = 0; i < N_BOUND; ++i)
        if (strcmp(name, bound[i].name) == 0) {
            void* p = as_ptr(addr);
            if (PyErr_Occurred()) return NULL;
            bound[i].fn = p;
            Py_RETURN_NONE;
        }
    PyErr_Format(PyExc_KeyError, "%s", name);
    return NULL;
}
static PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, "bind(name, address): the library's function behind an entry point"},
    {"hp_quantize_x_q8", (PyCFunction)(void*)py_quantize, METH_FASTCALL, NULL}, {"hp_gemv_q4k_q8", (PyCFunction)(void*)py_gemv, METH_FASTCALL, NULL},
    {"hp_argmax", (PyCFunction)(void*)py_argmax, METH_FASTCALL, NULL}, {"hp_accept_greedy", (PyCFunction)(void*)py_accept, METH_FASTCALL, NULL},
    {"hp_attn_decode", (PyCFunction)(void*)py_attn, METH_FASTCALL, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__calls(void) { return PyModule_Create(&module); }
