/* Calls of the C ABI that a Python program makes once per linear, without ctypes' argument
 * conversion: module elutq_b200._hlq_call.  Each function takes the address of the library's entry
 * point (from the ctypes binding, which stays the one place that loads the library) and its
 * arguments as Python ints, releases the GIL for the call and returns the hlq_status.
 * Measured (one call with 13 arguments): 0.4 us, through ctypes 2.1 us. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

typedef int (*linear_forward_fn)(int, int, int, int, const void *, int, void *, int, void *, size_t, const void *,
                                 void *);
typedef int (*group_forward_fn)(void *, int, void *);

/* Converts args[i]; false with a Python error set when it is not an int (None is NULL). */
static int as_u64(PyObject *o, unsigned long long *out) {
    if (o == Py_None) {
        *out = 0;
        return 1;
    }
    *out = PyLong_AsUnsignedLongLongMask(o);
    return !(*out == (unsigned long long)-1 && PyErr_Occurred());
}

static int convert(PyObject *const *args, Py_ssize_t nargs, Py_ssize_t want, unsigned long long *v) {
    if (nargs != want) {
        PyErr_Format(PyExc_TypeError, "%zd arguments expected, %zd given", want, nargs);
        return 0;
    }
    for (Py_ssize_t i = 0; i < want; ++i)
        if (!as_u64(args[i], &v[i])) return 0;
    if (!v[0]) {
        PyErr_SetString(PyExc_ValueError, "no entry point");
        return 0;
    }
    return 1;
}

/* linear_forward(fn, impl, m, k, n, x, x_dtype, y, y_dtype, workspace, workspace_bytes, weight, stream) */
static PyObject *linear_forward(PyObject *self, PyObject *const *args, Py_ssize_t nargs) {
    unsigned long long v[13];
    int rc;
    (void)self;
    if (!convert(args, nargs, 13, v)) return NULL;
    Py_BEGIN_ALLOW_THREADS
    rc = ((linear_forward_fn)(uintptr_t)v[0])((int)v[1], (int)v[2], (int)v[3], (int)v[4], (const void *)(uintptr_t)v[5],
                                              (int)v[6], (void *)(uintptr_t)v[7], (int)v[8], (void *)(uintptr_t)v[9],
                                              (size_t)v[10], (const void *)(uintptr_t)v[11], (void *)(uintptr_t)v[12]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

/* group_forward(fn, group, m, stream) */
static PyObject *group_forward(PyObject *self, PyObject *const *args, Py_ssize_t nargs) {
    unsigned long long v[4];
    int rc;
    (void)self;
    if (!convert(args, nargs, 4, v)) return NULL;
    Py_BEGIN_ALLOW_THREADS
    rc = ((group_forward_fn)(uintptr_t)v[0])((void *)(uintptr_t)v[1], (int)v[2], (void *)(uintptr_t)v[3]);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static PyMethodDef methods[] = {
    {"linear_forward", (PyCFunction)(void (*)(void))linear_forward, METH_FASTCALL, "hlq_linear_forward_impl"},
    {"group_forward", (PyCFunction)(void (*)(void))group_forward, METH_FASTCALL, "hlq_group_forward"},
    {NULL, NULL, 0, NULL},
};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_hlq_call", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__hlq_call(void) { return PyModule_Create(&module); }
