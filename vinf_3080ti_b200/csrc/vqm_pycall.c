/* The call a decode step makes most often, vqm_qmv, from Python without ctypes: with a function that does nothing a call takes 1.02 us
 * through ctypes and 0.18 through this (the driver's launch takes 2.2).  Arguments mean what they mean to ctypes and int().
 * Optional: limited API, so that one build serves every CPython from 3.10 on; without it the call goes through ctypes. */
#define PY_SSIZE_T_CLEAN
#define Py_LIMITED_API 0x030A0000
#include <Python.h>

typedef int (*qmv_fn)(void *, const char *, const char *, const char *, int);

/* qmv(function address, handle, weight, x, y, ntok) -> status; the GIL is released during the call */
static PyObject *py_qmv(PyObject *self, PyObject *const *args, Py_ssize_t n) {
    (void)self;
    if (n != 6) {
        PyErr_SetString(PyExc_TypeError, "qmv takes 6 arguments");
        return NULL;
    }
    const qmv_fn fn = (qmv_fn)PyLong_AsVoidPtr(args[0]);
    void *const handle = PyLong_AsVoidPtr(args[1]);
    if (PyErr_Occurred()) return NULL;
    const char *name[3];
    for (int i = 0; i < 3; ++i) {
        PyObject *const s = args[2 + i];
        if (!PyUnicode_Check(s)) {
            PyErr_Format(PyExc_AttributeError, "%R object has no attribute 'encode'", (PyObject *)Py_TYPE(s));
            return NULL;
        }
        name[i] = PyUnicode_AsUTF8AndSize(s, NULL);
        if (name[i] == NULL) return NULL;
    }
    PyObject *const whole = PyNumber_Long(args[5]);
    if (whole == NULL) return NULL;
    const int ntok = (int)PyLong_AsUnsignedLongMask(whole);
    Py_DECREF(whole);
    if (PyErr_Occurred()) return NULL;
    if (fn == NULL || handle == NULL) {
        PyErr_SetString(PyExc_ValueError, "the runtime is closed");
        return NULL;
    }
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = fn(handle, name[0], name[1], name[2], ntok);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(status);
}

static PyMethodDef methods[] = {{"qmv", (PyCFunction)(void (*)(void))py_qmv, METH_FASTCALL, "vqm_qmv"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_vqm_pycall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__vqm_pycall(void) { return PyModule_Create(&module); }
