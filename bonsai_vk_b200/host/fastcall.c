/* fastcall.c - CPython call layer of the op-level entry points that a caller issues once per kernel or two (lib.py). A ctypes call
 * with six to eighteen arguments takes about as long as the kernel launch behind it (two calls and launches: 7.0 to 8.2 us of host
 * time); here the arguments are converted in place (4.9 to 5.1 us, and 1024 x 4096 with its quantiser 7.1 -> 5.4 us, the GPU's time).
 * The functions are not linked: bind() takes their addresses in the library that lib.py has loaded; their types are the header's.
 * Handles are integers (0 = null). As with ctypes, whole numbers are taken modulo the parameter's width and the interpreter is
 * released during the call. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>

#include "bonsai_cuda.h"

/* the whole numbers of a call as 64-bit patterns; 0 where an argument is none */
static int whole(PyObject *const *a, Py_ssize_t n, uint64_t *v) {
    for (Py_ssize_t i = 0; i < n; ++i) {
        v[i] = PyLong_AsUnsignedLongLongMask(a[i]);
        if (v[i] == (uint64_t)-1 && PyErr_Occurred()) return 0;
    }
    return 1;
}
#define P(i) ((void *)(uintptr_t)v[i])
#define Z(i) ((size_t)v[i])
#define I(i) ((int)(uint32_t)v[i])

/* one entry point: NAME, number of arguments and the converted arguments, of the types that the header declares. What is no whole
 * number (a ctypes instance, or a mistake) goes to the ctypes function, which takes or refuses it. */
#define ENTRY(NAME, N, ARGS)                                                                     \
    static __typeof__(&NAME) p_##NAME;                                                           \
    static PyObject *c_##NAME;                                                                   \
    static PyObject *f_##NAME(PyObject *self, PyObject *const *a, Py_ssize_t n) {                \
        (void)self;                                                                              \
        if (n != N) return PyErr_Format(PyExc_TypeError, #NAME " takes %d arguments, got %zd", N, n); \
        if (!p_##NAME) return PyErr_Format(PyExc_RuntimeError, #NAME " is not bound");          \
        uint64_t v[N];                                                                           \
        if (!whole(a, N, v)) {                                                                   \
            PyErr_Clear();                                                                       \
            return PyObject_Vectorcall(c_##NAME, a, N, NULL);                                    \
        }                                                                                        \
        int rc;                                                                                  \
        Py_BEGIN_ALLOW_THREADS                                                                   \
        rc = p_##NAME ARGS;                                                                      \
        Py_END_ALLOW_THREADS                                                                     \
        return PyLong_FromLong(rc);                                                              \
    }

ENTRY(bn_act_quant_q81, 6, (P(0), P(1), Z(2), I(3), P(4), Z(5)))
ENTRY(bn_gemv_q81, 11, (P(0), P(1), Z(2), I(3), I(4), P(5), Z(6), P(7), Z(8), P(9), Z(10)))
ENTRY(bn_gemm_act_quant, 11, (P(0), P(1), Z(2), Z(3), I(4), I(5), P(6), Z(7), I(8), P(9), Z(10)))
ENTRY(bn_gemm_q81, 12, (P(0), P(1), Z(2), I(3), I(4), I(5), P(6), Z(7), I(8), P(9), Z(10), Z(11)))
ENTRY(bn_attn_insert, 18, (P(0), P(1), P(2), Z(3), P(4), Z(5), P(6), Z(7), I(8), I(9), P(10), Z(11), P(12), Z(13), P(14), Z(15), P(16), Z(17)))
ENTRY(bn_attn_attend, 11, (P(0), P(1), P(2), Z(3), I(4), P(5), Z(6), P(7), Z(8), P(9), Z(10)))

/* bind({name: (address, ctypes function)}) */
static PyObject *bind(PyObject *self, PyObject *table) {
    (void)self;
    if (!PyDict_Check(table)) return PyErr_Format(PyExc_TypeError, "bind takes a dict");
#define BIND(NAME)                                                                               \
    do {                                                                                         \
        PyObject *at, *slow, *e = PyDict_GetItemString(table, #NAME);                            \
        if (!e) return PyErr_Format(PyExc_KeyError, #NAME);                                      \
        if (!PyArg_ParseTuple(e, "OO", &at, &slow)) return NULL;                                 \
        void *f = PyLong_AsVoidPtr(at);                                                          \
        if (PyErr_Occurred()) return NULL;                                                       \
        *(void **)&p_##NAME = f;                                                                 \
        Py_INCREF(slow);                                                                         \
        Py_XSETREF(c_##NAME, slow);                                                              \
    } while (0)
    BIND(bn_act_quant_q81); BIND(bn_gemv_q81); BIND(bn_gemm_act_quant); BIND(bn_gemm_q81); BIND(bn_attn_insert); BIND(bn_attn_attend);
    Py_RETURN_NONE;
}

#define METHOD(NAME) {#NAME, (PyCFunction)(void (*)(void))f_##NAME, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {{"bind", bind, METH_O, NULL},  METHOD(bn_act_quant_q81), METHOD(bn_gemv_q81), METHOD(bn_gemm_act_quant),
                                METHOD(bn_gemm_q81), METHOD(bn_attn_insert), METHOD(bn_attn_attend), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&module); }
