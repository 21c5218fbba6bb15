/* fastcall.c - CPython call layer of the op-level entry points that a caller issues once per kernel or two (lib.py). A ctypes call
 * with six to eighteen arguments takes about as long as the kernel launch behind it (two calls and launches: 7.0 to 8.2 us of host
 * time); here the arguments are converted in place (4.9 to 5.1 us, and 1024 x 4096 with its quantiser 7.1 -> 5.4 us, the GPU's time).
 * The functions are not linked: bind() takes their addresses in the library that lib.py has loaded, so the two cannot differ.
 * Handles are integers (0 = null). As with ctypes, whole numbers are taken modulo the parameter's width and the interpreter is
 * released during the call. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>

typedef void *P;
typedef size_t Z;

/* argument i as a 64-bit pattern; errors are collected and looked at once */
static uint64_t arg(PyObject *const *a, Py_ssize_t i) { return PyLong_AsUnsignedLongLongMask(a[i]); }
#define AP(i) ((P)(uintptr_t)arg(a, i))
#define AZ(i) ((Z)arg(a, i))
#define AI(i) ((int)(uint32_t)arg(a, i))

/* one entry point: NAME, number of arguments, the C prototype and the converted arguments */
#define ENTRY(NAME, N, PROTO, DECL, ARGS)                                                        \
    static int(*p_##NAME) PROTO;                                                                 \
    static PyObject *f_##NAME(PyObject *self, PyObject *const *a, Py_ssize_t n) {                \
        (void)self;                                                                              \
        if (n != N) return PyErr_Format(PyExc_TypeError, #NAME " takes %d arguments, got %zd", N, n); \
        if (!p_##NAME) return PyErr_Format(PyExc_RuntimeError, #NAME " is not bound");          \
        DECL;                                                                                    \
        if (PyErr_Occurred()) return NULL;                                                       \
        int rc;                                                                                  \
        Py_BEGIN_ALLOW_THREADS                                                                   \
        rc = p_##NAME ARGS;                                                                      \
        Py_END_ALLOW_THREADS                                                                     \
        return PyLong_FromLong(rc);                                                              \
    }

ENTRY(bn_act_quant_q81, 6, (P, P, Z, int, P, Z),
      P c = AP(0); P x = AP(1); Z xo = AZ(2); int K = AI(3); P p = AP(4); Z po = AZ(5),
      (c, x, xo, K, p, po))
ENTRY(bn_gemv_q81, 11, (P, P, Z, int, int, P, Z, P, Z, P, Z),
      P c = AP(0); P w = AP(1); Z wo = AZ(2); int M = AI(3); int K = AI(4); P p = AP(5); Z po = AZ(6); P o = AP(7); Z oo = AZ(8); P d = AP(9); Z dof = AZ(10),
      (c, w, wo, M, K, p, po, o, oo, d, dof))
ENTRY(bn_gemm_act_quant, 11, (P, P, Z, Z, int, int, P, Z, int, P, Z),
      P c = AP(0); P x = AP(1); Z xo = AZ(2); Z xs = AZ(3); int K = AI(4); int nc = AI(5); P s = AP(6); Z so = AZ(7); int hb = AI(8); P im = AP(9); Z io = AZ(10),
      (c, x, xo, xs, K, nc, s, so, hb, im, io))
ENTRY(bn_gemm_q81, 12, (P, P, Z, int, int, int, P, Z, int, P, Z, Z),
      P c = AP(0); P w = AP(1); Z wo = AZ(2); int t = AI(3); int M = AI(4); int K = AI(5); P im = AP(6); Z io = AZ(7); int nc = AI(8); P o = AP(9); Z oo = AZ(10); Z os = AZ(11),
      (c, w, wo, t, M, K, im, io, nc, o, oo, os))
ENTRY(bn_attn_insert, 18, (P, P, P, Z, P, Z, P, Z, int, int, P, Z, P, Z, P, Z, P, Z),
      P c = AP(0); P d = AP(1); P kv = AP(2); Z kvo = AZ(3); P k = AP(4); Z ko = AZ(5); P v = AP(6); Z vo = AZ(7); int m = AI(8); int pos = AI(9); P q = AP(10); Z qo = AZ(11);
      P qn = AP(12); Z qno = AZ(13); P kn = AP(14); Z kno = AZ(15); P s = AP(16); Z so = AZ(17),
      (c, d, kv, kvo, k, ko, v, vo, m, pos, q, qo, qn, qno, kn, kno, s, so))
ENTRY(bn_attn_attend, 11, (P, P, P, Z, int, P, Z, P, Z, P, Z),
      P c = AP(0); P d = AP(1); P kv = AP(2); Z kvo = AZ(3); int pos = AI(4); P s = AP(5); Z so = AZ(6); P pg = AP(7); Z pgo = AZ(8); P g = AP(9); Z go = AZ(10),
      (c, d, kv, kvo, pos, s, so, pg, pgo, g, go))

/* bind({name: address}) */
static PyObject *bind(PyObject *self, PyObject *table) {
    (void)self;
    if (!PyDict_Check(table)) return PyErr_Format(PyExc_TypeError, "bind takes a dict");
#define BIND(NAME)                                                                               \
    do {                                                                                         \
        PyObject *v = PyDict_GetItemString(table, #NAME);                                        \
        if (!v) return PyErr_Format(PyExc_KeyError, #NAME);                                      \
        void *f = PyLong_AsVoidPtr(v);                                                           \
        if (PyErr_Occurred()) return NULL;                                                       \
        *(void **)&p_##NAME = f;                                                                 \
    } while (0)
    BIND(bn_act_quant_q81); BIND(bn_gemv_q81); BIND(bn_gemm_act_quant); BIND(bn_gemm_q81); BIND(bn_attn_insert); BIND(bn_attn_attend);
    Py_RETURN_NONE;
}

#define METHOD(NAME) {#NAME, (PyCFunction)(void (*)(void))f_##NAME, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {{"bind", bind, METH_O, NULL},  METHOD(bn_act_quant_q81), METHOD(bn_gemv_q81), METHOD(bn_gemm_act_quant),
                                METHOD(bn_gemm_q81), METHOD(bn_attn_insert), METHOD(bn_attn_attend), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&module); }
