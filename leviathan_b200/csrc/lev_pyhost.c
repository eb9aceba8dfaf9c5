/* Native calls of the entry points a Python host makes per token: the same C ABI that _lib.py binds through ctypes, with
 * the arguments converted here.  A ctypes call of a dozen arguments costs two microseconds, as much as the kernel launch
 * behind it; one of these costs a few tenths.  Handles and device addresses are Python integers (None: NULL), every
 * function returns the lev_status, and the interpreter lock is released while the library works. */
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "leviathan_cuda.h"

static long long I(PyObject* o) {
    if (o == Py_None) return 0;
    if (PyLong_CheckExact(o)) return PyLong_AsLongLong(o);
    PyObject* n = PyNumber_Index(o);
    if (!n) return -1;
    long long v = PyLong_AsLongLong(n);
    Py_DECREF(n);
    return v;
}
static void* P(PyObject* o) {
    if (o == Py_None) return NULL;
    return PyLong_AsVoidPtr(o);
}
static float F(PyObject* o) { return (float)PyFloat_AsDouble(o); }

/* name(arguments): n of them; BODY is the call.  Conversions come first: an error among them is raised, nothing is called. */
#define HOST_FN(NAME, N, DECL, ...)                                                                       \
    static PyObject* NAME(PyObject* self, PyObject* const* a, Py_ssize_t n) {                             \
        (void)self;                                                                                       \
        if (n != (N)) return PyErr_Format(PyExc_TypeError, #NAME " takes %d arguments, got %zd", (N), n); \
        int st;                                                                                           \
        DECL;                                                                                             \
        if (PyErr_Occurred()) return NULL;                                                                \
        Py_BEGIN_ALLOW_THREADS;                                                                           \
        st = __VA_ARGS__;                                                                                 \
        Py_END_ALLOW_THREADS;                                                                             \
        return PyLong_FromLong(st);                                                                       \
    }

HOST_FN(matvec, 11, lev_ctx* c = P(a[0]); lev_weights* w = P(a[1]); long long r0 = I(a[2]); long long rows = I(a[3]); float* x = P(a[4]);
        long long xc = I(a[5]); long long nc = I(a[6]); float* y = P(a[7]); long long cap = I(a[8]); long long sched = I(a[9]); long long fl = I(a[10]),
        lev_matvec(c, w, r0, rows, x, xc, (int)nc, y, cap, (int)sched, (unsigned)fl))
HOST_FN(matvec_fused, 14, lev_ctx* c = P(a[0]); lev_weights* w = P(a[1]); long long r0 = I(a[2]); long long rows = I(a[3]); float* x = P(a[4]);
        long long xc = I(a[5]); long long nc = I(a[6]); lev_fusion f; f.prologue = (int)I(a[7]); f.norm_weight = P(a[8]); f.eps = F(a[9]);
        f.residual = P(a[10]); f.alpha = F(a[11]); float* y = P(a[12]); long long cap = I(a[13]),
        lev_matvec_fused(c, w, r0, rows, x, xc, (int)nc, &f, y, cap))
HOST_FN(matvec_chain, 4, lev_ctx* c = P(a[0]); long long k = I(a[1]); lev_chain_op* ops = P(a[2]); long long fl = I(a[3]),
        lev_matvec_chain(c, (int)k, ops, (unsigned)fl))
HOST_FN(rmsnorm, 8, lev_ctx* c = P(a[0]); float* x = P(a[1]); long long v = I(a[2]); long long k = I(a[3]); float* w = P(a[4]); float e = F(a[5]);
        float* y = P(a[6]); float* inv = P(a[7]), lev_rmsnorm(c, x, v, k, w, e, y, inv))
HOST_FN(axpy, 6, lev_ctx* c = P(a[0]); float al = F(a[1]); float* x = P(a[2]); float* r = P(a[3]); long long k = I(a[4]); float* y = P(a[5]),
        lev_axpy(c, al, x, r, k, y))
HOST_FN(act_bf16, 4, lev_ctx* c = P(a[0]); float* x = P(a[1]); long long k = I(a[2]); void* y = P(a[3]), lev_act_bf16(c, x, k, y))
HOST_FN(gemm_prefill, 6, lev_ctx* c = P(a[0]); lev_weights* w = P(a[1]); void* x = P(a[2]); long long t = I(a[3]); float* y = P(a[4]);
        long long fl = I(a[5]), lev_gemm_prefill(c, w, x, t, y, (unsigned)fl))
HOST_FN(moe_layer, 9, lev_ctx* c = P(a[0]); lev_moe_weights* w = P(a[1]); float* x = P(a[2]); long long t = I(a[3]); long long k = I(a[4]);
        float* y = P(a[5]); int32_t* idx = P(a[6]); float* wt = P(a[7]); long long fl = I(a[8]),
        lev_moe_layer(c, w, x, t, (int)k, y, idx, wt, (unsigned)fl))
HOST_FN(moe_layer_residual, 9, lev_ctx* c = P(a[0]); lev_moe_weights* w = P(a[1]); float* x = P(a[2]); long long t = I(a[3]); long long k = I(a[4]);
        float* r = P(a[5]); float al = F(a[6]); float* y = P(a[7]); long long fl = I(a[8]),
        lev_moe_layer_residual(c, w, x, t, (int)k, r, al, y, (unsigned)fl))
HOST_FN(kv_append, 10, lev_ctx* c = P(a[0]); lev_kv_layout* l = P(a[1]); void* kp = P(a[2]); void* vp = P(a[3]); int32_t* tb = P(a[4]);
        int32_t* s = P(a[5]); int32_t* p = P(a[6]); long long nc = I(a[7]); float* k = P(a[8]); float* v = P(a[9]),
        lev_kv_append(c, l, kp, vp, tb, s, p, (int)nc, k, v))
HOST_FN(attn_decode, 13, lev_ctx* c = P(a[0]); lev_kv_layout* l = P(a[1]); void* kp = P(a[2]); void* vp = P(a[3]); int32_t* tb = P(a[4]);
        int32_t* s = P(a[5]); int32_t* p = P(a[6]); long long nc = I(a[7]); long long qh = I(a[8]); float* q = P(a[9]); long long win = I(a[10]);
        float sc = F(a[11]); float* y = P(a[12]), lev_attn_decode(c, l, kp, vp, tb, s, p, (int)nc, (int)qh, q, (int)win, sc, y))

#define ENTRY(NAME) {#NAME, (PyCFunction)(void (*)(void))NAME, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {ENTRY(matvec), ENTRY(matvec_fused), ENTRY(matvec_chain), ENTRY(rmsnorm), ENTRY(axpy),
                                ENTRY(act_bf16), ENTRY(gemm_prefill), ENTRY(moe_layer), ENTRY(moe_layer_residual), ENTRY(kv_append),
                                ENTRY(attn_decode), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pyhost", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__pyhost(void) { return PyModule_Create(&module); }
