// CPython entry to the C ABI calls that a decode step or a linear makes once per weight.
//
// A ctypes call of these functions spends 2.3-2.7 us on converting its 12 to 16 arguments, about as long as the
// kernel launch behind it and, for the smallest GEMVs, longer than the kernel; the same call through a METH_FASTCALL
// function takes 0.6 us.  With it, without a torch.cuda.Stream object per call and with the decode linear's two or more launches
// in one call, quantiser + GEMV of 1024 x 4096 Q8_0 from Python went from 21 to 8.9 us a pass and the eleven launches of an 8B
// model's decoder layer from 108 to 58 us (the GPU's own time: 4.2 and 54).
//
// Arguments are the C function's, in its order: pointers and integers as Python integers (None = NULL), the scale as a
// float; the result is the status code.  The GIL is released around the call, as ctypes does: a launch may block when the
// device's queue is full.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include "tpb200.h"

static void *ptr(PyObject *o) {
    return o == Py_None ? NULL : PyLong_AsVoidPtr(o);
}
static int64_t i64(PyObject *o) { return (int64_t)PyLong_AsLongLong(o); }
static int i32(PyObject *o) { return (int)PyLong_AsLong(o); }
static float f32(PyObject *o) { return (float)PyFloat_AsDouble(o); }

// argument i as a pointer, a 64-bit or 32-bit integer, a float
#define P(i) ptr(a[i])
#define L(i) i64(a[i])
#define I(i) i32(a[i])
#define F(i) f32(a[i])
#define CHECK_ARGS(name, want)                                                                  \
    if (n != (want)) {                                                                          \
        PyErr_Format(PyExc_TypeError, name " takes %d arguments (%zd given)", (want), n);       \
        return NULL;                                                                            \
    }
#define CALL(expr)                        \
    int rc;                               \
    if (PyErr_Occurred()) return NULL;    \
    Py_BEGIN_ALLOW_THREADS                \
    rc = (expr);                          \
    Py_END_ALLOW_THREADS                  \
    return PyLong_FromLong(rc)

static PyObject *q8_1_quantize(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    CHECK_ARGS("tpb_q8_1_quantize", 5);
    tpb_handle_t h = (tpb_handle_t)P(0);
    void *st = P(1), *x = P(2), *xq = P(4);
    int64_t elems = L(3);
    CALL(tpb_q8_1_quantize(h, st, (const float *)x, elems, xq));
}

static PyObject *gguf_gemv_q8n(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    CHECK_ARGS("tpb_gguf_gemv_q8n", 12);
    tpb_handle_t h = (tpb_handle_t)P(0);
    void *st = P(1), *y = P(3), *w = P(4), *xq = P(8);
    int fmt = I(2), ng = I(9), row_off = I(10), n_total = I(11);
    float scale = F(5);
    int64_t rows = L(6), cols = L(7);
    CALL(tpb_gguf_gemv_q8n(h, st, fmt, (float *)y, w, scale, rows, cols, xq, ng, row_off, n_total));
}

static PyObject *q8_0_gemv_f32(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    CHECK_ARGS("tpb_q8_0_gemv_f32", 8);
    tpb_handle_t h = (tpb_handle_t)P(0);
    void *st = P(1), *y = P(2), *x = P(3), *w = P(4);
    float scale = F(5);
    int64_t rows = L(6), cols = L(7);
    CALL(tpb_q8_0_gemv_f32(h, st, (float *)y, (const float *)x, w, scale, rows, cols));
}

// The decode linear: tpb_q8_1_quantize of all m rows, then one tpb_q8_0_gemv_q8n per eight of them.
static PyObject *q8_0_linear(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    CHECK_ARGS("q8_0_linear", 10);
    tpb_handle_t h = (tpb_handle_t)P(0);
    void *st = P(1), *y = P(2), *x = P(3), *w = P(5), *xq = P(9);
    int m = I(4);
    float scale = F(6);
    int64_t rows = L(7), cols = L(8);
    int rc;
    if (PyErr_Occurred()) return NULL;
    Py_BEGIN_ALLOW_THREADS
    rc = tpb_q8_1_quantize(h, st, (const float *)x, (int64_t)m * cols, xq);
    for (int r0 = 0; r0 < m && rc == TPB_OK; r0 += 8)
        rc = tpb_q8_0_gemv_q8n(h, st, (float *)y + (size_t)r0 * (size_t)rows, w, scale, rows, cols, xq, m - r0 < 8 ? m - r0 : 8, r0, m);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

static PyObject *convrot_prep(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    CHECK_ARGS("tpb_convrot_prep", 10);
    tpb_handle_t h = (tpb_handle_t)P(0);
    void *st = P(1), *x = P(2), *q = P(7), *s = P(8), *sum = P(9);
    int dt = I(3), bits = I(6);
    int64_t m = L(4), k = L(5);
    CALL(tpb_convrot_prep(h, st, x, dt, m, k, bits, (int8_t *)q, (float *)s, (int32_t *)sum));
}

static PyObject *convrot_gemm(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    CHECK_ARGS("tpb_convrot_gemm", 14);
    tpb_handle_t h = (tpb_handle_t)P(0);
    void *st = P(1), *y = P(2), *q = P(5), *s = P(6), *sum = P(7), *w = P(8), *ws = P(10);
    int dt = I(3), bits = I(9);
    int64_t ldy = L(4), m = L(11), rows = L(12), k = L(13);
    CALL(tpb_convrot_gemm(h, st, y, dt, ldy, (const int8_t *)q, (const float *)s, (const int32_t *)sum, w, bits, (const float *)ws, m,
                          rows, k));
}

static PyObject *convrot_linear(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    CHECK_ARGS("tpb_convrot_linear", 16);
    tpb_handle_t h = (tpb_handle_t)P(0);
    void *st = P(1), *y = P(2), *x = P(5), *q = P(7), *s = P(8), *sum = P(9), *w = P(10), *ws = P(12);
    int ydt = I(3), xdt = I(6), bits = I(11);
    int64_t ldy = L(4), m = L(13), rows = L(14), k = L(15);
    CALL(tpb_convrot_linear(h, st, y, ydt, ldy, x, xdt, (int8_t *)q, (float *)s, (int32_t *)sum, w, bits, (const float *)ws, m, rows,
                            k));
}

static PyMethodDef methods[] = {
    {"tpb_q8_1_quantize", (PyCFunction)(void (*)(void))q8_1_quantize, METH_FASTCALL, NULL},
    {"tpb_gguf_gemv_q8n", (PyCFunction)(void (*)(void))gguf_gemv_q8n, METH_FASTCALL, NULL},
    {"tpb_q8_0_gemv_f32", (PyCFunction)(void (*)(void))q8_0_gemv_f32, METH_FASTCALL, NULL},
    {"q8_0_linear", (PyCFunction)(void (*)(void))q8_0_linear, METH_FASTCALL, NULL},
    {"tpb_convrot_prep", (PyCFunction)(void (*)(void))convrot_prep, METH_FASTCALL, NULL},
    {"tpb_convrot_gemm", (PyCFunction)(void (*)(void))convrot_gemm, METH_FASTCALL, NULL},
    {"tpb_convrot_linear", (PyCFunction)(void (*)(void))convrot_linear, METH_FASTCALL, NULL},
    {NULL, NULL, 0, NULL},
};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tpbcall", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__tpbcall(void) { return PyModule_Create(&module); }
