/* The Python side of the hot entry points: one C call per operator instead of a ctypes call.
 *
 * A decode step is many launches of a few microseconds each, so the host has to issue a call in
 * less time than the kernel before it runs.  Through ctypes, torch.cuda.current_stream() and the
 * properties of GGUFTensor a call cost 9 - 12 us on the host (a 16-bit two-bit trunk's layer,
 * seven calls and two regions, 69 us against 18 us on the GPU); here the arguments are read from
 * the objects in C, those of torch's from torch itself where there is a module for it (okf_pytensor.cpp), else by method and
 * attribute look-ups.  The functions return the okf_status; the callers turn it into an exception.
 * The library and that module are resolved by address (bind), so this one links against nothing.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>
#include <string.h>

#include "../../include/okf_cuda.h"

/* ---- what bind() resolves -------------------------------------------------------------- */

typedef int (*gemv_fn)(okf_ctx *, int, const okf_weights *, uint64_t, uint32_t, uint32_t, const void *, int, float *, okf_stream);
typedef int (*gemm_fn)(okf_ctx *, int, const okf_weights *, uint64_t, uint32_t, uint32_t, const void *, int, uint32_t, void *, int,
                       okf_stream);
enum { FN_GEMM, FN_GEMM_TILE, FN_GEMM_NOALLOC, FN_COUNT_GEMM };
static gemm_fn gemm_fns[FN_COUNT_GEMM];
static gemv_fn gemv_p;
static int (*parallel_begin_p)(okf_ctx *);
static int (*parallel_end_p)(okf_ctx *);
static int (*dequant_p)(okf_ctx *, int, const okf_weights *, uint64_t, uint64_t, float *, okf_stream);
static int (*embed_p)(okf_ctx *, int, const okf_weights *, uint64_t, uint32_t, uint32_t, const int32_t *, uint32_t, float *, okf_stream);
static int (*argmax_p)(okf_ctx *, const float *, uint32_t, uint32_t, int32_t *, okf_stream);
static int (*norm_p)(okf_ctx *, float *, const float *, const float *, float *, uint32_t, uint32_t, float, uint32_t, uint32_t, okf_stream);
static int (*silu_p)(okf_ctx *, float *, const float *, size_t, okf_stream);
static int (*matmul_host_p)(okf_ctx *, int, const okf_weights *, uint64_t, uint32_t, uint32_t, const float *, uint32_t, float *);

static PyObject *dt_f32, *dt_f16, *dt_bf16;         /* torch.float32, ... */
static PyObject *get_device_p, *raw_stream_p;       /* torch._C._cuda_getDevice, _cuda_getCurrentRawStream */
static PyObject *s_ctx, *s_addr, *s_stream, *s_cuda_stream, *s_type, *s_dims, *s_offset, *s_dtype, *s_data_ptr;

/* okf_pytensor.cpp's functions for the torch that is loaded, NULL: there are none */
static int (*tensor_address_p)(PyObject *o, void **out);
static int (*tensor_dtype_p)(PyObject *o, int *out);
static int (*current_stream_p)(void **out);

/* ---- reading the arguments --------------------------------------------------------------- */

/* an int (or anything int() takes, as the operators always did) modulo 2^64; -1 with an error set */
static int as_u64(PyObject *o, uint64_t *out) {
    if (PyLong_Check(o)) {
        *out = PyLong_AsUnsignedLongLongMask(o);
        return *out == (uint64_t)-1 && PyErr_Occurred() ? -1 : 0;
    }
    PyObject *n = PyNumber_Long(o);
    if (!n) return -1;
    *out = PyLong_AsUnsignedLongLongMask(n);
    Py_DECREF(n);
    return *out == (uint64_t)-1 && PyErr_Occurred() ? -1 : 0;
}
static int attr_u64(PyObject *o, PyObject *name, uint64_t *out) {
    PyObject *v = PyObject_GetAttr(o, name);
    if (!v) return -1;
    const int rc = as_u64(v, out);
    Py_DECREF(v);
    return rc;
}
/* a Context's or a Weights' handle */
static int addr_of(PyObject *o, void **out) {
    uint64_t v;
    if (attr_u64(o, s_addr, &v)) return -1;
    *out = (void *)(uintptr_t)v;
    return 0;
}
static int ctx_of(PyObject *enc, okf_ctx **out) {
    PyObject *c = PyObject_GetAttr(enc, s_ctx);
    if (!c) return -1;
    const int rc = addr_of(c, (void **)out);
    Py_DECREF(c);
    return rc;
}
static int data_ptr(PyObject *t, void **out) {
    if (tensor_address_p && tensor_address_p(t, out)) return 0;
    PyObject *v = PyObject_CallMethodNoArgs(t, s_data_ptr);
    if (!v) return -1;
    uint64_t p;
    const int rc = as_u64(v, &p);
    Py_DECREF(v);
    *out = (void *)(uintptr_t)p;
    return rc;
}
static int dtype_of(PyObject *t, int *out) {
    if (tensor_dtype_p && tensor_dtype_p(t, out)) return 0;
    PyObject *d = PyObject_GetAttr(t, s_dtype);
    if (!d) return -1;
    int rc = 0;
    if (d == dt_f32) *out = OKF_F32;
    else if (d == dt_f16) *out = OKF_F16;
    else if (d == dt_bf16) *out = OKF_BF16;
    else {
        PyErr_SetObject(PyExc_KeyError, d);
        rc = -1;
    }
    Py_DECREF(d);
    return rc;
}
/* the encoder's stream, or the stream that is current on the current device */
static int stream_of(PyObject *enc, okf_stream *out) {
    PyObject *s = PyObject_GetAttr(enc, s_stream);
    if (!s) return -1;
    uint64_t v = 0;
    int rc;
    if (s == Py_None) {
        if (current_stream_p && current_stream_p(out)) {
            Py_DECREF(s);
            return 0;
        }
        rc = -1;
        PyObject *dev = PyObject_CallNoArgs(get_device_p);
        if (dev) {
            PyObject *raw = PyObject_CallOneArg(raw_stream_p, dev);
            Py_DECREF(dev);
            if (raw) {
                rc = as_u64(raw, &v);
                Py_DECREF(raw);
            }
        }
    } else {
        rc = attr_u64(s, s_cuda_stream, &v);
    }
    Py_DECREF(s);
    *out = (okf_stream)(uintptr_t)v;
    return rc;
}
/* a GGUFTensor: dims[0] = K, dims[1] = M (1 if there is no such axis) */
typedef struct { int type; uint32_t k, m; uint64_t off; } tensor_t;
static int tensor_of(PyObject *w, tensor_t *t) {
    uint64_t v;
    if (attr_u64(w, s_type, &v)) return -1;
    t->type = (int)v;
    if (attr_u64(w, s_offset, &t->off)) return -1;
    PyObject *dims = PyObject_GetAttr(w, s_dims);
    if (!dims) return -1;
    int rc = -1;
    const Py_ssize_t nd = PySequence_Size(dims);
    PyObject *d0 = nd < 0 ? NULL : PySequence_GetItem(dims, 0);
    if (d0 && !as_u64(d0, &v)) {
        t->k = (uint32_t)v;
        t->m = 1;
        rc = 0;
        if (nd > 1) {
            PyObject *d1 = PySequence_GetItem(dims, 1);
            rc = d1 ? as_u64(d1, &v) : -1;
            t->m = (uint32_t)v;
            Py_XDECREF(d1);
        }
    }
    Py_XDECREF(d0);
    Py_DECREF(dims);
    return rc;
}
static int args_are(Py_ssize_t n, Py_ssize_t want) {
    if (n == want) return 0;
    PyErr_Format(PyExc_TypeError, "%zd arguments expected, %zd given", want, n);
    return -1;
}

#define CALL(rc, call)                                 \
    do {                                               \
        Py_BEGIN_ALLOW_THREADS rc = (call);            \
        Py_END_ALLOW_THREADS                           \
    } while (0)

/* ---- the operators ----------------------------------------------------------------------- */

/* gemm(enc, which, w, X, out, off, N) */
static PyObject *py_gemm(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *off, *x, *out; okf_stream st; tensor_t t; uint64_t which, nn; int xdt, odt, rc;
    if (args_are(n, 7) || ctx_of(a[0], &ctx) || as_u64(a[1], &which) || tensor_of(a[2], &t) || data_ptr(a[3], &x) ||
        dtype_of(a[3], &xdt) || data_ptr(a[4], &out) || dtype_of(a[4], &odt) || addr_of(a[5], &off) || as_u64(a[6], &nn) ||
        stream_of(a[0], &st))
        return NULL;
    if (which >= FN_COUNT_GEMM) { PyErr_SetString(PyExc_ValueError, "no such entry point"); return NULL; }
    CALL(rc, gemm_fns[which](ctx, t.type, off, t.off, t.k, t.m, x, xdt, (uint32_t)nn, out, odt, st));
    return PyLong_FromLong(rc);
}
/* gemv(enc, w, x, out, off, x_off_bytes, out_off_bytes) */
static PyObject *py_gemv(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *off, *x, *out; okf_stream st; tensor_t t; uint64_t xo, oo; int xdt, rc;
    if (args_are(n, 7) || ctx_of(a[0], &ctx) || tensor_of(a[1], &t) || data_ptr(a[2], &x) || dtype_of(a[2], &xdt) ||
        data_ptr(a[3], &out) || addr_of(a[4], &off) || as_u64(a[5], &xo) || as_u64(a[6], &oo) || stream_of(a[0], &st))
        return NULL;
    CALL(rc, gemv_p(ctx, t.type, off, t.off, t.k, t.m, (uint8_t *)x + xo, xdt, (float *)((uint8_t *)out + oo), st));
    return PyLong_FromLong(rc);
}
/* parallel_begin(enc), parallel_end(enc) */
static PyObject *py_parallel_begin(PyObject *self, PyObject *enc) {
    okf_ctx *ctx;
    if (ctx_of(enc, &ctx)) return NULL;
    return PyLong_FromLong(parallel_begin_p(ctx));
}
static PyObject *py_parallel_end(PyObject *self, PyObject *enc) {
    okf_ctx *ctx; int rc;
    if (ctx_of(enc, &ctx)) return NULL;
    CALL(rc, parallel_end_p(ctx));
    return PyLong_FromLong(rc);
}
/* dequant(enc, off, out, n, type, weight_off, out_off_bytes) */
static PyObject *py_dequant(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *off, *out; okf_stream st; uint64_t cnt, ty, wo, oo; int rc;
    if (args_are(n, 7) || ctx_of(a[0], &ctx) || addr_of(a[1], &off) || data_ptr(a[2], &out) || as_u64(a[3], &cnt) ||
        as_u64(a[4], &ty) || as_u64(a[5], &wo) || as_u64(a[6], &oo) || stream_of(a[0], &st))
        return NULL;
    CALL(rc, dequant_p(ctx, (int)ty, off, wo, cnt, (float *)((uint8_t *)out + oo), st));
    return PyLong_FromLong(rc);
}
/* embed(enc, ids, off, out, n_embd, N, type, rows, weight_off) */
static PyObject *py_embed(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *ids, *off, *out; okf_stream st; uint64_t k, nn, ty, rows, wo; int rc;
    if (args_are(n, 9) || ctx_of(a[0], &ctx) || data_ptr(a[1], &ids) || addr_of(a[2], &off) || data_ptr(a[3], &out) ||
        as_u64(a[4], &k) || as_u64(a[5], &nn) || as_u64(a[6], &ty) || as_u64(a[7], &rows) || as_u64(a[8], &wo) ||
        stream_of(a[0], &st))
        return NULL;
    CALL(rc, embed_p(ctx, (int)ty, off, wo, (uint32_t)k, (uint32_t)rows, ids, (uint32_t)nn, out, st));
    return PyLong_FromLong(rc);
}
/* argmax(enc, x, out, n, rows) */
static PyObject *py_argmax(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *x, *out; okf_stream st; uint64_t len, rows; int rc;
    if (args_are(n, 5) || ctx_of(a[0], &ctx) || data_ptr(a[1], &x) || data_ptr(a[2], &out) || as_u64(a[3], &len) ||
        as_u64(a[4], &rows) || stream_of(a[0], &st))
        return NULL;
    CALL(rc, argmax_p(ctx, x, (uint32_t)len, (uint32_t)rows, out, st));
    return PyLong_FromLong(rc);
}
/* norm(enc, x, r or None, weight, y, n, rows, eps, x_stride, y_stride) */
static PyObject *py_norm(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *x, *r = NULL, *w, *y; okf_stream st; uint64_t len, rows, xs, ys; int rc;
    if (args_are(n, 10) || ctx_of(a[0], &ctx) || data_ptr(a[1], &x) || (a[2] != Py_None && data_ptr(a[2], &r)) ||
        data_ptr(a[3], &w) || data_ptr(a[4], &y) || as_u64(a[5], &len) || as_u64(a[6], &rows) || as_u64(a[8], &xs) ||
        as_u64(a[9], &ys) || stream_of(a[0], &st))
        return NULL;
    const double eps = PyFloat_AsDouble(a[7]);
    if (eps == -1.0 && PyErr_Occurred()) return NULL;
    CALL(rc, norm_p(ctx, x, r, w, y, (uint32_t)len, (uint32_t)rows, (float)eps, (uint32_t)xs, (uint32_t)ys, st));
    return PyLong_FromLong(rc);
}
/* silu(enc, a, b, n) */
static PyObject *py_silu(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *x, *y; okf_stream st; uint64_t len; int rc;
    if (args_are(n, 4) || ctx_of(a[0], &ctx) || data_ptr(a[1], &x) || data_ptr(a[2], &y) || as_u64(a[3], &len) ||
        stream_of(a[0], &st))
        return NULL;
    CALL(rc, silu_p(ctx, x, y, (size_t)len, st));
    return PyLong_FromLong(rc);
}
/* matmul_at(ctx, w, off, x_addr, N, out_addr): raw host addresses */
static PyObject *py_matmul_at(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *off; tensor_t t; uint64_t x, nn, out; int rc;
    if (args_are(n, 6) || addr_of(a[0], (void **)&ctx) || tensor_of(a[1], &t) || addr_of(a[2], &off) || as_u64(a[3], &x) ||
        as_u64(a[4], &nn) || as_u64(a[5], &out))
        return NULL;
    CALL(rc, matmul_host_p(ctx, t.type, off, t.off, t.k, t.m, (const float *)(uintptr_t)x, (uint32_t)nn, (float *)(uintptr_t)out));
    return PyLong_FromLong(rc);
}
static int floats(PyObject *o, Py_buffer *b, int flags) {
    if (PyObject_GetBuffer(o, b, flags | PyBUF_FORMAT | PyBUF_C_CONTIGUOUS)) {
        PyErr_Clear();
        return 0;
    }
    if (b->itemsize == 4 && b->format && !strcmp(b->format, "f")) return 1;
    PyBuffer_Release(b);
    return 0;
}
/* matmul_host(ctx, w, off, X, N, out) on arrays; None when X or out is no C-contiguous float32 array */
static PyObject *py_matmul_host(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    okf_ctx *ctx; void *off; tensor_t t; uint64_t nn; int rc;
    if (args_are(n, 6) || addr_of(a[0], (void **)&ctx) || tensor_of(a[1], &t) || addr_of(a[2], &off) || as_u64(a[4], &nn))
        return NULL;
    Py_buffer x, out;
    if (!floats(a[3], &x, 0)) Py_RETURN_NONE;
    if (!floats(a[5], &out, PyBUF_WRITABLE)) {
        PyBuffer_Release(&x);
        Py_RETURN_NONE;
    }
    PyObject *got = NULL;
    if ((uint64_t)x.len != nn * t.k * 4 || (uint64_t)out.len != nn * t.m * 4) {
        PyErr_SetString(PyExc_AssertionError, "X holds N x K and out N x M floats");
    } else {
        CALL(rc, matmul_host_p(ctx, t.type, off, t.off, t.k, t.m, x.buf, (uint32_t)nn, out.buf));
        got = PyLong_FromLong(rc);
    }
    PyBuffer_Release(&x);
    PyBuffer_Release(&out);
    return got;
}

/* bind(addresses: dict of name -> int, (float32, float16, bfloat16), get_device, raw_stream, (okf_pytensor.cpp's three addresses) or None) */
static int resolve(PyObject *d, const char *name, void *slot) {
    PyObject *v = PyDict_GetItemString(d, name);
    uint64_t p;
    if (!v) {
        PyErr_SetString(PyExc_KeyError, name);
        return -1;
    }
    if (as_u64(v, &p)) return -1;
    *(void **)slot = (void *)(uintptr_t)p;
    return 0;
}
static PyObject *py_bind(PyObject *self, PyObject *args) {
    PyObject *d, *f32, *f16, *bf16, *dev, *raw, *direct;
    unsigned long long at[3] = {0, 0, 0};
    if (!PyArg_ParseTuple(args, "O!(OOO)OOO", &PyDict_Type, &d, &f32, &f16, &bf16, &dev, &raw, &direct)) return NULL;
    if (direct != Py_None && !PyArg_ParseTuple(direct, "KKK", &at[0], &at[1], &at[2])) return NULL;
    if (resolve(d, "okf_gemm", &gemm_fns[FN_GEMM]) || resolve(d, "okf_gemm_tile", &gemm_fns[FN_GEMM_TILE]) ||
        resolve(d, "okf_gemm_noalloc", &gemm_fns[FN_GEMM_NOALLOC]) || resolve(d, "okf_gemv", &gemv_p) ||
        resolve(d, "okf_parallel_begin", &parallel_begin_p) || resolve(d, "okf_parallel_end", &parallel_end_p) ||
        resolve(d, "okf_dequant", &dequant_p) || resolve(d, "okf_embed_batch", &embed_p) ||
        resolve(d, "okf_argmax_rows", &argmax_p) || resolve(d, "okf_add_rmsnorm", &norm_p) ||
        resolve(d, "okf_silu_mul", &silu_p) || resolve(d, "okf_matmul_host", &matmul_host_p))
        return NULL;
    dt_f32 = Py_NewRef(f32);
    dt_f16 = Py_NewRef(f16);
    dt_bf16 = Py_NewRef(bf16);
    get_device_p = Py_NewRef(dev);
    raw_stream_p = Py_NewRef(raw);
    tensor_address_p = (int (*)(PyObject *, void **))(uintptr_t)at[0];
    tensor_dtype_p = (int (*)(PyObject *, int *))(uintptr_t)at[1];
    current_stream_p = (int (*)(void **))(uintptr_t)at[2];
    Py_RETURN_NONE;
}

#define FAST(f) (PyCFunction)(void (*)(void))(f), METH_FASTCALL, NULL
static PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, NULL},
    {"gemm", FAST(py_gemm)},
    {"gemv", FAST(py_gemv)},
    {"parallel_begin", py_parallel_begin, METH_O, NULL},
    {"parallel_end", py_parallel_end, METH_O, NULL},
    {"dequant", FAST(py_dequant)},
    {"embed", FAST(py_embed)},
    {"argmax", FAST(py_argmax)},
    {"norm", FAST(py_norm)},
    {"silu", FAST(py_silu)},
    {"matmul_at", FAST(py_matmul_at)},
    {"matmul_host", FAST(py_matmul_host)},
    {NULL, NULL, 0, NULL},
};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_okfcall", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__okfcall(void) {
    static const struct { PyObject **slot; const char *name; } names[] = {
        {&s_ctx, "ctx"}, {&s_addr, "_addr"}, {&s_stream, "stream"}, {&s_cuda_stream, "cuda_stream"}, {&s_type, "type"},
        {&s_dims, "dims"}, {&s_offset, "offset"}, {&s_dtype, "dtype"}, {&s_data_ptr, "data_ptr"},
    };
    for (size_t i = 0; i < sizeof(names) / sizeof(names[0]); i++)
        if (!(*names[i].slot = PyUnicode_InternFromString(names[i].name))) return NULL;
    return PyModule_Create(&module);
}
