/* The per-call half of muser_b200/operator.py in C: tensors, handles and Python numbers -> one call of the C ABI.
 *
 * A decode step of a small layer is ten calls of kernels that take 2 to 6 us, and the host took 6.8 us to make each: about
 * 3 in the launch, 1 to 1.6 in ctypes' argument conversion, 1 in building an epilogue structure, 1.2 in
 * torch.cuda.current_stream().  Here a call costs some tenths of a microsecond besides the launch.  Nothing is kept between
 * calls: addresses, dtypes and the stream are asked for every time, and the library is entered without the GIL, as ctypes
 * does it.  What ctypes refuses with ArgumentError is refused with it here.  muser_b200/_call_py.py is the same over ctypes.
 */
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>
#include <string.h>

#include "../../include/muser_cuda.h"

static struct {
    PyObject *dtypes;      /* torch.dtype -> MUSER_DTYPE_* */
    PyObject *f32;         /* torch.float32 */
    PyObject *raw_stream;  /* device -> the thread's current stream as an int; needs an initialized torch.cuda */
    PyObject *stream;      /* the same through torch.cuda, which initializes it */
    PyObject *error;       /* MuserCudaError */
    PyObject *argument_error;
    int stream_ready;
} g;
static PyObject *s_data_ptr, *s_dtype, *s_value, *s_handle;
static PyObject *s_keys[7]; /* row_scale, residual, norm_weight, norm_eps, out_scale, softcap, all_reduce */

static __typeof__(&muser_cuda_quantized_matmul) f_matmul;
static __typeof__(&muser_cuda_quantized_matmul_group) f_group;
static __typeof__(&muser_cuda_ffn_gate_up_silu) f_gate_up;
static __typeof__(&muser_cuda_nvfp4_matmul) f_nv_matmul;
static __typeof__(&muser_cuda_nvfp4_matmul_prequant) f_nv_prequant;
static __typeof__(&muser_cuda_nvfp4_matmul_group_prequant) f_nv_group;
static __typeof__(&muser_cuda_nvfp4_ffn_gate_up_silu_requant) f_nv_requant;
static __typeof__(&muser_cuda_quantize_nvfp4_activation) f_quantize;
static __typeof__(&muser_cuda_rmsnorm_quantize_nvfp4_activation) f_norm_quantize;
static __typeof__(&muser_cuda_fused_norm_residual_rms_norm) f_norm_residual;
static __typeof__(&muser_cuda_sigmoid_gate) f_sigmoid;
static __typeof__(&muser_cuda_head_rms_norm) f_head_norm;

/* ---- conversions: 0 on success, -1 with an exception set ---- */
static int refuse(const char *what, PyObject *o) {
    PyErr_Clear();
    PyErr_Format(g.argument_error, "%s expected instead of %s instance", what, Py_TYPE(o)->tp_name);
    return -1;
}
static int to_u64(PyObject *o, uint64_t *out) {
    if (!PyLong_Check(o)) return refuse("int", o);
    *out = PyLong_AsUnsignedLongLongMask(o);
    return 0;
}
static int to_u32(PyObject *o, uint32_t *out) {
    uint64_t v;
    if (to_u64(o, &v)) return -1;
    *out = (uint32_t)v;
    return 0;
}
static int to_f32(PyObject *o, float *out) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return refuse("real number", o);
    *out = (float)v;
    return 0;
}
/* what c_float(o) gives, for the arguments that the interface wraps so: TypeError, not ArgumentError, where it is no number */
static int to_c_float(PyObject *o, float *out) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) return -1;
    *out = (float)v;
    return 0;
}
/* what float(o) gives, for the arguments that the interface converts itself */
static int to_float(PyObject *o, float *out) {
    double v;
    if (PyFloat_CheckExact(o)) {
        v = PyFloat_AS_DOUBLE(o);
    } else {
        PyObject *f = PyNumber_Float(o);
        if (!f) return -1;
        v = PyFloat_AS_DOUBLE(f);
        Py_DECREF(f);
    }
    *out = (float)v;
    return 0;
}
static int as_address(PyObject *v, void **out) { /* steals v */
    if (!v) return -1;
    if (v == Py_None) {
        *out = NULL;
    } else if (!PyLong_Check(v)) {
        refuse("int", v);
        Py_DECREF(v);
        return -1;
    } else {
        *out = (void *)(uintptr_t)PyLong_AsUnsignedLongLongMask(v);
    }
    Py_DECREF(v);
    return 0;
}
static int to_ptr(PyObject *tensor, void **out) { return as_address(PyObject_CallMethodNoArgs(tensor, s_data_ptr), out); }
static int to_ptr_or_null(PyObject *tensor, void **out) {
    if (tensor == Py_None) {
        *out = NULL;
        return 0;
    }
    return to_ptr(tensor, out);
}
static int to_handle(PyObject *owner, void *out) { /* Context or Weight: its ._h, a c_void_p, or None once it is freed */
    PyObject *h = PyObject_GetAttr(owner, s_handle);
    if (!h) return -1;
    if (h == Py_None) {
        Py_DECREF(h);
        *(void **)out = NULL;
        return 0;
    }
    PyObject *v = PyObject_GetAttr(h, s_value);
    Py_DECREF(h);
    return as_address(v, (void **)out);
}
static int to_dtype(PyObject *tensor, uint32_t *out) {
    PyObject *d = PyObject_GetAttr(tensor, s_dtype);
    if (!d) return -1;
    PyObject *code = PyDict_GetItemWithError(g.dtypes, d);
    if (!code && !PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, d);
    Py_DECREF(d);
    return code ? to_u32(code, out) : -1;
}
static int to_stream(PyObject *device, void **out) {
    PyObject *v = PyObject_CallOneArg(g.stream_ready ? g.raw_stream : g.stream, device);
    if (v && !g.stream_ready) g.stream_ready = 1;
    return as_address(v, out);
}
static int fail_f32(void) {
    PyObject *e = PyObject_CallFunction(g.error, "is", 1, "norm_weight must be f32");
    if (e) PyErr_SetObject(g.error, e);
    Py_XDECREF(e);
    return -1;
}

/* operator._epilogue: *used says whether the call needs the structure at all */
static int to_epilogue(PyObject *row_scale, PyObject *residual, PyObject *norm_weight, PyObject *norm_eps, PyObject *out_scale, PyObject *softcap,
                       PyObject *all_reduce, muser_cuda_epilogue *ep, int *used) {
    const int reduce = all_reduce ? PyObject_IsTrue(all_reduce) : 0;
    void *p[3] = {NULL, NULL, NULL};
    if (reduce < 0) return -1;
    memset(ep, 0, sizeof(*ep));
    ep->out_scale = 1.0f;
    if ((out_scale && to_float(out_scale, &ep->out_scale)) || (softcap && to_float(softcap, &ep->softcap))) return -1;
    *used = row_scale != Py_None || residual != Py_None || norm_weight != Py_None || ep->out_scale != 1.0f || ep->softcap != 0.0f || reduce;
    if (!*used) return 0;
    if (norm_weight != Py_None) {
        PyObject *d = PyObject_GetAttr(norm_weight, s_dtype);
        if (!d) return -1;
        Py_DECREF(d);
        if (d != g.f32) return fail_f32(); /* (dtypes are singletons) */
    }
    if (to_ptr_or_null(row_scale, &p[0]) || to_ptr_or_null(residual, &p[1]) || (norm_eps && to_float(norm_eps, &ep->norm_eps)) || to_ptr_or_null(norm_weight, &p[2]))
        return -1;
    ep->row_scale = p[0], ep->residual = p[1], ep->norm_weight = p[2], ep->all_reduce = (uint32_t)reduce;
    return 0;
}

#define ARGS(n)                                                                                                  \
    if (argc != (n)) {                                                                                           \
        PyErr_Format(PyExc_TypeError, "%d arguments expected, %zd given", (n), argc);                            \
        return NULL;                                                                                             \
    }
#define CALL(...)                                                                                                \
    int st;                                                                                                      \
    Py_BEGIN_ALLOW_THREADS st = (int)(__VA_ARGS__);                                                              \
    Py_END_ALLOW_THREADS return PyLong_FromLong(st)

/* (ctx, device, weight, x, y, tokens, row_scale, residual, norm_weight, norm_eps, out_scale, softcap[, all_reduce]) */
static PyObject *matmul(PyObject *const *a, Py_ssize_t argc, int nvfp4) {
    void *ctx, *w, *x, *y, *stream;
    uint32_t xd, yd, tokens;
    muser_cuda_epilogue ep;
    int used;
    ARGS(nvfp4 ? 12 : 13)
    if (to_epilogue(a[6], a[7], a[8], a[9], a[10], a[11], nvfp4 ? NULL : a[12], &ep, &used) || to_handle(a[0], &ctx) || to_handle(a[2], &w) ||
        to_ptr(a[3], &x) || to_dtype(a[3], &xd) || to_ptr(a[4], &y) || to_dtype(a[4], &yd) || to_u32(a[5], &tokens) || to_stream(a[1], &stream))
        return NULL;
    CALL(nvfp4 ? f_nv_matmul(ctx, w, x, xd, y, yd, tokens, used ? &ep : NULL, stream) : f_matmul(ctx, w, x, xd, y, yd, tokens, used ? &ep : NULL, stream));
}
static PyObject *quantized_matmul(PyObject *self, PyObject *const *a, Py_ssize_t argc) { return matmul(a, argc, 0); }
static PyObject *nvfp4_matmul(PyObject *self, PyObject *const *a, Py_ssize_t argc) { return matmul(a, argc, 1); }

static int epilogue_of_dict(PyObject *dict, muser_cuda_epilogue *ep, int *used) {
    PyObject *v[7];
    Py_ssize_t found = 0;
    for (int i = 0; i < 7; ++i) {
        v[i] = PyDict_GetItemWithError(dict, s_keys[i]);
        if (!v[i] && PyErr_Occurred()) return -1;
        found += v[i] != NULL;
        if (!v[i] && i < 3) v[i] = Py_None;
    }
    if (found != PyDict_GET_SIZE(dict)) {
        PyErr_SetString(PyExc_TypeError, "_epilogue() got an unexpected keyword argument");
        return -1;
    }
    return to_epilogue(v[0], v[1], v[2], v[3], v[4], v[5], v[6], ep, used);
}
/* (ctx, device, weights, x, outputs, tokens, epilogues): weights as len() and iteration give them, outputs any iterable; epilogues
 * None or epilogues[i], a mapping of keywords or None each */
static int epilogue_of(PyObject *given_as, muser_cuda_epilogue *ep, int *used) {
    const int given = given_as != Py_None ? PyObject_IsTrue(given_as) : 0;
    if (given < 0) return -1;
    *used = 0;
    if (!given) return 0;
    if (PyDict_Check(given_as)) return epilogue_of_dict(given_as, ep, used);
    PyObject *dict = PyDict_New(); /* (lives until the tensors' addresses are read, as they do) */
    int st = dict ? PyDict_Update(dict, given_as) : -1;
    if (st && PyErr_ExceptionMatches(PyExc_AttributeError)) /* it has no keys() */
        PyErr_Format(PyExc_TypeError, "an epilogue is a mapping or None, not %s", Py_TYPE(given_as)->tp_name);
    if (!st) st = epilogue_of_dict(dict, ep, used);
    Py_XDECREF(dict);
    return st;
}
static PyObject *quantized_matmul_group(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    enum { kMost = 16 }; /* (the library takes four; longer lists are its to refuse) */
    muser_cuda_group_item items[kMost];
    muser_cuda_epilogue eps[kMost];
    void *ctx, *x, *stream;
    uint32_t xd, tokens;
    ARGS(7)
    PyObject *ws = PyObject_Size(a[2]) < 0 ? NULL : PySequence_Fast(a[2], "weights must be a sequence");
    PyObject *ys = ws ? PySequence_Fast(a[4], "outputs must be a sequence") : NULL;
    const int given = ys && a[6] != Py_None ? PyObject_IsTrue(a[6]) : 0;
    const Py_ssize_t n = ws ? PySequence_Fast_GET_SIZE(ws) : 0;
    int ok = ws && ys && given >= 0;
    memset(items, 0, sizeof(items));
    for (Py_ssize_t i = 0; ok && i < n && i < kMost && i < PySequence_Fast_GET_SIZE(ys); ++i) {
        int used = 0;
        PyObject *y = PySequence_Fast_GET_ITEM(ys, i);
        void *w, *yp;
        if (given) {
            PyObject *at = PyLong_FromSsize_t(i), *e = at ? PyObject_GetItem(a[6], at) : NULL;
            ok = e && !epilogue_of(e, &eps[i], &used);
            Py_XDECREF(at);
            Py_XDECREF(e);
        }
        ok = ok && !to_handle(PySequence_Fast_GET_ITEM(ws, i), &w) && !to_ptr(y, &yp) &&
             !to_dtype(y, &items[i].y_dtype);
        if (!ok) break;
        items[i].w = w, items[i].y = yp, items[i].epilogue = used ? &eps[i] : NULL;
    }
    Py_XDECREF(ws);
    Py_XDECREF(ys);
    if (!ok || to_handle(a[0], &ctx) || to_ptr(a[3], &x) || to_dtype(a[3], &xd) || to_u32(a[5], &tokens) || to_stream(a[1], &stream)) return NULL;
    CALL(f_group(ctx, items, (uint32_t)n, x, xd, tokens, stream));
}

/* (ctx, device, gate, up, x, y, tokens, norm_weight, norm_eps) */
static PyObject *gate_up_silu(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    void *ctx, *gate, *up, *x, *y, *stream;
    uint32_t xd, yd, tokens;
    muser_cuda_epilogue ep;
    int used;
    ARGS(9)
    if (to_epilogue(Py_None, Py_None, a[7], a[8], NULL, NULL, NULL, &ep, &used) || to_handle(a[0], &ctx) || to_handle(a[2], &gate) || to_handle(a[3], &up) ||
        to_ptr(a[4], &x) || to_dtype(a[4], &xd) || to_ptr(a[5], &y) || to_dtype(a[5], &yd) || to_u32(a[6], &tokens) || to_stream(a[1], &stream))
        return NULL;
    CALL(f_gate_up(ctx, gate, up, x, xd, y, yd, tokens, used ? &ep : NULL, stream));
}

/* (ctx, device, weight, packed, scales, y, tokens, row_scale, residual) */
static PyObject *nvfp4_prequant(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    void *ctx, *w, *packed, *scales, *y, *stream;
    uint32_t yd, tokens;
    muser_cuda_epilogue ep;
    int used;
    ARGS(9)
    if (to_epilogue(a[7], a[8], Py_None, NULL, NULL, NULL, NULL, &ep, &used) || to_handle(a[0], &ctx) || to_handle(a[2], &w) || to_ptr(a[3], &packed) ||
        to_ptr(a[4], &scales) || to_ptr(a[5], &y) || to_dtype(a[5], &yd) || to_u32(a[6], &tokens) || to_stream(a[1], &stream))
        return NULL;
    CALL(f_nv_prequant(ctx, w, packed, scales, y, yd, tokens, used ? &ep : NULL, stream));
}

/* (ctx, device, weights, packed, scales, outputs, tokens) */
static PyObject *nvfp4_group_prequant(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    enum { kMost = 16 };
    const muser_cuda_weight *w[kMost] = {NULL};
    void *y[kMost] = {NULL}, *ctx, *packed, *scales, *stream;
    uint32_t yd = 0, tokens;
    ARGS(7)
    PyObject *ws = PyObject_Size(a[2]) < 0 ? NULL : PySequence_Fast(a[2], "weights must be a sequence");
    PyObject *ys = ws && !PySequence_Check(a[5]) ? PyErr_Format(PyExc_TypeError, "'%s' object is not subscriptable", Py_TYPE(a[5])->tp_name)
                   : ws                          ? PySequence_Fast(a[5], "outputs must be a sequence")
                                                 : NULL;
    const Py_ssize_t n = ws ? PySequence_Fast_GET_SIZE(ws) : 0, n_y = ys ? PySequence_Fast_GET_SIZE(ys) : 0;
    int ok = ys != NULL;
    if (ok && (n_y == 0 || n_y > n)) {
        PyErr_SetString(PyExc_IndexError, n_y ? "invalid index" : "list index out of range");
        ok = 0;
    }
    for (Py_ssize_t i = 0; ok && i < n && i < kMost; ++i) ok = !to_handle(PySequence_Fast_GET_ITEM(ws, i), &w[i]);
    for (Py_ssize_t i = 0; ok && i < n_y && i < kMost; ++i) ok = !to_ptr(PySequence_Fast_GET_ITEM(ys, i), &y[i]);
    ok = ok && !to_dtype(PySequence_Fast_GET_ITEM(ys, 0), &yd);
    Py_XDECREF(ws);
    Py_XDECREF(ys);
    if (!ok || to_handle(a[0], &ctx) || to_ptr(a[3], &packed) || to_ptr(a[4], &scales) || to_u32(a[6], &tokens) || to_stream(a[1], &stream)) return NULL;
    CALL(f_nv_group(ctx, w, (uint32_t)n, packed, scales, y, yd, tokens, stream));
}

/* (ctx, device, gate, up, packed, scales, tokens, out_input_scale_inv, out_packed, out_scales) */
static PyObject *nvfp4_gate_up_requant(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    void *ctx, *gate, *up, *packed, *scales, *op, *os, *stream;
    uint32_t tokens;
    float isi;
    ARGS(10)
    if (to_handle(a[0], &ctx) || to_handle(a[2], &gate) || to_handle(a[3], &up) || to_ptr(a[4], &packed) || to_ptr(a[5], &scales) || to_u32(a[6], &tokens) ||
        to_c_float(a[7], &isi) || to_ptr(a[8], &op) || to_ptr(a[9], &os) || to_stream(a[1], &stream))
        return NULL;
    CALL(f_nv_requant(ctx, gate, up, packed, scales, tokens, isi, op, os, stream));
}

/* (ctx, device, x, tokens, n_in, input_scale_inv, norm_weight, norm_eps, packed, scales) */
static PyObject *quantize_activation(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    void *ctx, *x, *nw, *packed, *scales, *stream;
    uint32_t xd, tokens;
    uint64_t n_in;
    float isi, eps = 0.0f;
    ARGS(10)
    if (to_handle(a[0], &ctx) || to_ptr(a[2], &x) || to_dtype(a[2], &xd) || to_u32(a[3], &tokens) || to_u64(a[4], &n_in) || to_f32(a[5], &isi) ||
        to_ptr_or_null(a[6], &nw) || (a[6] != Py_None && to_float(a[7], &eps)) || to_ptr(a[8], &packed) || to_ptr(a[9], &scales) || to_stream(a[1], &stream))
        return NULL;
    CALL(a[6] != Py_None ? f_norm_quantize(ctx, x, xd, tokens, n_in, nw, eps, isi, packed, scales, stream)
                         : f_quantize(ctx, x, xd, tokens, n_in, isi, packed, scales, stream));
}

/* (ctx, device, hidden, src, output, weight1, weight2, tokens, n, eps1, eps2) */
static PyObject *norm_residual_norm(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    void *ctx, *hidden, *src, *out, *w1, *w2, *stream;
    uint32_t tokens, n;
    float eps1, eps2;
    ARGS(11)
    if (to_handle(a[0], &ctx) || to_ptr(a[2], &hidden) || to_ptr(a[3], &src) || to_ptr_or_null(a[4], &out) || to_ptr(a[5], &w1) || to_ptr_or_null(a[6], &w2) ||
        to_u32(a[7], &tokens) || to_u32(a[8], &n) || to_c_float(a[9], &eps1) || to_c_float(a[10], &eps2) || to_stream(a[1], &stream))
        return NULL;
    CALL(f_norm_residual(ctx, hidden, src, out, w1, w2, tokens, n, eps1, eps2, stream));
}

/* (ctx, device, x, gate, count) */
static PyObject *sigmoid_gate(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    void *ctx, *x, *gate, *stream;
    uint64_t count;
    ARGS(5)
    if (to_handle(a[0], &ctx) || to_ptr(a[2], &x) || to_ptr(a[3], &gate) || to_u64(a[4], &count) || to_stream(a[1], &stream)) return NULL;
    CALL(f_sigmoid(ctx, x, gate, count, stream));
}

/* (ctx, device, x, weight, eps, tokens, heads, head_dim) */
static PyObject *head_rms_norm(PyObject *self, PyObject *const *a, Py_ssize_t argc) {
    void *ctx, *x, *w, *stream;
    uint32_t tokens, heads, head_dim;
    float eps;
    ARGS(8)
    if (to_handle(a[0], &ctx) || to_ptr(a[2], &x) || to_ptr(a[3], &w) || to_c_float(a[4], &eps) || to_u32(a[5], &tokens) || to_u32(a[6], &heads) ||
        to_u32(a[7], &head_dim) || to_stream(a[1], &stream))
        return NULL;
    CALL(f_head_norm(ctx, x, w, eps, tokens, heads, head_dim, stream));
}

/* bind(library path, dtypes, torch.float32, raw_stream, stream, MuserCudaError, ArgumentError) */
static PyObject *bind(PyObject *self, PyObject *args) {
    const char *path;
    PyObject *o[6];
    if (!PyArg_ParseTuple(args, "sO!OOOOO", &path, &PyDict_Type, &o[0], &o[1], &o[2], &o[3], &o[4], &o[5])) return NULL;
    void *lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (!lib) {
        PyErr_SetString(PyExc_ImportError, dlerror());
        return NULL;
    }
    const struct {
        const char *name;
        void *slot;
    } want[] = {{"muser_cuda_quantized_matmul", &f_matmul}, {"muser_cuda_quantized_matmul_group", &f_group}, {"muser_cuda_ffn_gate_up_silu", &f_gate_up},
                {"muser_cuda_nvfp4_matmul", &f_nv_matmul}, {"muser_cuda_nvfp4_matmul_prequant", &f_nv_prequant},
                {"muser_cuda_nvfp4_matmul_group_prequant", &f_nv_group}, {"muser_cuda_nvfp4_ffn_gate_up_silu_requant", &f_nv_requant},
                {"muser_cuda_quantize_nvfp4_activation", &f_quantize}, {"muser_cuda_rmsnorm_quantize_nvfp4_activation", &f_norm_quantize},
                {"muser_cuda_fused_norm_residual_rms_norm", &f_norm_residual}, {"muser_cuda_sigmoid_gate", &f_sigmoid},
                {"muser_cuda_head_rms_norm", &f_head_norm}};
    for (size_t i = 0; i < sizeof(want) / sizeof(want[0]); ++i) {
        void *p = dlsym(lib, want[i].name);
        if (!p) {
            PyErr_Format(PyExc_ImportError, "%s lacks %s", path, want[i].name);
            return NULL;
        }
        memcpy(want[i].slot, &p, sizeof(p));
    }
    PyObject **slots[6] = {&g.dtypes, &g.f32, &g.raw_stream, &g.stream, &g.error, &g.argument_error};
    for (int i = 0; i < 6; ++i) {
        Py_INCREF(o[i]);
        Py_XSETREF(*slots[i], o[i]);
    }
    g.stream_ready = 0;
    Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, NULL}, FAST(quantized_matmul), FAST(nvfp4_matmul), FAST(quantized_matmul_group), FAST(gate_up_silu),
                                FAST(nvfp4_prequant), FAST(nvfp4_group_prequant), FAST(nvfp4_gate_up_requant), FAST(quantize_activation),
                                FAST(norm_residual_norm), FAST(sigmoid_gate), FAST(head_rms_norm), {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_call", NULL, -1, methods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__call(void) {
    static const char *keys[7] = {"row_scale", "residual", "norm_weight", "norm_eps", "out_scale", "softcap", "all_reduce"};
    for (int i = 0; i < 7; ++i)
        if (!(s_keys[i] = PyUnicode_InternFromString(keys[i]))) return NULL;
    if (!(s_data_ptr = PyUnicode_InternFromString("data_ptr")) || !(s_dtype = PyUnicode_InternFromString("dtype")) ||
        !(s_value = PyUnicode_InternFromString("value")) || !(s_handle = PyUnicode_InternFromString("_h")))
        return NULL;
    return PyModule_Create(&module);
}
