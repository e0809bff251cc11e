// CPython side of the binding: the calls a program makes many times per step, without the
// interpreter work of the ctypes path.
//
// What bounds a small call is the host: one launch costs the CUDA runtime 2.3 us, and the Python code
// around it (torch.cuda.current_stream() 3.0 us, building a descriptor 4.2 us, a ctypes call 0.8 us) cost
// more than that.  Each function here takes the arguments of the Python function of the same name in
// llmt_b200/__init__.py, and handles the ordinary case; whatever it does not recognise (a wrong type,
// shape or rank, an unknown keyword) it hands to that Python function, which holds the checks and the
// messages.  Both fill in the same descriptor and call the same C entry point.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include "../../include/llmt_b200.h"

// The entry points of the loaded library (bind() fills them in, in the order of kNames).
typedef struct {
    int (*gemm)(const llmt_b200_gemm_desc*, void*, const void*, const void*, void*);
    uint64_t (*gemm_workspace_bytes_for)(const llmt_b200_gemm_desc*, const void*, const void*);
    int (*gemm_grouped)(const llmt_b200_gemm_desc*, void* const*, const void* const*, const void* const*, int32_t, void*);
    int (*zero_grads)(float*, int64_t, void*);
    int (*softmax_fwd)(void*, const void*, int64_t, int64_t, int64_t, int32_t, int32_t, void*);
    int (*softmax_bwd)(void*, const void*, const void*, int64_t, int64_t, int32_t, void*);
    int (*gemm_softmax_fwd)(const llmt_b200_gemm_desc*, void*, const void*, const void*, int32_t, float*, void*);
    int (*gemm_softmax_bwd)(const llmt_b200_gemm_desc*, void*, const void*, const void*, const void*, const float*, int32_t, void*);
    int (*rowdot)(float*, const void*, const void*, int64_t, int64_t, int64_t, int64_t, int32_t, void*);
    int (*head_split)(void*, void*, void*, const void*, int64_t, int64_t, int64_t, int64_t, int32_t, void*);
    int (*head_merge)(void*, const void*, int64_t, int64_t, int64_t, int64_t, int32_t, void*);
    int (*cross_entropy_fwd)(float*, float*, const float*, const int32_t*, const float*, int64_t, int64_t, int64_t, void*);
    int (*cross_entropy_bwd)(float*, const float*, const int32_t*, const float*, float, int64_t, int64_t, int64_t, int64_t, void*);
    int (*lm_head_ce_fwd)(const llmt_b200_gemm_desc*, void*, const void*, const void*, const int32_t*, const float*, float*, float*, void*);
    int (*lm_head_ce_bwd)(const llmt_b200_gemm_desc*, void*, const void*, const void*, const int32_t*, const float*, float, int32_t, void*);
} Entry;
static const char* const kNames[] = {"gemm", "gemm_workspace_bytes_for", "gemm_grouped", "zero_grads", "softmax_fwd", "softmax_bwd",
                                     "gemm_softmax_fwd", "gemm_softmax_bwd", "rowdot", "head_split", "head_merge",
                                     "cross_entropy_fwd", "cross_entropy_bwd", "lm_head_ce_fwd", "lm_head_ce_bwd"};
#define N_ENTRIES ((Py_ssize_t)(sizeof(kNames) / sizeof(kNames[0])))
_Static_assert(sizeof(Entry) == sizeof(kNames), "one pointer per name");

static Entry E;
static int g_bound = 0;
static PyObject *g_binder, *g_raise, *g_scratch;            // Python: loads the library; raises for a status; allocates scratch
static PyObject *g_raw_stream, *g_get_device;               // torch's current stream handle of a device, and its current device
static PyObject *g_float32, *g_bfloat16, *g_int32;
static PyObject* g_desc_type;                               // the ctypes structure GemmDesc
static PyObject *s_data_ptr, *s_shape, *s_stride, *s_dtype, *s_cuda_stream, *s_nbytes;

static int ensure_bound(void) {
    if (g_bound) return 0;
    PyObject* r = PyObject_CallNoArgs(g_binder);
    if (r == NULL) return -1;
    Py_DECREF(r);
    return g_bound ? 0 : -1;
}

// Everything below returns 0 / a value on success; -1 means "not the ordinary case" WITHOUT an exception
// set (errors of the attribute lookups are cleared): the caller then takes the Python function.
typedef struct {
    void* ptr;
    int nd;
    int64_t shape[4], stride[4];
    int dtype;   // LLMT_B200_FP32 / _BF16, 2 = int32
} Tensor;

static int as_ptr(PyObject* o, void** out) {
    PyObject* v = PyObject_CallMethodNoArgs(o, s_data_ptr);
    if (v == NULL) { PyErr_Clear(); return -1; }
    *out = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    if (*out == NULL && PyErr_Occurred()) { PyErr_Clear(); return -1; }
    return 0;
}
static int as_optional_ptr(PyObject* o, void** out) {
    if (o == NULL || o == Py_None) { *out = NULL; return 0; }
    return as_ptr(o, out);
}
static int read_tuple(PyObject* t, int64_t* out, int most) {   // steals t
    if (t == NULL) { PyErr_Clear(); return -1; }
    int n = -1;
    if (PyTuple_Check(t) && PyTuple_GET_SIZE(t) <= most) {
        n = (int)PyTuple_GET_SIZE(t);
        for (int i = 0; i < n; ++i) {
            out[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(t, i));
            if (out[i] == -1 && PyErr_Occurred()) { PyErr_Clear(); n = -1; break; }
        }
    }
    Py_DECREF(t);
    return n;
}
static int as_tensor(PyObject* o, Tensor* t) {
    if (as_ptr(o, &t->ptr) < 0) return -1;
    t->nd = read_tuple(PyObject_GetAttr(o, s_shape), t->shape, 4);
    if (t->nd < 0 || read_tuple(PyObject_CallMethodNoArgs(o, s_stride), t->stride, 4) != t->nd) return -1;
    PyObject* d = PyObject_GetAttr(o, s_dtype);
    if (d == NULL) { PyErr_Clear(); return -1; }
    t->dtype = d == g_float32 ? LLMT_B200_FP32 : d == g_bfloat16 ? LLMT_B200_BF16 : d == g_int32 ? 2 : -1;
    Py_DECREF(d);
    return t->dtype < 0 ? -1 : 0;
}
static int is_contiguous(const Tensor* t) {
    int64_t want = 1;
    for (int i = t->nd - 1; i >= 0; --i) {
        if (t->shape[i] != 1 && t->stride[i] != want) return 0;
        want *= t->shape[i];
    }
    return 1;
}
static int64_t numel(const Tensor* t) {
    int64_t n = 1;
    for (int i = 0; i < t->nd; ++i) n *= t->shape[i];
    return n;
}
static int as_stream(PyObject* o, void** out) {
    PyObject* v;
    if (o == NULL || o == Py_None) {
        PyObject* dev = PyObject_CallNoArgs(g_get_device);
        if (dev == NULL) { PyErr_Clear(); return -1; }
        v = PyObject_CallOneArg(g_raw_stream, dev);
        Py_DECREF(dev);
    } else {
        v = PyObject_GetAttr(o, s_cuda_stream);
    }
    if (v == NULL) { PyErr_Clear(); return -1; }
    *out = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    if (*out == NULL && PyErr_Occurred()) { PyErr_Clear(); return -1; }
    return 0;
}
static int as_desc(PyObject* o, llmt_b200_gemm_desc* out) {   // a ctypes GemmDesc
    Py_buffer b;
    if (!PyObject_TypeCheck(o, (PyTypeObject*)g_desc_type)) return -1;
    if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) < 0) { PyErr_Clear(); return -1; }
    const int ok = b.len == (Py_ssize_t)sizeof *out;
    if (ok) memcpy(out, b.buf, sizeof *out);
    PyBuffer_Release(&b);
    return ok ? 0 : -1;
}
static int as_float(PyObject* o, float dflt, float* out) {
    if (o == NULL) { *out = dflt; return 0; }
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return -1; }
    *out = (float)v;
    return 0;
}
static int as_int(PyObject* o, int32_t* out) {
    if (o == NULL) { *out = 0; return 0; }
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return -1; }
    *out = (int32_t)v;
    return 0;
}
static int as_bool(PyObject* o, int32_t* out) {
    if (o == NULL) { *out = 0; return 0; }
    const int v = PyObject_IsTrue(o);
    if (v < 0) { PyErr_Clear(); return -1; }
    *out = v;
    return 0;
}

// Positional and keyword arguments into out[0 .. n-1] (NULL where absent); -1: not this function's.
static int arguments(PyObject* const* args, Py_ssize_t nargs, PyObject* kw, const char* const* names, int n, int required,
                     PyObject** out) {
    memset(out, 0, sizeof(PyObject*) * (size_t)n);
    if (nargs > n) return -1;
    for (Py_ssize_t i = 0; i < nargs; ++i) out[i] = args[i];
    const Py_ssize_t nkw = kw != NULL ? PyTuple_GET_SIZE(kw) : 0;
    for (Py_ssize_t i = 0; i < nkw; ++i) {
        PyObject* key = PyTuple_GET_ITEM(kw, i);
        int at = 0;
        while (at < n && PyUnicode_CompareWithASCIIString(key, names[at]) != 0) ++at;
        if (at == n || out[at] != NULL) return -1;
        out[at] = args[nargs + i];
    }
    for (int i = 0; i < required; ++i)
        if (out[i] == NULL) return -1;
    return 0;
}

static PyObject* finish(int status) {
    if (status == LLMT_B200_OK) Py_RETURN_NONE;
    PyObject* code = PyLong_FromLong(status);
    if (code == NULL) return NULL;
    PyObject* r = PyObject_CallOneArg(g_raise, code);   // raises LlmtB200Error
    Py_DECREF(code);
    return r;
}

// The library call itself runs without the interpreter lock, as a ctypes call does: a launch may wait for room in the queue.
#define RUN(call)                                                                    \
    do {                                                                             \
        int st;                                                                      \
        Py_BEGIN_ALLOW_THREADS                                                       \
        st = (call);                                                                 \
        Py_END_ALLOW_THREADS                                                         \
        return finish(st);                                                           \
    } while (0)
#define FAST(name) static PyObject* fast_##name(PyObject* slow, PyObject* const* args, Py_ssize_t nargs, PyObject* kw)
#define SLOW() return PyObject_Vectorcall(slow, args, (size_t)nargs, kw)
#define BEGIN(required, ...)                                                         \
    static const char* const names[] = {__VA_ARGS__};                                \
    enum { kN = sizeof(names) / sizeof(names[0]) };                                  \
    PyObject* v[kN];                                                                 \
    if (ensure_bound() < 0) return NULL;                                             \
    if (arguments(args, nargs, kw, names, kN, (required), v) < 0) SLOW()
#define NEED(cond) do { if (!(cond)) SLOW(); } while (0)

FAST(gemm_desc) {
    BEGIN(4, "desc", "c", "a", "b", "stream");
    llmt_b200_gemm_desc d;
    void *c, *a, *b, *s;
    NEED(as_desc(v[0], &d) == 0 && as_ptr(v[1], &c) == 0 && as_ptr(v[2], &a) == 0 && as_ptr(v[3], &b) == 0 && as_stream(v[4], &s) == 0);
    RUN(E.gemm(&d, c, a, b, s));
}

static int pitch_ok(const Tensor* t) { return t->stride[t->nd - 1] == 1 || t->shape[t->nd - 1] == 1; }

FAST(gemm) {
    BEGIN(3, "c", "a", "b", "trans_a", "trans_b", "alpha", "beta", "bias", "gelu", "dbias", "dbias_beta", "workspace", "stream",
          "tile_n", "splits", "cta_pairs");
    Tensor c, a, b;
    void* s;
    llmt_b200_gemm_desc d;
    memset(&d, 0, sizeof d);
    int32_t gelu;
    NEED(as_tensor(v[0], &c) == 0 && as_tensor(v[1], &a) == 0 && as_tensor(v[2], &b) == 0 && as_stream(v[12], &s) == 0);
    NEED(a.nd == b.nd && a.nd == c.nd && (a.nd == 2 || a.nd == 3) && a.dtype == b.dtype && a.dtype < 2 && c.dtype < 2);
    NEED(pitch_ok(&a) && pitch_ok(&b) && pitch_ok(&c));
    NEED(as_bool(v[3], &d.trans_a) == 0 && as_bool(v[4], &d.trans_b) == 0 && as_float(v[5], 1.0f, &d.alpha) == 0 &&
         as_float(v[6], 0.0f, &d.beta) == 0 && as_bool(v[8], &gelu) == 0 && as_float(v[10], 0.0f, &d.dbias_beta) == 0 &&
         as_int(v[13], &d.plan_tile_n) == 0 && as_int(v[14], &d.plan_splits) == 0 && as_int(v[15], &d.plan_cta_pairs) == 0);
    const int r = a.nd - 2;
    d.m = d.trans_a ? a.shape[r + 1] : a.shape[r];
    d.k = d.trans_a ? a.shape[r] : a.shape[r + 1];
    d.n = d.trans_b ? b.shape[r] : b.shape[r + 1];
    NEED((d.trans_b ? b.shape[r + 1] : b.shape[r]) == d.k && c.shape[r] == d.m && c.shape[r + 1] == d.n);
    d.batch = 1;
    if (r) {
        d.batch = a.shape[0];
        NEED(b.shape[0] == d.batch && c.shape[0] == d.batch);
        d.stride_a = a.stride[0]; d.stride_b = b.stride[0]; d.stride_c = c.stride[0];
    }
    d.lda = a.stride[r]; d.ldb = b.stride[r]; d.ldc = c.stride[r];
    d.dtype_ab = a.dtype; d.dtype_c = c.dtype;
    if (v[7] != NULL && v[7] != Py_None) {
        Tensor bias;
        NEED(as_tensor(v[7], &bias) == 0 && bias.dtype < 2);
        d.bias = bias.ptr;
        d.bias_dtype = bias.dtype;
        d.epilogue |= LLMT_B200_EPI_BIAS;
    }
    if (gelu) d.epilogue |= LLMT_B200_EPI_GELU;
    void* dbias;
    NEED(as_optional_ptr(v[9], &dbias) == 0);
    d.dbias = (float*)dbias;
    if (dbias == NULL) d.dbias_beta = 0.0f;
    PyObject* scratch = NULL;
    if (v[11] != NULL && v[11] != Py_None) {
        PyObject* nb = PyObject_GetAttr(v[11], s_nbytes);
        if (nb == NULL) PyErr_Clear();
        NEED(nb != NULL);
        d.workspace_bytes = PyLong_AsUnsignedLongLong(nb);
        Py_DECREF(nb);
        if (PyErr_Occurred()) PyErr_Clear();
        NEED(as_ptr(v[11], &d.workspace) == 0);
    } else {
        const uint64_t need = E.gemm_workspace_bytes_for(&d, a.ptr, b.ptr);
        if (need > 0) {
            PyObject* n = PyLong_FromUnsignedLongLong(need);
            scratch = n != NULL ? PyObject_CallFunctionObjArgs(g_scratch, n, v[0], v[12] != NULL ? v[12] : Py_None, NULL) : NULL;
            Py_XDECREF(n);
            if (scratch == NULL) return NULL;   // out of memory: torch's own error
            if (as_ptr(scratch, &d.workspace) < 0) { Py_DECREF(scratch); SLOW(); }
            d.workspace_bytes = need;
        }
    }
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = E.gemm(&d, c.ptr, a.ptr, b.ptr, s);
    Py_END_ALLOW_THREADS
    Py_XDECREF(scratch);
    return finish(st);
}

// group_run(descs address, c, a, b addresses, count, stream)
FAST(group_run) {
    BEGIN(5, "descs", "c", "a", "b", "count", "stream");
    void *d, *c, *a, *b, *s;
    int32_t n;
    d = PyLong_AsVoidPtr(v[0]); c = PyLong_AsVoidPtr(v[1]); a = PyLong_AsVoidPtr(v[2]); b = PyLong_AsVoidPtr(v[3]);
    if (PyErr_Occurred()) return NULL;
    NEED(as_int(v[4], &n) == 0 && as_stream(v[5], &s) == 0);
    RUN(E.gemm_grouped((const llmt_b200_gemm_desc*)d, (void* const*)c, (const void* const*)a, (const void* const*)b, n, s));
}

FAST(zero_grads) {
    BEGIN(1, "span", "stream");
    Tensor t;
    void* s;
    NEED(as_tensor(v[0], &t) == 0 && t.dtype == LLMT_B200_FP32 && is_contiguous(&t) && as_stream(v[1], &s) == 0);
    RUN(E.zero_grads((float*)t.ptr, numel(&t), s));
}

FAST(softmax_fwd) {
    BEGIN(3, "y", "x", "causal", "stream");
    Tensor x;
    void *y, *s;
    int32_t causal;
    NEED(as_tensor(v[1], &x) == 0 && x.nd >= 2 && x.dtype < 2 && as_ptr(v[0], &y) == 0 && as_bool(v[2], &causal) == 0 && as_stream(v[3], &s) == 0);
    const int64_t tq = x.shape[x.nd - 2], tk = x.shape[x.nd - 1];
    NEED(tk > 0);
    RUN(E.softmax_fwd(y, x.ptr, numel(&x) / tk, tq, tk, x.dtype, causal, s));
}

FAST(softmax_bwd) {
    BEGIN(3, "ds", "p", "dp", "stream");
    Tensor p;
    void *ds, *dp, *s;
    NEED(as_tensor(v[1], &p) == 0 && p.nd >= 1 && p.dtype < 2 && as_ptr(v[0], &ds) == 0 && as_ptr(v[2], &dp) == 0 && as_stream(v[3], &s) == 0);
    const int64_t tk = p.shape[p.nd - 1];
    NEED(tk > 0);
    RUN(E.softmax_bwd(ds, p.ptr, dp, numel(&p) / tk, tk, p.dtype, s));
}

FAST(gemm_softmax_fwd) {
    BEGIN(5, "desc", "probs", "a", "b", "causal", "lse", "stream");
    llmt_b200_gemm_desc d;
    void *p, *a, *b, *lse, *s;
    int32_t causal;
    NEED(as_desc(v[0], &d) == 0 && as_ptr(v[1], &p) == 0 && as_ptr(v[2], &a) == 0 && as_ptr(v[3], &b) == 0 && as_bool(v[4], &causal) == 0 &&
         as_optional_ptr(v[5], &lse) == 0 && as_stream(v[6], &s) == 0);
    RUN(E.gemm_softmax_fwd(&d, p, a, b, causal, (float*)lse, s));
}

FAST(gemm_softmax_bwd) {
    BEGIN(7, "desc", "ds", "a", "b", "probs", "row_dot", "causal", "stream");
    llmt_b200_gemm_desc d;
    void *ds, *a, *b, *p, *rd, *s;
    int32_t causal;
    NEED(as_desc(v[0], &d) == 0 && as_ptr(v[1], &ds) == 0 && as_ptr(v[2], &a) == 0 && as_ptr(v[3], &b) == 0 && as_ptr(v[4], &p) == 0 &&
         as_ptr(v[5], &rd) == 0 && as_bool(v[6], &causal) == 0 && as_stream(v[7], &s) == 0);
    RUN(E.gemm_softmax_bwd(&d, ds, a, b, p, (const float*)rd, causal, s));
}

FAST(rowdot) {
    BEGIN(3, "out", "x", "y", "stream");
    Tensor o, x, y;
    void* s;
    NEED(as_tensor(v[0], &o) == 0 && as_tensor(v[1], &x) == 0 && as_tensor(v[2], &y) == 0 && as_stream(v[3], &s) == 0);
    NEED(x.nd == y.nd && x.nd >= 1 && x.dtype == y.dtype && x.dtype < 2 && memcmp(x.shape, y.shape, sizeof(int64_t) * (size_t)x.nd) == 0);
    const int64_t cols = x.shape[x.nd - 1];
    NEED(cols > 0 && o.dtype == LLMT_B200_FP32 && numel(&o) == numel(&x) / cols && is_contiguous(&x) && is_contiguous(&y));
    RUN(E.rowdot((float*)o.ptr, x.ptr, y.ptr, numel(&x) / cols, cols, cols, cols, x.dtype, s));
}

FAST(head_split) {
    BEGIN(4, "q", "k", "v", "qkv", "stream");
    Tensor q, w;
    void *k, *vv, *s;
    NEED(as_tensor(v[0], &q) == 0 && q.nd == 4 && as_tensor(v[3], &w) == 0 && w.dtype < 2 && as_ptr(v[1], &k) == 0 && as_ptr(v[2], &vv) == 0 &&
         as_stream(v[4], &s) == 0);
    RUN(E.head_split(q.ptr, k, vv, w.ptr, q.shape[0], q.shape[1], q.shape[2], q.shape[3], w.dtype, s));
}

FAST(head_merge) {
    BEGIN(2, "y", "x", "stream");
    Tensor x;
    void *y, *s;
    NEED(as_tensor(v[1], &x) == 0 && x.nd == 4 && x.dtype < 2 && as_ptr(v[0], &y) == 0 && as_stream(v[2], &s) == 0);
    RUN(E.head_merge(y, x.ptr, x.shape[0], x.shape[1], x.shape[2], x.shape[3], x.dtype, s));
}

FAST(cross_entropy_fwd) {
    BEGIN(5, "loss", "row_nll", "logits", "targets", "mask", "stream");
    Tensor l, t, m;
    void *loss, *nll, *s;
    NEED(as_tensor(v[2], &l) == 0 && as_tensor(v[3], &t) == 0 && as_tensor(v[4], &m) == 0 && as_ptr(v[0], &loss) == 0 && as_ptr(v[1], &nll) == 0 &&
         as_stream(v[5], &s) == 0);
    NEED(l.dtype == LLMT_B200_FP32 && t.dtype == 2 && m.dtype == LLMT_B200_FP32 && l.nd >= 1 && l.shape[l.nd - 1] > 0);
    const int64_t n = l.shape[l.nd - 1];
    RUN(E.cross_entropy_fwd((float*)loss, (float*)nll, (const float*)l.ptr, (const int32_t*)t.ptr, (const float*)m.ptr, numel(&l) / n, n,
                                      l.nd > 1 ? l.stride[l.nd - 2] : n, s));
}

FAST(cross_entropy_bwd) {
    BEGIN(4, "dlogits", "logits", "targets", "mask", "dloss", "stream");
    Tensor d, l;
    void *t, *m, *s;
    float g;
    NEED(as_tensor(v[0], &d) == 0 && as_tensor(v[1], &l) == 0 && as_ptr(v[2], &t) == 0 && as_ptr(v[3], &m) == 0 && as_float(v[4], 1.0f, &g) == 0 &&
         as_stream(v[5], &s) == 0);
    NEED(d.dtype == LLMT_B200_FP32 && l.dtype == LLMT_B200_FP32 && d.nd == l.nd && l.nd >= 1 && l.shape[l.nd - 1] > 0 &&
         memcmp(d.shape, l.shape, sizeof(int64_t) * (size_t)l.nd) == 0);
    const int64_t n = l.shape[l.nd - 1];
    RUN(E.cross_entropy_bwd((float*)d.ptr, (const float*)l.ptr, (const int32_t*)t, (const float*)m, g, numel(&l) / n, n,
                                      l.nd > 1 ? l.stride[l.nd - 2] : n, d.nd > 1 ? d.stride[d.nd - 2] : n, s));
}

FAST(lm_head_ce_fwd) {
    BEGIN(8, "desc", "logits", "a", "b", "targets", "mask", "row_nll", "loss", "stream");
    llmt_b200_gemm_desc d;
    void *l, *a, *b, *t, *m, *nll, *loss, *s;
    NEED(as_desc(v[0], &d) == 0 && as_optional_ptr(v[1], &l) == 0 && as_ptr(v[2], &a) == 0 && as_ptr(v[3], &b) == 0 && as_ptr(v[4], &t) == 0 &&
         as_ptr(v[5], &m) == 0 && as_ptr(v[6], &nll) == 0 && as_ptr(v[7], &loss) == 0 && as_stream(v[8], &s) == 0);
    RUN(E.lm_head_ce_fwd(&d, l, a, b, (const int32_t*)t, (const float*)m, (float*)nll, (float*)loss, s));
}

FAST(lm_head_ce_bwd) {
    BEGIN(6, "desc", "dlogits", "a", "b", "targets", "mask", "dloss", "stats_valid", "stream");
    llmt_b200_gemm_desc d;
    void *l, *a, *b, *t, *m, *s;
    float g;
    int32_t valid;
    NEED(as_desc(v[0], &d) == 0 && as_ptr(v[1], &l) == 0 && as_ptr(v[2], &a) == 0 && as_ptr(v[3], &b) == 0 && as_ptr(v[4], &t) == 0 &&
         as_ptr(v[5], &m) == 0 && as_float(v[6], 1.0f, &g) == 0 && as_bool(v[7], &valid) == 0 && as_stream(v[8], &s) == 0);
    RUN(E.lm_head_ce_bwd(&d, l, a, b, (const int32_t*)t, (const float*)m, g, valid, s));
}

// ---------------------------------------------------------------------------------- module

typedef PyObject* (*FastFn)(PyObject*, PyObject* const*, Py_ssize_t, PyObject*);
static const struct { const char* name; FastFn fn; } kFast[] = {
#define ROW(name) {#name, fast_##name}
    {"_group_run", fast_group_run}, ROW(gemm), ROW(gemm_desc), ROW(zero_grads), ROW(softmax_fwd), ROW(softmax_bwd), ROW(gemm_softmax_fwd),
    ROW(gemm_softmax_bwd), ROW(rowdot), ROW(head_split), ROW(head_merge), ROW(cross_entropy_fwd), ROW(cross_entropy_bwd),
    ROW(lm_head_ce_fwd), ROW(lm_head_ce_bwd)};

// What stands in the Python function's place: calls go to the native function, every attribute that it does not have itself
// is the Python function's, and it is pickled by name as a function is.
typedef struct {
    PyObject_HEAD
    vectorcallfunc vectorcall;
    FastFn fn;
    PyObject *slow, *dict, *weak;
} Fast;
static PyObject* fast_vectorcall(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kw) {
    Fast* f = (Fast*)self;
    return f->fn(f->slow, args, PyVectorcall_NARGS(nargsf), kw);
}
static PyObject* fast_getattro(PyObject* self, PyObject* name) {
    PyObject* r = PyObject_GenericGetAttr(self, name);
    if (r != NULL || !PyErr_ExceptionMatches(PyExc_AttributeError)) return r;
    PyErr_Clear();
    return PyObject_GetAttr(((Fast*)self)->slow, name);
}
static PyObject* fast_descr_get(PyObject* self, PyObject* obj, PyObject* type) {
    (void)type;
    if (obj == NULL || obj == Py_None) { Py_INCREF(self); return self; }
    return PyMethod_New(self, obj);
}
static PyObject* fast_repr(PyObject* self) { return PyUnicode_FromFormat("<native form of %R>", ((Fast*)self)->slow); }
static PyObject* fast_reduce(PyObject* self, PyObject* unused) {
    (void)unused;
    return PyObject_GetAttrString(self, "__qualname__");
}
static int fast_traverse(PyObject* self, visitproc visit, void* arg) {
    Py_VISIT(((Fast*)self)->slow);
    Py_VISIT(((Fast*)self)->dict);
    return 0;
}
static int fast_clear(PyObject* self) {
    Py_CLEAR(((Fast*)self)->dict);
    return 0;
}
static void fast_dealloc(PyObject* self) {
    PyObject_GC_UnTrack(self);
    if (((Fast*)self)->weak != NULL) PyObject_ClearWeakRefs(self);
    fast_clear(self);
    Py_CLEAR(((Fast*)self)->slow);
    PyObject_GC_Del(self);
}
static PyMethodDef kFastMethods[] = {{"__reduce__", fast_reduce, METH_NOARGS, NULL}, {NULL, NULL, 0, NULL}};
static PyGetSetDef kFastGetSet[] = {{"__dict__", PyObject_GenericGetDict, PyObject_GenericSetDict, NULL, NULL}, {NULL, NULL, NULL, NULL, NULL}};
static PyTypeObject FastType = {
    PyVarObject_HEAD_INIT(NULL, 0)
    .tp_name = "llmt_b200._native.Function", .tp_basicsize = sizeof(Fast),
    .tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL,
    .tp_vectorcall_offset = offsetof(Fast, vectorcall), .tp_call = PyVectorcall_Call, .tp_getattro = fast_getattro,
    .tp_setattro = PyObject_GenericSetAttr, .tp_dictoffset = offsetof(Fast, dict), .tp_weaklistoffset = offsetof(Fast, weak),
    .tp_descr_get = fast_descr_get, .tp_repr = fast_repr, .tp_methods = kFastMethods, .tp_getset = kFastGetSet,
    .tp_traverse = fast_traverse, .tp_clear = fast_clear, .tp_dealloc = fast_dealloc};

// fast(python_function): the native function of that name, with the Python one behind it.
static PyObject* py_fast(PyObject* self, PyObject* slow) {
    (void)self;
    PyObject* name = PyObject_GetAttrString(slow, "__name__");
    const char* text = name != NULL ? PyUnicode_AsUTF8(name) : NULL;
    Fast* r = NULL;
    for (size_t i = 0; text != NULL && r == NULL && i < sizeof(kFast) / sizeof(kFast[0]); ++i) {
        if (strcmp(text, kFast[i].name) != 0) continue;
        r = PyObject_GC_New(Fast, &FastType);
        if (r == NULL) break;
        r->vectorcall = fast_vectorcall;
        r->fn = kFast[i].fn;
        r->dict = r->weak = NULL;
        Py_INCREF(slow);
        r->slow = slow;
        PyObject_GC_Track((PyObject*)r);
    }
    if (r == NULL && !PyErr_Occurred()) PyErr_Format(PyExc_ValueError, "no native function for %R", slow);
    Py_XDECREF(name);
    if (r == NULL) return NULL;
    // its name, module, documentation, annotations and __wrapped__ (which gives it the signature)
    PyObject* functools = PyImport_ImportModule("functools");
    PyObject* wrapped = functools != NULL ? PyObject_CallMethod(functools, "update_wrapper", "OO", (PyObject*)r, slow) : NULL;
    Py_XDECREF(functools);
    Py_DECREF(r);
    return wrapped;
}

// setup(binder, raise, scratch): what the native functions call back into.
static PyObject* py_setup(PyObject* self, PyObject* args) {
    (void)self;
    PyObject *b, *r, *s;
    if (!PyArg_ParseTuple(args, "OOO", &b, &r, &s)) return NULL;
    Py_INCREF(b); Py_INCREF(r); Py_INCREF(s);
    g_binder = b; g_raise = r; g_scratch = s;
    Py_RETURN_NONE;
}

// bind(addresses in the order of NAMES, torch's raw-stream and device getters, float32, bfloat16, int32, GemmDesc)
static PyObject* py_bind(PyObject* self, PyObject* args) {
    (void)self;
    PyObject *list, *rs, *gd, *f, *h, *i32, *desc;
    if (!PyArg_ParseTuple(args, "O!OOOOOO!", &PyTuple_Type, &list, &rs, &gd, &f, &h, &i32, &PyType_Type, &desc)) return NULL;
    if (PyTuple_GET_SIZE(list) != N_ENTRIES) return PyErr_Format(PyExc_ValueError, "bind: %zd addresses expected", N_ENTRIES);
    void* p[sizeof(kNames) / sizeof(kNames[0])];
    for (Py_ssize_t i = 0; i < N_ENTRIES; ++i) {
        p[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(list, i));
        if (p[i] == NULL) return PyErr_Occurred() ? NULL : PyErr_Format(PyExc_ValueError, "bind: null address for %s", kNames[i]);
    }
    memcpy(&E, p, sizeof E);
    Py_INCREF(rs); Py_INCREF(gd); Py_INCREF(f); Py_INCREF(h); Py_INCREF(i32); Py_INCREF(desc);
    g_raw_stream = rs; g_get_device = gd; g_float32 = f; g_bfloat16 = h; g_int32 = i32; g_desc_type = desc;
    g_bound = 1;
    Py_RETURN_NONE;
}

static PyMethodDef kMethods[] = {{"fast", py_fast, METH_O, "The native form of a Python function of this binding."},
                                 {"setup", py_setup, METH_VARARGS, "Callbacks of the native functions."},
                                 {"bind", py_bind, METH_VARARGS, "Entry points of the loaded library."},
                                 {NULL, NULL, 0, NULL}};
static struct PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Native call path of llmt_b200.", -1, kMethods, NULL, NULL, NULL, NULL};

PyMODINIT_FUNC PyInit__native(void) {
    if (PyType_Ready(&FastType) < 0) return NULL;
    PyObject* m = PyModule_Create(&kModule);
    if (m == NULL) return NULL;
    s_data_ptr = PyUnicode_InternFromString("data_ptr");
    s_shape = PyUnicode_InternFromString("shape");
    s_stride = PyUnicode_InternFromString("stride");
    s_dtype = PyUnicode_InternFromString("dtype");
    s_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    s_nbytes = PyUnicode_InternFromString("nbytes");
    PyObject* names = PyTuple_New(N_ENTRIES);
    if (names == NULL || s_data_ptr == NULL || s_shape == NULL || s_stride == NULL || s_dtype == NULL || s_cuda_stream == NULL || s_nbytes == NULL) {
        Py_DECREF(m);
        return NULL;
    }
    for (Py_ssize_t i = 0; i < N_ENTRIES; ++i) PyTuple_SET_ITEM(names, i, PyUnicode_FromString(kNames[i]));
    if (PyModule_AddObject(m, "NAMES", names) < 0) { Py_DECREF(m); return NULL; }
    return m;
}
