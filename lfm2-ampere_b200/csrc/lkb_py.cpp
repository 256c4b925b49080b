// lkb_py.cpp - CPython bindings of the entry points that prefill and single-projection hosts call most.
//
// The same calls through ctypes cost 1 to 2 us each beside the launch, and a GEMM descriptor 7: up to eighteen arguments converted one by one, every
// tensor looked at from Python three times.  Here a call reads its tensors through torch's own objects.  Each function takes its Python
// wrapper's arguments (api.py, which has the names and defaults) in order, adds the current stream, and returns the entry point's status.
// Host time, us: one projection with its norm and residual (two calls and a copy) 14.1 -> 11.0, a prefill layer of the model (nine launches, four
// descriptors) 69 -> 34.
#define PY_SSIZE_T_CLEAN
#include <torch/csrc/autograd/python_variable.h>
#include "../../include/lkb.h"

static PyObject * g_stream, * g_device;
static PyObject * g_act_type, * g_ctypes_object, * g_argument_error;        // PfAct, the base of every ctypes object, what a refused argument raises

// The address of anything else with a tensor's is_cuda, is_contiguous() and data_ptr(): subclasses that override them, wrappers of memory of their own.
static void * other_ptr(PyObject * t, int * bad) {
    PyObject * cuda = PyObject_GetAttrString(t, "is_cuda"), * whole = NULL, * at = NULL;
    int yes = cuda ? PyObject_IsTrue(cuda) : -1;
    if (yes > 0) whole = PyObject_CallMethod(t, "is_contiguous", NULL), yes = whole ? PyObject_IsTrue(whole) : -1;
    if (!yes) PyErr_SetString(PyExc_AssertionError, "device-resident contiguous tensors only");
    else if (yes < 0 && PyErr_ExceptionMatches(PyExc_AttributeError)) PyErr_SetString(PyExc_TypeError, "a tensor is wanted");
    void * p = NULL;
    if (yes > 0) at = PyObject_CallMethod(t, "data_ptr", NULL), p = at ? PyLong_AsVoidPtr(at) : NULL;
    Py_XDECREF(cuda); Py_XDECREF(whole); Py_XDECREF(at);
    if (PyErr_Occurred()) *bad = 1;
    return p;
}
// A tensor's address; NULL for None.  Sets *bad with an exception pending.
static void * as_ptr(PyObject * t, int * bad) {
    if (*bad || t == Py_None) return nullptr;
    if (!THPVariable_CheckExact(t)) return other_ptr(t, bad);
    try {
        const at::Tensor & v = THPVariable_Unpack(t);
        if (!v.is_cuda() || !v.is_contiguous()) { PyErr_SetString(PyExc_AssertionError, "device-resident contiguous tensors only"); *bad = 1; return nullptr; }
        return v.data_ptr();
    } catch (const std::exception & e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        *bad = 1;
        return nullptr;
    }
}
// What a number of another type raises: the same text under ctypes' exception.
static void refuse() {
    if (!PyErr_ExceptionMatches(PyExc_TypeError) || !g_argument_error) return;
    PyObject * type, * value, * trace;
    PyErr_Fetch(&type, &value, &trace);
    PyErr_Format(g_argument_error, "%S", value ? value : type);
    Py_XDECREF(type); Py_XDECREF(value); Py_XDECREF(trace);
}
static long long as_int(PyObject * o, int * bad) {               // masked to the field it goes into, as ctypes does
    if (*bad) return 0;
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
    if (v == (unsigned long long) -1 && PyErr_Occurred()) { refuse(); *bad = 1; }
    return (long long) v;
}
static float as_float(PyObject * o, int * bad) {
    if (*bad) return 0.0f;
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) { refuse(); *bad = 1; }
    return (float) v;
}
// The bytes of an object of the ctypes type given; a subclass may be longer.  They stay where they are while the caller holds the object, as it does for the call.
static void * as_struct(PyObject * o, PyObject * type, size_t size, int * bad) {
    if (*bad) return nullptr;
    *bad = 1;
    const int is = type ? PyObject_IsInstance(o, type) : 0;
    if (is < 0) return nullptr;
    Py_buffer b;
    if (!is || PyObject_GetBuffer(o, &b, PyBUF_WRITABLE)) {
        PyErr_Clear();
        if (!g_argument_error || !type) PyErr_SetString(PyExc_RuntimeError, "no types set");
        else PyErr_Format(g_argument_error, "expected %s instance instead of %s", ((PyTypeObject *) type)->tp_name, Py_TYPE(o)->tp_name);
        return nullptr;
    }
    void * const p = b.buf;
    const size_t len = (size_t) b.len;
    PyBuffer_Release(&b);
    if (len < size) { PyErr_SetString(g_argument_error, "a shorter structure than the one wanted"); return nullptr; }
    *bad = 0;
    return p;
}
// What lookup(device()) gives, or lookup() where there is no device function.
static lkb_stream_t current_stream(int * bad) {
    if (*bad) return nullptr;
    PyObject * s = nullptr;
    if (!g_stream) PyErr_SetString(PyExc_RuntimeError, "no stream lookup set");
    else if (!g_device) s = PyObject_CallNoArgs(g_stream);
    else if (PyObject * d = PyObject_CallNoArgs(g_device)) { s = PyObject_CallOneArg(g_stream, d); Py_DECREF(d); }
    if (!s) { *bad = 1; return nullptr; }
    lkb_stream_t st = (lkb_stream_t) PyLong_AsVoidPtr(s);
    Py_DECREF(s);
    if (PyErr_Occurred()) *bad = 1;
    return st;
}

// converts to whatever pointer the entry point takes
struct Ptr { void * p; template <class T> operator T *() const { return (T *) p; } };
#define P(i) Ptr{as_ptr(a[i], &bad)}
#define I(i) (int) as_int(a[i], &bad)
#define F(i) as_float(a[i], &bad)
#define ACT(i) const lkb_pf_act * act = (const lkb_pf_act *) as_struct(a[i], g_act_type, sizeof(lkb_pf_act), &bad)
#define GEMM(i) const lkb_pf_gemm * g = (const lkb_pf_gemm *) as_struct(a[i], g_ctypes_object, sizeof(lkb_pf_gemm), &bad)      /* any type, as by ctypes.byref */
// Arguments first, in order; then the call, without the interpreter's lock (a launch may block when the device's queue is full).
#define ENTRY(name, count, args, call) \
    static PyObject * f_##name(PyObject * self, PyObject * const * a, Py_ssize_t n) { \
        (void) self; \
        if (n != count) { PyErr_SetString(PyExc_TypeError, #name " takes " #count " arguments"); return NULL; } \
        int bad = 0, r; \
        args; \
        const lkb_stream_t st = current_stream(&bad); \
        if (bad) return NULL; \
        Py_BEGIN_ALLOW_THREADS \
        r = call; \
        Py_END_ALLOW_THREADS \
        return PyLong_FromLong(r); \
    }

ENTRY(rmsnorm_q8_1, 7, Ptr x = P(0); Ptr w = P(1); int m = I(2); float eps = F(3); Ptr y32 = P(4); Ptr y16 = P(5); Ptr q = P(6),
      lkb_rmsnorm_q8_1(x, w, m, eps, y32, y16, q, st))
ENTRY(gemv_q4_0, 9, Ptr qs = P(0); Ptr d = P(1); Ptr xq = P(2); int rows = I(3); int bpr = I(4); Ptr y = P(5); int add = I(6); Ptr ssq = P(7); float eps = F(8),
      lkb_gemv_q4_0(qs, d, xq, rows, bpr, y, add, ssq, eps, st))
ENTRY(gemv_q6_K, 10, Ptr ql = P(0); Ptr qh = P(1); Ptr sc = P(2); Ptr d = P(3); Ptr xq = P(4); int rows = I(5); int sbpr = I(6); Ptr y = P(7); Ptr ssq = P(8);
      float eps = F(9), lkb_gemv_q6_K(ql, qh, sc, d, xq, rows, sbpr, y, ssq, eps, st))
ENTRY(argmax_part, 4, Ptr v = P(0); int m = I(1); Ptr pv = P(2); Ptr pi = P(3), lkb_argmax_part(v, m, pv, pi, st))
ENTRY(argmax_final, 5, Ptr pv = P(0); Ptr pi = P(1); int m = I(2); Ptr tok = P(3); Ptr pos = P(4), lkb_argmax_final(pv, pi, m, tok, pos, st))
ENTRY(pf_embed, 8, Ptr ql = P(0); Ptr qh = P(1); Ptr sc = P(2); Ptr d = P(3); Ptr toks = P(4); Ptr x = P(5); int cols = I(6); int m = I(7),
      lkb_pf_embed(ql, qh, sc, d, toks, x, cols, m, st))
ENTRY(pf_norm, 7, Ptr x = P(0); Ptr w = P(1); int plain = I(2); ACT(3); Ptr inv = P(4); Ptr h = P(5); int m = I(6), lkb_pf_norm(x, w, plain, *act, inv, h, m, st))
ENTRY(pf_norm_router_select, 13, Ptr x = P(0); Ptr w = P(1); ACT(2); Ptr inv = P(3); Ptr h = P(4); int m = I(5); int small = I(6); Ptr wr = P(7); Ptr bias = P(8);
      Ptr sel = P(9); Ptr sig = P(10); Ptr idx = P(11); Ptr wo = P(12), lkb_pf_norm_router_select(x, w, *act, inv, h, m, small, wr, bias, sel, sig, idx, wo, st))
ENTRY(pf_moe_route, 7, Ptr idx = P(0); int m = I(1); Ptr cnt = P(2); Ptr off = P(3); Ptr tiles = P(4); Ptr nt = P(5); Ptr perm = P(6),
      lkb_pf_moe_route(idx, m, cnt, off, tiles, nt, perm, st))
ENTRY(pf_gemm_dense, 1, GEMM(0), lkb_pf_gemm_dense(g, st))
ENTRY(pf_gemm_moe, 2, GEMM(0); int mt = I(1), lkb_pf_gemm_moe(g, mt, st))
ENTRY(pf_gemm_swiglu, 2, GEMM(0); int mt = I(1), lkb_pf_gemm_swiglu(g, mt, st))
ENTRY(pf_moe_combine_norm, 7, Ptr x = P(0); Ptr d = P(1); Ptr w = P(2); Ptr nw = P(3); ACT(4); Ptr inv = P(5); int m = I(6),
      lkb_pf_moe_combine_norm(x, d, w, nw, *act, inv, m, st))
ENTRY(pf_conv_next, 5, Ptr y = P(0); Ptr cw = P(1); Ptr hist = P(2); ACT(3); int m = I(4), lkb_pf_conv_next(y, cw, hist, *act, m, st))
ENTRY(pf_qknr, 9, Ptr y = P(0); Ptr qn = P(1); Ptr kn = P(2); int pos = I(3); Ptr qh = P(4); Ptr kc = P(5); Ptr vc = P(6); int m = I(7); float theta = F(8),
      lkb_pf_qknr(y, qn, kn, pos, qh, kc, vc, m, theta, st))
ENTRY(pf_attn, 6, Ptr qh = P(0); int m = I(1); int pos = I(2); Ptr kc = P(3); Ptr vc = P(4); Ptr o = P(5), lkb_pf_attn(qh, m, pos, kc, vc, o, st))
ENTRY(pf_quant_rows, 5, Ptr x = P(0); int ld = I(1); int kb = I(2); ACT(3); int rows = I(4), lkb_pf_quant_rows(x, ld, kb, *act, rows, st))

// The fields of an lkb_pf_gemm, in the order of api.make_pf_gemm's arguments, into the ctypes structure given first.
static PyObject * f_fill_pf_gemm(PyObject * self, PyObject * const * a, Py_ssize_t n) {
    (void) self;
    if (n != 20) { PyErr_SetString(PyExc_TypeError, "fill_pf_gemm takes 20 arguments"); return NULL; }
    int bad = 0;
    lkb_pf_gemm * const g = (lkb_pf_gemm *) as_struct(a[0], g_ctypes_object, sizeof(lkb_pf_gemm), &bad);
    PyObject * segs = bad ? NULL : PySequence_Fast(a[1], "segs: a sequence of (qs, d)"), * ends = segs ? PySequence_Fast(a[2], "seg_end: a sequence") : NULL;
    const Py_ssize_t ns = segs ? PySequence_Fast_GET_SIZE(segs) : 0, ne = ends ? PySequence_Fast_GET_SIZE(ends) : 0;
    if (!ends) bad = 1;
    else if (ns < 1 || ne < 1) { PyErr_SetString(PyExc_IndexError, "no weight segment"); bad = 1; }
    for (Py_ssize_t i = 0; i < 3 && !bad; ++i) {
        PyObject * pair = PySequence_Fast(PySequence_Fast_GET_ITEM(segs, i < ns ? i : ns - 1), "a segment: (qs, d)");
        if (!pair || PySequence_Fast_GET_SIZE(pair) != 2) {
            if (pair) PyErr_SetString(PyExc_ValueError, "a segment: (qs, d)");
            bad = 1;
        } else {
            g->qs[i] = as_ptr(PySequence_Fast_GET_ITEM(pair, 0), &bad);
            g->d[i] = as_ptr(PySequence_Fast_GET_ITEM(pair, 1), &bad);
            g->seg_end[i] = (int) as_int(PySequence_Fast_GET_ITEM(ends, i < ne ? i : ne - 1), &bad);
        }
        Py_XDECREF(pair);
    }
    if (!bad) {
        g->N = I(3); g->bpr = I(4); g->aqs = P(5); g->asc = P(6);
        g->ntok = I(7); g->exp_stride = as_int(a[8], &bad); g->perm = P(9); g->tiles = P(10); g->ntiles = P(11);
        g->a_shift = I(12); g->scale = P(13); g->out = P(14); g->out_ld = I(15); g->add = I(16); g->oqs = P(17); g->osc = P(18); g->okb = I(19);
    }
    Py_XDECREF(segs); Py_XDECREF(ends);
    if (bad) return NULL;
    Py_RETURN_NONE;
}
static PyObject * f_ptr(PyObject * self, PyObject * t) {
    (void) self;
    int bad = 0;
    void * const p = as_ptr(t, &bad);
    if (bad) return NULL;
    if (t == Py_None) Py_RETURN_NONE;
    return PyLong_FromVoidPtr(p);
}
static PyObject * f_set_stream_lookup(PyObject * self, PyObject * const * a, Py_ssize_t n) {
    (void) self;
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "set_stream_lookup takes a lookup and a device function or None"); return NULL; }
    Py_INCREF(a[0]);
    Py_XSETREF(g_stream, a[0]);
    Py_XINCREF(a[1] == Py_None ? NULL : a[1]);
    Py_XSETREF(g_device, a[1] == Py_None ? NULL : a[1]);
    Py_RETURN_NONE;
}

static PyObject * f_set_types(PyObject * self, PyObject * const * a, Py_ssize_t n) {
    (void) self;
    if (n != 3 || !PyType_Check(a[0]) || !PyType_Check(a[1]) || !PyExceptionClass_Check(a[2])) {
        PyErr_SetString(PyExc_TypeError, "set_types takes PfAct, the base of ctypes objects and an exception");
        return NULL;
    }
    Py_INCREF(a[0]); Py_XSETREF(g_act_type, a[0]);
    Py_INCREF(a[1]); Py_XSETREF(g_ctypes_object, a[1]);
    Py_INCREF(a[2]); Py_XSETREF(g_argument_error, a[2]);
    Py_RETURN_NONE;
}

#define M(name) {#name, (PyCFunction) (void (*)(void)) f_##name, METH_FASTCALL, NULL}
static PyMethodDef methods[] = {
    M(rmsnorm_q8_1), M(gemv_q4_0), M(gemv_q6_K), M(argmax_part), M(argmax_final), M(pf_embed), M(pf_norm), M(pf_norm_router_select), M(pf_moe_route),
    M(pf_gemm_dense), M(pf_gemm_moe), M(pf_gemm_swiglu), M(pf_moe_combine_norm), M(pf_conv_next), M(pf_qknr), M(pf_attn), M(pf_quant_rows), M(fill_pf_gemm),
    M(set_stream_lookup), M(set_types), {"ptr", f_ptr, METH_O, NULL}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__fast(void) {
    PyObject * m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "built_for", LKB_BUILT_FOR)) Py_CLEAR(m);       // the torch whose objects it reads; the package looks at it
    return m;
}
