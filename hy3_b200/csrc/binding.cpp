/*
 * binding.cpp -- the per-step calls of Hy3Attn (attn.py) as native functions: batch_set, append, decode_step, prefill.
 *
 * A decode step of a short context takes 6 to 9 us on the GPU; the same call through ctypes cost the host 6.6 us (four to seven
 * tensors asked for their strides, types and addresses one attribute at a time, 11 to 15 arguments converted one by one).  Here the
 * checks are the same and made on every call, on the tensors themselves.  The C ABI stays the way in: the functions' addresses come
 * from the library that _lib.py loaded (bind()).
 */
#include <Python.h>

#include <torch/csrc/autograd/python_variable.h>

#include "../../include/hy3_attn.h"

namespace {

decltype(&hy3a_batch_set) f_batch_set;
decltype(&hy3a_append) f_append;
decltype(&hy3a_decode_step) f_decode_step;
decltype(&hy3a_prefill) f_prefill;

constexpr int64_t kH = HY3A_N_HEAD, kD = HY3A_HEAD_DIM;

PyObject *refuse(const char *what) {
    PyErr_SetString(PyExc_AssertionError, what);
    return nullptr;
}
/* a tensor argument: nullptr for None */
bool tensor(PyObject *o, const at::Tensor *&t) {
    t = nullptr;
    if (o == Py_None) return true;
    if (!THPVariable_Check(o)) { PyErr_SetString(PyExc_TypeError, "expected a torch.Tensor or None"); return false; }
    t = &THPVariable_Unpack(o);
    return true;
}
template <class T> T *ptr(const at::Tensor *t) { return t ? static_cast<T *>(t->data_ptr()) : nullptr; }
/* fp32 rows of dense heads: n of them, row stride free */
bool rows(const at::Tensor *t, int64_t n) {
    if (!t) return true;
    const int64_t d = t->dim();
    return d >= 2 && t->size(0) == n && t->scalar_type() == at::kFloat && t->stride(d - 1) == 1 && t->stride(d - 2) == kD;
}
size_t stride0(const at::Tensor *t) { return t ? (size_t)t->stride(0) : 0; }

/* a C-contiguous host buffer */
struct buffer {
    Py_buffer b;
    bool held = false;
    ~buffer() { if (held) PyBuffer_Release(&b); }
    bool get(PyObject *o) {
        if (PyObject_GetBuffer(o, &b, PyBUF_C_CONTIGUOUS)) return false;
        held = true;
        return true;
    }
};

/* C++ exceptions (a tensor without storage, without strides) become Python's */
template <PyObject *(*F)(PyObject *const *, Py_ssize_t)>
PyObject *guarded(PyObject *, PyObject *const *a, Py_ssize_t na) {
    try {
        return F(a, na);
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

int as_int(PyObject *o) {
    const long v = PyLong_AsLong(o);
    if (v != (int)v) PyErr_SetString(PyExc_OverflowError, "value does not fit an int");
    return (int)v;
}
/* the leading arguments of the per-layer calls: ctx, layer */
bool head(PyObject *const *a, hy3a_ctx *&h, int &layer) {
    h = (hy3a_ctx *)PyLong_AsVoidPtr(a[0]);
    if (!h && PyErr_Occurred()) return false;
    layer = as_int(a[1]);
    return !PyErr_Occurred();
}

/* batch_set(ctx, seq, slot, pos): int32 arrays of the same length */
PyObject *batch_set(PyObject *const *a, Py_ssize_t na) {
    if (na != 4) return refuse("batch_set: 4 arguments");
    hy3a_ctx *h = (hy3a_ctx *)PyLong_AsVoidPtr(a[0]);
    if (!h && PyErr_Occurred()) return nullptr;
    buffer v[3];
    for (int i = 0; i < 3; i++) if (!v[i].get(a[1 + i])) return nullptr;
    if (v[0].b.itemsize != 4 || v[1].b.itemsize != 4 || v[2].b.itemsize != 4 || v[0].b.len != v[1].b.len || v[0].b.len != v[2].b.len)
        return refuse("batch_set: int32 arrays of one length");
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f_batch_set(h, (int)(v[0].b.len / 4), (const int *)v[0].b.buf, (const int *)v[1].b.buf, (const int *)v[2].b.buf);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
/* append(ctx, layer, n, q, k, v, q_out, q_out16) */
PyObject *append(PyObject *const *a, Py_ssize_t na) {
    if (na != 8) return refuse("append: 8 arguments");
    hy3a_ctx *h;
    int layer;
    if (!head(a, h, layer)) return nullptr;
    const int64_t n = PyLong_AsLongLong(a[2]);
    const at::Tensor *q, *k, *v, *qo, *q16;
    if (PyErr_Occurred() || !tensor(a[3], q) || !tensor(a[4], k) || !tensor(a[5], v) || !tensor(a[6], qo) || !tensor(a[7], q16)) return nullptr;
    if (!q || !k != !v) return refuse("append: q, and k with v");
    if (!rows(q, n) || !rows(k, n) || !rows(v, n)) return refuse("append: q, k, v are fp32 with n rows of dense heads");
    if (q16 && (q16->scalar_type() != at::kHalf || !q16->is_contiguous() || q16->numel() != n * kH * kD)) return refuse("append: q_out16 is contiguous fp16 [n, 64, 128]");
    const float *qp = ptr<const float>(q), *kp = ptr<const float>(k), *vp = ptr<const float>(v);
    float *qop = ptr<float>(qo);
    void *q16p = ptr<void>(q16);
    const size_t sq = stride0(q), sk = stride0(k), sv = stride0(v), so = stride0(qo);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f_append(h, layer, qp, sq, kp, sk, vp, sv, qop, so, q16p);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
/* decode_step(ctx, layer, n, q, k, v, q_out, out, partials) */
PyObject *decode_step(PyObject *const *a, Py_ssize_t na) {
    if (na != 9) return refuse("decode_step: 9 arguments");
    hy3a_ctx *h;
    int layer;
    if (!head(a, h, layer)) return nullptr;
    const int64_t n = PyLong_AsLongLong(a[2]);
    const at::Tensor *q, *k, *v, *qo, *out, *part;
    if (PyErr_Occurred() || !tensor(a[3], q) || !tensor(a[4], k) || !tensor(a[5], v) || !tensor(a[6], qo) || !tensor(a[7], out) || !tensor(a[8], part)) return nullptr;
    if (!q || !k != !v) return refuse("decode_step: q, and k with v");
    if (!rows(q, n) || !rows(k, n) || !rows(v, n)) return refuse("decode_step: q, k, v are fp32 with n rows of dense heads");
    const float *qp = ptr<const float>(q), *kp = ptr<const float>(k), *vp = ptr<const float>(v);
    float *qop = ptr<float>(qo), *op = ptr<float>(out), *pp = ptr<float>(part);
    const size_t sq = stride0(q), sk = stride0(k), sv = stride0(v), sqo = stride0(qo), so = stride0(out);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f_decode_step(h, layer, qp, sq, kp, sk, vp, sv, qop, sqo, op, so, pp);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
/* prefill(ctx, layer, seq, base_slot, q16, out) */
PyObject *prefill(PyObject *const *a, Py_ssize_t na) {
    if (na != 6) return refuse("prefill: 6 arguments");
    hy3a_ctx *h;
    int layer;
    if (!head(a, h, layer)) return nullptr;
    const int seq = as_int(a[2]), base = PyErr_Occurred() ? 0 : as_int(a[3]);
    const at::Tensor *q16, *out;
    if (PyErr_Occurred() || !tensor(a[4], q16) || !tensor(a[5], out)) return nullptr;
    if (!q16 || !out || q16->dim() < 1 || q16->scalar_type() != at::kHalf || !q16->is_contiguous()) return refuse("prefill: q16 is contiguous fp16, out a tensor");
    const int nq = (int)q16->size(0);
    const void *qp = ptr<const void>(q16);
    float *op = ptr<float>(out);
    const size_t so = stride0(out);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f_prefill(h, layer, seq, base, nq, qp, op, so);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
/* bind(addresses of hy3a_batch_set, hy3a_append, hy3a_decode_step, hy3a_prefill) */
PyObject *bind(PyObject *const *a, Py_ssize_t na) {
    if (na != 4) return refuse("bind: 4 addresses");
    void *f[4];
    for (int i = 0; i < 4; i++) {
        f[i] = PyLong_AsVoidPtr(a[i]);
        if (PyErr_Occurred()) return nullptr;
    }
    f_batch_set = (decltype(f_batch_set))f[0]; f_append = (decltype(f_append))f[1]; f_decode_step = (decltype(f_decode_step))f[2]; f_prefill = (decltype(f_prefill))f[3];
    Py_RETURN_NONE;
}

#define METHOD(name) {#name, (PyCFunction)(void (*)(void))guarded<name>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {METHOD(bind), METHOD(batch_set), METHOD(append), METHOD(decode_step), METHOD(prefill), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods};

} /* namespace */

/* `torch_key`: the torch it was built for; the loader compares */
PyMODINIT_FUNC PyInit__native(void) {
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch_key", HY3A_TORCH_KEY)) Py_CLEAR(m);
    return m;
}
