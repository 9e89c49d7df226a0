// The host side of the Python calls that a serving or training loop makes per step, in native code: argument checks,
// output tensors, the current stream and the call into libztattn.so.
//
// Written in Python the same work took 10-20 us a call (a torch.Size per shape compared, a device context, a ctypes call
// of a dozen converted arguments), more than the kernels of a small step: a decode step of one sequence was 37 us of
// host time over 20 us of kernels.  Here it is a few us plus the launches: 2.7 us an append, 4.2 a short decode step, 6.0 a
// forward of one launch, 6.5 of two (8.5 with its planes kept and the log-sum-exp), 13.4 a backward of three (one output to four allocated).
//
// Every function answers None when the arguments are not the plain case it handles (wrong shapes, types or devices
// included) and False when the library refused the call; the Python caller then takes its own path, which raises the
// error that belongs to the arguments.  Nothing is computed here.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>

#include "../../../include/zt_attn.h"

namespace {

const at::Tensor *tensor(PyObject *o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// A contiguous f32 CUDA tensor of `dims` dimensions on q's device (null q: any).
const at::Tensor *f32(PyObject *o, int dims, const at::Tensor *q = nullptr) {
    const at::Tensor *t = tensor(o);
    if (!t || !t->is_cuda() || t->scalar_type() != at::kFloat || t->dim() != dims || !t->is_contiguous()) return nullptr;
    return q && t->device() != q->device() ? nullptr : t;
}
bool is_shape(const at::Tensor &t, std::initializer_list<int64_t> shape) { return t.sizes() == at::IntArrayRef(shape); }
bool ints(PyObject *const *args, int n, int *out) {
    for (int i = 0; i < n; ++i) {
        const long v = PyLong_AsLong(args[i]);
        if (v == -1 && PyErr_Occurred()) {
            PyErr_Clear();
            return false;
        }
        if (v < -2147483647L || v > 2147483647L) return false;
        out[i] = (int)v;
    }
    return true;
}
template <typename F>
int without_gil(F &&call) {
    int rc;
    Py_BEGIN_ALLOW_THREADS;
    rc = call();
    Py_END_ALLOW_THREADS;
    return rc;
}
zt_stream_t stream_of(const at::Tensor &t) { return (zt_stream_t)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
const float *in(const at::Tensor *t) { return t->const_data_ptr<float>(); }
float *out_of(const at::Tensor &t) { return t.data_ptr<float>(); }
// nullptr for None; `*ok` false when it is neither None nor a CUDA tensor of at least n bytes.
void *scratch(PyObject *o, size_t n, const at::Tensor &on, bool *ok) {
    *ok = true;
    if (o == Py_None) return nullptr;
    const at::Tensor *t = tensor(o);
    *ok = t && t->is_cuda() && t->device() == on.device() && (size_t)t->nbytes() >= n;
    return *ok ? t->data_ptr() : nullptr;
}
PyObject *none() { Py_RETURN_NONE; }
PyObject *refused() { Py_RETURN_FALSE; }
// A tuple of tensors; an undefined one becomes None.  `token`: one more element.
PyObject *pack(std::initializer_list<at::Tensor> tensors, const unsigned long long *token = nullptr) {
    const Py_ssize_t n = (Py_ssize_t)tensors.size();
    PyObject *r = PyTuple_New(n + (token ? 1 : 0));
    if (!r) return nullptr;
    Py_ssize_t i = 0;
    for (const at::Tensor &t : tensors) PyTuple_SET_ITEM(r, i++, t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None));
    if (token) PyTuple_SET_ITEM(r, n, PyLong_FromUnsignedLongLong(*token));
    return r;
}

// q [B, T, H D], k and v [B, T, G D] that agree.
struct Qkv {
    const at::Tensor *q, *k, *v;
    int B, T, H, G, D;
    bool take(PyObject *const *args) {
        int n[3];
        q = f32(args[0], 3);
        if (!q || !(k = f32(args[1], 3, q)) || !(v = f32(args[2], 3, q)) || !ints(args + 3, 3, n)) return false;
        H = n[0], G = n[1], D = n[2];
        if (H < 1 || G < 1 || D < 1 || H % G != 0 || q->size(0) < 1 || q->size(0) > 65535 || q->size(1) < 1 || q->size(1) > 2147483647LL) return false;
        B = (int)q->size(0), T = (int)q->size(1);
        return q->size(2) == (int64_t)H * D && is_shape(*k, {B, T, (int64_t)G * D}) && k->sizes() == v->sizes();
    }
};

// attention_forward(q, k, v, H, G, D, want_lse, keep_buffer | None, keep_bytes) -> (out, lse | None, token)
PyObject *attention_forward(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    Qkv s;
    if (n_args != 9 || !s.take(args)) return none();
    const size_t keep_bytes = PyLong_AsSize_t(args[8]);
    if (PyErr_Occurred()) return nullptr;
    bool ok;
    void *keep = scratch(args[7], keep_bytes, *s.q, &ok);
    if (!ok) return none();
    const int want_lse = PyObject_IsTrue(args[6]);
    if (want_lse < 0) return nullptr;
    const bool keeps = args[7] != Py_None;
    const c10::cuda::CUDAGuard guard(s.q->device());
    const at::Tensor out = at::empty(s.q->sizes(), s.q->options());
    const at::Tensor lse = want_lse ? at::empty({s.B, s.T, s.H}, s.q->options()) : at::Tensor();
    unsigned long long token = 0;
    const zt_stream_t stream = stream_of(*s.q);
    const int rc = without_gil([&] {
        float *l = lse.defined() ? out_of(lse) : nullptr;
        if (!keeps) return zt_attn_forward_batched(in(s.q), in(s.k), in(s.v), out_of(out), l, s.B, s.T, s.H, s.G, s.D, stream);
        return zt_attn_forward_batched_keep(in(s.q), in(s.k), in(s.v), out_of(out), l, keep_bytes ? keep : nullptr, keep_bytes,
                                            s.B, s.T, s.H, s.G, s.D, stream, &token);
    });
    return rc != 0 ? refused() : pack({out, lse}, &token);
}

// attention_backward(q, k, v, H, G, D, out, lse, dout, buffer | None, bytes, token) -> (dq, dk, dv)
PyObject *attention_backward(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    Qkv s;
    if (n_args != 12 || !s.take(args)) return none();
    const at::Tensor *out = f32(args[6], 3, s.q), *lse = f32(args[7], 3, s.q), *dout = f32(args[8], 3, s.q);
    if (!out || !lse || !dout || out->sizes() != s.q->sizes() || dout->sizes() != s.q->sizes() || !is_shape(*lse, {s.B, s.T, s.H}))
        return none();
    const size_t bytes = PyLong_AsSize_t(args[10]);
    const unsigned long long token = PyLong_AsUnsignedLongLong(args[11]);
    if (PyErr_Occurred()) return nullptr;
    bool ok;
    void *ws = scratch(args[9], bytes, *s.q, &ok);
    if (!ok) return none();
    const c10::cuda::CUDAGuard guard(s.q->device());
    const at::Tensor dq = at::empty(s.q->sizes(), s.q->options()), dk = at::empty(s.k->sizes(), s.k->options());
    const at::Tensor dv = at::empty(s.v->sizes(), s.v->options()), delta = at::empty(lse->sizes(), lse->options());
    const zt_stream_t stream = stream_of(*s.q);
    const int rc = without_gil([&] {
        return zt_attn_backward_batched_kept(in(s.q), in(s.k), in(s.v), in(out), in(lse), in(dout), out_of(dq), out_of(dk), out_of(dv),
                                             out_of(delta), bytes ? ws : nullptr, bytes, s.B, s.T, s.H, s.G, s.D, stream, token);
    });
    return rc != 0 ? refused() : pack({dq, dk, dv});
}

// block_forward(q, k, v, H, G, D, wo, rope_buffer, rope_bytes, proj_buffer, proj_bytes, pos, theta) -> (y, ctx, lse, token)
PyObject *block_forward(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    Qkv s;
    int pos;
    if (n_args != 13 || !s.take(args) || !ints(args + 11, 1, &pos)) return none();
    const at::Tensor *wo = f32(args[6], 2, s.q);
    if (!wo || wo->size(0) != (int64_t)s.H * s.D || wo->size(1) > 2147483647LL) return none();
    const size_t rope_bytes = PyLong_AsSize_t(args[8]), proj_bytes = PyLong_AsSize_t(args[10]);
    const double theta = PyFloat_AsDouble(args[12]);
    if (PyErr_Occurred()) return nullptr;
    bool ok, ok2;
    void *rope = scratch(args[7], rope_bytes, *s.q, &ok), *proj = scratch(args[9], proj_bytes, *s.q, &ok2);
    if (!ok || !ok2) return none();
    const int n = (int)wo->size(1);
    const c10::cuda::CUDAGuard guard(s.q->device());
    const at::Tensor ctx = at::empty(s.q->sizes(), s.q->options()), lse = at::empty({s.B, s.T, s.H}, s.q->options());
    const at::Tensor y = at::empty({s.B, s.T, n}, s.q->options());
    unsigned long long token = 0;
    const zt_stream_t stream = stream_of(*s.q);
    const int rc = without_gil([&] {
        return zt_attn_block_forward(in(s.q), in(s.k), in(s.v), in(wo), out_of(ctx), out_of(lse), out_of(y), rope, rope_bytes, proj,
                                     proj_bytes, s.B, s.T, s.H, s.G, s.D, n, pos, theta, stream, &token);
    });
    return rc != 0 ? refused() : pack({y, ctx, lse}, &token);
}

// block_backward(q, k, v, H, G, D, wo, ctx, lse, dy, dwo, rope_buffer, rope_bytes, proj_buffer, proj_bytes, pos, theta, token)
// -> (dq, dk, dv), dwo added to.  The projection's gradients, then those of the rotated attention.
PyObject *block_backward(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    Qkv s;
    int pos;
    if (n_args != 18 || !s.take(args) || !ints(args + 15, 1, &pos)) return none();
    const at::Tensor *wo = f32(args[6], 2, s.q), *ctx = f32(args[7], 3, s.q), *lse = f32(args[8], 3, s.q);
    const at::Tensor *dy = f32(args[9], 3, s.q), *dwo = f32(args[10], 2, s.q);
    if (!wo || !ctx || !lse || !dy || !dwo || wo->size(0) != (int64_t)s.H * s.D || wo->size(1) > 2147483647LL || dwo->sizes() != wo->sizes() ||
        ctx->sizes() != s.q->sizes() || !is_shape(*lse, {s.B, s.T, s.H}) || !is_shape(*dy, {s.B, s.T, wo->size(1)}))
        return none();
    const size_t rope_bytes = PyLong_AsSize_t(args[12]), proj_bytes = PyLong_AsSize_t(args[14]);
    const double theta = PyFloat_AsDouble(args[16]);
    const unsigned long long token = PyLong_AsUnsignedLongLong(args[17]);
    if (PyErr_Occurred()) return nullptr;
    bool ok, ok2;
    void *rope = scratch(args[11], rope_bytes, *s.q, &ok), *proj = scratch(args[13], proj_bytes, *s.q, &ok2);
    if (!ok || !ok2) return none();
    const c10::cuda::CUDAGuard guard(s.q->device());
    const at::Tensor dctx = at::empty(s.q->sizes(), s.q->options()), dq = at::empty(s.q->sizes(), s.q->options());
    const at::Tensor dk = at::empty(s.k->sizes(), s.k->options()), dv = at::empty(s.v->sizes(), s.v->options());
    const at::Tensor delta = at::empty(lse->sizes(), lse->options());
    const zt_stream_t stream = stream_of(*s.q);
    const int rc = without_gil([&] {
        if (zt_proj_backward(in(ctx), in(wo), in(dy), out_of(dctx), out_of(*dwo), proj, proj_bytes, s.B, s.T, s.H * s.D, (int)wo->size(1), stream))
            return 1;
        return zt_attn_backward_rope_batched(in(s.q), in(s.k), in(s.v), in(ctx), in(lse), in(&dctx), out_of(dq), out_of(dk), out_of(dv),
                                             out_of(delta), rope, rope_bytes, s.B, s.T, s.H, s.G, s.D, pos, theta, stream, token);
    });
    return rc != 0 ? refused() : pack({dq, dk, dv});
}

// forward_at(q, k, v, out (the holder's flat buffers), t, H, G, D, group_q, max_tile, q_offset, n_keys) -> True
PyObject *forward_at(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    int n[8];
    if (n_args != 12 || !ints(args + 4, 8, n)) return none();
    const at::Tensor *q = f32(args[0], 1), *k, *v, *out;
    if (!q || !(k = f32(args[1], 1, q)) || !(v = f32(args[2], 1, q)) || !(out = f32(args[3], 1, q))) return none();
    const int64_t wq = (int64_t)n[1] * n[3], wk = (int64_t)n[2] * n[3];
    if (n[0] < 1 || n[7] < 1 || wq < 1 || wk < 1 || n[0] * wq > q->numel() || n[0] * wq > out->numel() || n[7] * wk > k->numel() || n[7] * wk > v->numel())
        return none();
    const c10::cuda::CUDAGuard guard(q->device());
    const zt_stream_t stream = stream_of(*q);
    const int rc = without_gil([&] {
        return zt_attn_forward(in(q), in(k), in(v), out_of(*out), n[0], n[1], n[2], n[3], n[4], n[5], n[6], n[7], stream);
    });
    if (rc != 0) return refused();
    Py_RETURN_TRUE;
}

// decode(q, k_cache, v_cache, n_keys, H, G, D, buffer, bytes, out | None, want_lse) -> (out, lse | None)
PyObject *decode(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    int n[3];
    if (n_args != 11 || !ints(args + 4, 3, n)) return none();
    const int H = n[0], G = n[1], D = n[2];
    const at::Tensor *q = f32(args[0], 2), *k, *v, *nk = tensor(args[3]), *given = nullptr;
    if (!q || !(k = f32(args[1], 3, q)) || !(v = f32(args[2], 3, q)) || !nk || H < 1 || G < 1 || D < 1 || H % G != 0) return none();
    const int64_t B = k->size(0), n_ctx = k->size(1);
    if (B < 1 || B > 65535 || n_ctx < 1 || n_ctx > 2147483647LL || !is_shape(*q, {B, (int64_t)H * D}) || k->size(2) != (int64_t)G * D ||
        k->sizes() != v->sizes() || !nk->is_cuda() || nk->device() != q->device() || nk->scalar_type() != at::kInt ||
        !is_shape(*nk, {B}) || !nk->is_contiguous())
        return none();
    if (args[9] != Py_None && (!(given = f32(args[9], 2, q)) || given->sizes() != q->sizes())) return none();
    const size_t bytes = PyLong_AsSize_t(args[8]);
    if (PyErr_Occurred()) return nullptr;
    bool ok;
    void *ws = scratch(args[7], bytes, *q, &ok);
    if (!ok || !ws) return none();
    const int want_lse = PyObject_IsTrue(args[10]);
    if (want_lse < 0) return nullptr;
    const c10::cuda::CUDAGuard guard(q->device());
    const at::Tensor out = given ? *given : at::empty(q->sizes(), q->options());
    const at::Tensor lse = want_lse ? at::empty({B, (int64_t)H}, q->options()) : at::Tensor();
    const zt_stream_t stream = stream_of(*q);
    const int rc = without_gil([&] {
        return zt_attn_decode(in(q), in(k), in(v), nk->const_data_ptr<int>(), out_of(out), lse.defined() ? out_of(lse) : nullptr, ws, bytes,
                              (int)B, (int)n_ctx, H, G, D, stream);
    });
    return rc != 0 ? refused() : pack({out, lse});
}

// kv_append(k, v, len, k_rows, v_rows, full_count) -> True
PyObject *kv_append(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    if (n_args != 6) return none();
    const at::Tensor *k = f32(args[0], 3), *v, *kr, *vr, *len = tensor(args[2]), *full = tensor(args[5]);
    if (!k || !(v = f32(args[1], 3, k)) || !(kr = f32(args[3], 2, k)) || !(vr = f32(args[4], 2, k)) || !len || !full) return none();
    const int64_t B = k->size(0), n_ctx = k->size(1), width = k->size(2);
    for (const at::Tensor *t : {len, full})
        if (!t->is_cuda() || t->device() != k->device() || t->scalar_type() != at::kInt || t->dim() != 1 || !t->is_contiguous()) return none();
    if (!is_shape(*kr, {B, width}) || kr->sizes() != vr->sizes() || len->size(0) != B || full->size(0) < 1 || k->sizes() != v->sizes() ||
        B < 1 || B > 2147483647LL || n_ctx > 2147483647LL || width > 2147483647LL)
        return none();
    const c10::cuda::CUDAGuard guard(k->device());
    const zt_stream_t stream = stream_of(*k);
    const int rc = without_gil([&] {
        return zt_kv_append(out_of(*k), out_of(*v), len->data_ptr<int>(), in(kr), in(vr), full->data_ptr<int>(), (int)B, (int)n_ctx, 1,
                            (int)width, stream);
    });
    if (rc != 0) return refused();
    Py_RETURN_TRUE;
}

// Out of memory: the caller's own path meets it again and raises torch's error for it.
template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
PyObject *guarded(PyObject *self, PyObject *const *args, Py_ssize_t n) {
    try {
        return F(self, args, n);
    } catch (const c10::OutOfMemoryError &) {
        return none();
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

#define ZT_METHOD(f) {#f, (PyCFunction)(void *)guarded<f>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ZT_METHOD(attention_forward), ZT_METHOD(attention_backward), ZT_METHOD(block_forward), ZT_METHOD(block_backward),
                         ZT_METHOD(forward_at), ZT_METHOD(decode), ZT_METHOD(kv_append), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_zt_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__zt_torch(void) { return PyModule_Create(&module); }
