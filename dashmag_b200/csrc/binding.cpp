// The entry points' host side in native code, for calls as a program makes them: plain CUDA tensors on the current device,
// in the layouts the library reads in place.  A short call is bound by its host time - one decoding step spends 13 us on the
// device and spent 24 in Python around it: the parameter struct, four allocations, thirteen arguments through ctypes.
//
// Every function either makes the whole call - fills the parameters, allocates the outputs and the scratch, calls the C ABI on
// the current stream - and returns the outputs, or an int, the C ABI's error code; or it returns None without having done
// anything, and the Python code it stands in front of makes the call or raises what there is to raise.  None is the answer to
// everything out of the ordinary: a tensor of another kind or device, a shape or dtype the Python side would refuse or copy, a
// number its C type does not hold, a mode or a transform that wants to see the allocations.
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/SmallVector.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/PyInterpreter.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "../../include/dash_attn.h"

namespace {

// The C ABI of the library that is loaded (use(), below).
struct Library {
    decltype(&dash_attn_forward_workspace) forward_workspace;
    decltype(&dash_attn_forward) forward;
    decltype(&dash_attn_backward_workspace) backward_workspace;
    decltype(&dash_attn_backward) backward;
    decltype(&dash_attn_decode_workspace) decode_workspace;
    decltype(&dash_attn_decode) decode;
    decltype(&dash_attn_decode_append) decode_append;
    decltype(&dash_attn_decode_append_rope_workspace) decode_append_rope_workspace;
    decltype(&dash_attn_decode_append_rope) decode_append_rope;
    decltype(&dash_sample_workspace) sample_workspace;
    decltype(&dash_sample) sample;
} lib;

// ---- what a call hands over ------------------------------------------------------------------------
// The tensors a call's parameters point into that are not its arguments: an attribute may be a property whose tensor nobody else
// holds, and what a mask or a Rope holds another thread may replace while the library is called without the interpreter's lock.
using Held = c10::SmallVector<at::Tensor, 2>;

struct Ref {   // an owned reference
    PyObject *p;
    explicit Ref(PyObject *o) : p(o) {}
    ~Ref() { Py_XDECREF(p); }
    Ref(const Ref &) = delete;
    Ref &operator=(const Ref &) = delete;
};

// Allocations and the call into the library without the interpreter's lock, as torch.empty and ctypes make them: an allocation may
// wait for the driver or for memory to be given back, a launch for room in the GPU's queue.
struct Unlocked {
    PyThreadState *state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }   // on the way out of an exception too: it is raised with the lock
};
template <typename F> int unlocked(F call) {
    Unlocked u;
    return call();
}

PyObject *nothing_done() {
    PyErr_Clear();
    Py_RETURN_NONE;
}

// Whether a torch-function mode would see what the Python side asks torch for.  A default device is such a mode too, but one that has
// nothing to say about allocations whose device is given.
PyObject *default_device_mode = nullptr;   // its type (use(), below)
bool watched() {
    if (!at::impl::torch_function_mode_enabled()) return false;
    for (int64_t i = 0; i < at::impl::PythonTorchFunctionTLS::stack_len(); ++i)
        if (reinterpret_cast<PyObject *>(Py_TYPE(at::impl::PythonTorchFunctionTLS::get_stack_at(i)->ptr(getPyInterpreter()))) != default_device_mode) return true;
    return false;
}

// A plain strided CUDA tensor: torch.Tensor or Parameter itself, no wrapper, no mode that watches, of functions or of dispatch.
const at::Tensor *plain(PyObject *o) {
    if (!THPVariable_CheckExact(o) || watched()) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || at::isTensorSubclassLike(t)) return nullptr;
    return &t;
}

int code_of(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return DASH_ATTN_F32;
        case at::kBFloat16: return DASH_ATTN_BF16;
        case at::kHalf: return DASH_ATTN_F16;
        default: return -1;
    }
}
int index_bytes(at::ScalarType t) { return t == at::kInt ? 4 : t == at::kLong ? 8 : 0; }

bool fits32(const at::Tensor &t) {
    for (int64_t n : t.sizes())
        if (n > INT32_MAX) return false;
    return true;
}
void *pointer(const at::Tensor &t) { return t.numel() == 0 ? nullptr : t.data_ptr(); }

bool attr_true(PyObject *o, const char *name, int32_t *out) {
    Ref v(PyObject_GetAttrString(o, name));
    if (!v.p) return false;
    const int r = PyObject_IsTrue(v.p);
    *out = r;
    return r >= 0;
}
bool int64_of(PyObject *o, int64_t *out) {
    if (!PyLong_Check(o)) return false;
    int overflow = 0;
    *out = PyLong_AsLongLongAndOverflow(o, &overflow);
    return overflow == 0 && !(*out == -1 && PyErr_Occurred());
}
bool float_of(PyObject *o, float *out) {
    if (!PyFloat_Check(o) && !PyLong_Check(o)) return false;
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) return false;
    if (std::isfinite(d) && std::fabs(d) > FLT_MAX) return false;
    *out = (float)d;
    return true;
}
bool side_of(PyObject *window, const char *name, int64_t *out) {
    Ref v(PyObject_GetAttrString(window, name));
    if (!v.p) return false;
    if (v.p == Py_None) {
        *out = -1;
        return true;
    }
    return int64_of(v.p, out);
}
// options.window and options.scale.
bool window_and_scale(PyObject *options, int32_t *has_window, int64_t *left, int64_t *right, int32_t *has_scale, float *scale) {
    Ref w(PyObject_GetAttrString(options, "window"));
    if (!w.p) return false;
    *has_window = w.p != Py_None;
    *left = *right = 0;
    if (*has_window && (!side_of(w.p, "left", left) || !side_of(w.p, "right", right))) return false;
    Ref s(PyObject_GetAttrString(options, "scale"));
    if (!s.p) return false;
    *has_scale = s.p != Py_None;
    *scale = 0.f;
    return !*has_scale || float_of(s.p, scale);
}

bool on_current_device(const at::Tensor &t) { return t.get_device() == c10::cuda::current_device(); }
dash_attn_stream_t stream_of(const at::Tensor &t) {
    return reinterpret_cast<dash_attn_stream_t>(c10::cuda::getCurrentCUDAStream(t.get_device()).stream());
}
at::Tensor scratch(size_t bytes, const at::Tensor &like) {
    return bytes ? at::empty({(int64_t)bytes}, like.options().dtype(at::kByte).requires_grad(false)) : at::Tensor();
}
at::Tensor fresh(at::IntArrayRef sizes, const at::Tensor &like, at::ScalarType dtype) {
    return at::empty(sizes, like.options().dtype(dtype).requires_grad(false));
}
void strides(int64_t *to, const at::Tensor &t) {
    for (int i = 0; i < t.dim(); ++i) to[i] = t.stride(i);
}
PyObject *wrapped(std::initializer_list<at::Tensor> outs) {
    Ref tuple(PyTuple_New((Py_ssize_t)outs.size()));
    if (!tuple.p) return nullptr;
    Py_ssize_t i = 0;
    for (const at::Tensor &t : outs) {
        PyObject *o = THPVariable_Wrap(t);
        if (!o) return nullptr;
        PyTuple_SET_ITEM(tuple.p, i++, o);
    }
    Py_INCREF(tuple.p);
    return tuple.p;
}

// ---- training --------------------------------------------------------------------------------------
// The parameters of a training call; `held` keeps what they point to.  False: not for us.
bool train_params(dash_attn_params &p, Held &held, const at::Tensor &q, const at::Tensor &k, const at::Tensor &v, PyObject *mask, PyObject *options) {
    if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || !fits32(q) || !fits32(k) || !fits32(v)) return false;
    const int code = code_of(q.scalar_type());
    if (code < 0 || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return false;
    if (v.size(0) != k.size(0) || k.get_device() != q.get_device() || v.get_device() != q.get_device() || !on_current_device(q)) return false;
    p.dtype = code;
    p.b = (int32_t)q.size(0); p.tq = (int32_t)q.size(1); p.hq = (int32_t)q.size(2); p.d = (int32_t)q.size(3);
    p.k_b = (int32_t)k.size(0); p.tk = (int32_t)k.size(1); p.hkv = (int32_t)k.size(2); p.k_d = (int32_t)k.size(3);
    p.v_tk = (int32_t)v.size(1); p.v_hkv = (int32_t)v.size(2); p.v_d = (int32_t)v.size(3);
    strides(p.q_stride, q);
    strides(p.k_stride, k);
    strides(p.v_stride, v);
    Ref kind(PyObject_GetAttrString(mask, "kind"));
    if (!kind.p || !PyUnicode_Check(kind.p)) return false;
    if (PyUnicode_CompareWithASCIIString(kind.p, "none") == 0) {
        p.mask_kind = DASH_ATTN_MASK_NONE;
    } else if (PyUnicode_CompareWithASCIIString(kind.p, "key_padding") == 0) {
        Ref o(PyObject_GetAttrString(mask, "key_padding_mask"));
        const at::Tensor *m = o.p ? plain(o.p) : nullptr;
        if (!m || m->dim() != 2 || !fits32(*m) || m->get_device() != q.get_device()) return false;
        const at::ScalarType s = m->scalar_type();
        p.key_padding_elem_bytes = s == at::kBool || s == at::kByte || s == at::kChar ? 1 : s == at::kInt ? 4 : 0;
        if (p.key_padding_elem_bytes == 0) return false;
        p.mask_kind = DASH_ATTN_MASK_KEY_PADDING;
        held.push_back(*m);
        p.key_padding = m->data_ptr();
        for (int i = 0; i < 2; ++i) {
            p.key_padding_shape[i] = (int32_t)m->size(i);
            p.key_padding_stride[i] = m->stride(i);
        }
    } else if (PyUnicode_CompareWithASCIIString(kind.p, "packed") == 0) {
        Ref oq(PyObject_GetAttrString(mask, "cu_seqlens_q")), ok(PyObject_GetAttrString(mask, "cu_seqlens_k"));
        const at::Tensor *cq = oq.p ? plain(oq.p) : nullptr, *ck = ok.p ? plain(ok.p) : nullptr;
        if (!cq || !ck || cq->dim() != 1 || ck->dim() != 1 || cq->scalar_type() != ck->scalar_type() || !fits32(*cq) || !fits32(*ck)) return false;
        if (cq->get_device() != q.get_device() || ck->get_device() != q.get_device() || !cq->is_contiguous() || !ck->is_contiguous()) return false;
        p.index_elem_bytes = index_bytes(cq->scalar_type());
        if (p.index_elem_bytes == 0) return false;
        p.mask_kind = DASH_ATTN_MASK_PACKED;
        held.push_back(*cq);
        held.push_back(*ck);
        p.cu_seqlens_q = cq->data_ptr();
        p.cu_seqlens_k = ck->data_ptr();
        p.cu_seqlens_q_len = (int32_t)cq->size(0);
        p.cu_seqlens_k_len = (int32_t)ck->size(0);
    } else {
        return false;
    }
    return window_and_scale(options, &p.has_window, &p.window_left, &p.window_right, &p.has_scale, &p.scale) &&
           attr_true(options, "causal", &p.causal) && attr_true(options, "deterministic", &p.deterministic);
}

// forward(query, key, value, mask, options) -> (out, lse)
PyObject *forward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 5) return nothing_done();
    const at::Tensor *q = plain(args[0]), *k = plain(args[1]), *v = plain(args[2]);
    dash_attn_params p{};
    Held held;
    if (!q || !k || !v || !train_params(p, held, *q, *k, *v, args[3], args[4])) return nothing_done();
    at::Tensor out, lse;
    const int rc = unlocked([&] {
        out = fresh(q->sizes(), *q, q->scalar_type());
        lse = fresh(q->sizes().slice(0, 3), *q, at::kFloat);
        const size_t need = lib.forward_workspace(&p);
        at::Tensor ws = scratch(need, *q);
        return lib.forward(&p, pointer(*q), pointer(*k), pointer(*v), pointer(out), static_cast<float *>(pointer(lse)), need ? ws.data_ptr() : nullptr, need,
                           stream_of(*q));
    });
    if (rc != DASH_ATTN_OK) return PyLong_FromLong(rc);
    return wrapped({out, lse});
    END_HANDLE_TH_ERRORS
}

// backward(query, key, value, output, lse, grad_output, mask, options) -> (dq, dk, dv)
PyObject *backward(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8) return nothing_done();
    const at::Tensor *q = plain(args[0]), *k = plain(args[1]), *v = plain(args[2]), *o = plain(args[3]), *lse = plain(args[4]), *g = plain(args[5]);
    dash_attn_params p{};
    Held held;
    if (!q || !k || !v || !o || !lse || !g || !train_params(p, held, *q, *k, *v, args[6], args[7])) return nothing_done();
    const int device = (int)q->get_device();
    if (o->sizes() != q->sizes() || g->sizes() != q->sizes() || lse->sizes() != q->sizes().slice(0, 3) || o->scalar_type() != q->scalar_type() ||
        g->scalar_type() != q->scalar_type() || lse->scalar_type() != at::kFloat || !lse->is_contiguous() || o->get_device() != device ||
        g->get_device() != device || lse->get_device() != device)
        return nothing_done();
    strides(p.o_stride, *o);
    strides(p.do_stride, *g);
    at::Tensor dq, dk, dv;
    const int rc = unlocked([&] {
        dq = fresh(q->sizes(), *q, q->scalar_type());
        dk = fresh(k->sizes(), *q, q->scalar_type());
        dv = fresh(v->sizes(), *q, q->scalar_type());
        const size_t need = lib.backward_workspace(&p);
        at::Tensor ws = scratch(need, *q);
        return lib.backward(&p, pointer(*q), pointer(*k), pointer(*v), pointer(*o), static_cast<const float *>(pointer(*lse)), pointer(*g), pointer(dq),
                            pointer(dk), pointer(dv), need ? ws.data_ptr() : nullptr, need, stream_of(*q));
    });
    if (rc != DASH_ATTN_OK) return PyLong_FromLong(rc);
    return wrapped({dq, dk, dv});
    END_HANDLE_TH_ERRORS
}

// ---- decoding --------------------------------------------------------------------------------------
bool decode_params(dash_attn_decode_params &p, const at::Tensor &q, const at::Tensor &k, const at::Tensor &v, PyObject *lengths, PyObject *options) {
    if (q.dim() != 3 || k.dim() != 4 || v.dim() != 4 || !fits32(q) || !fits32(k) || !fits32(v)) return false;
    const int code = code_of(q.scalar_type());
    if (code < 0 || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return false;
    if (k.get_device() != q.get_device() || v.get_device() != q.get_device() || !on_current_device(q)) return false;
    p.dtype = code;
    p.b = (int32_t)q.size(0); p.hq = (int32_t)q.size(1); p.d = (int32_t)q.size(2);
    p.k_b = (int32_t)k.size(0); p.s = (int32_t)k.size(1); p.hkv = (int32_t)k.size(2); p.k_d = (int32_t)k.size(3);
    p.v_b = (int32_t)v.size(0); p.v_s = (int32_t)v.size(1); p.v_hkv = (int32_t)v.size(2); p.v_d = (int32_t)v.size(3);
    strides(p.q_stride, q);
    strides(p.k_stride, k);
    strides(p.v_stride, v);
    if (lengths != Py_None) {
        const at::Tensor *l = plain(lengths);
        if (!l || l->dim() != 1 || !fits32(*l) || !l->is_contiguous() || l->get_device() != q.get_device()) return false;
        p.lengths_elem_bytes = index_bytes(l->scalar_type());
        if (p.lengths_elem_bytes == 0) return false;
        p.lengths = l->data_ptr();
        p.lengths_len = (int32_t)l->size(0);
    }
    int64_t right;
    return window_and_scale(options, &p.has_window, &p.window_left, &right, &p.has_scale, &p.scale);
}

// A new row of the cache, [B, Hkv, D].
bool new_row(const at::Tensor *t, const at::Tensor &k) {
    return t && t->dim() == 3 && t->size(0) == k.size(0) && t->size(1) == k.size(2) && t->size(2) == k.size(3) && t->scalar_type() == k.scalar_type() &&
           t->is_contiguous() && t->get_device() == k.get_device();
}

// decode(query, key, value, cache_lengths, options) -> (out,)
PyObject *decode(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 5) return nothing_done();
    const at::Tensor *q = plain(args[0]), *k = plain(args[1]), *v = plain(args[2]);
    dash_attn_decode_params p{};
    if (!q || !k || !v || !decode_params(p, *q, *k, *v, args[3], args[4])) return nothing_done();
    at::Tensor out;
    const int rc = unlocked([&] {
        out = fresh(q->sizes(), *q, q->scalar_type());
        const size_t need = lib.decode_workspace(&p);
        at::Tensor ws = scratch(need, *q);
        return lib.decode(&p, pointer(*q), pointer(*k), pointer(*v), pointer(out), need ? ws.data_ptr() : nullptr, need, stream_of(*q));
    });
    if (rc != DASH_ATTN_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// decode_append(query, new_key, new_value, key, value, cache_lengths, options) -> out
PyObject *decode_append(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 7) return nothing_done();
    const at::Tensor *q = plain(args[0]), *nk = plain(args[1]), *nv = plain(args[2]), *k = plain(args[3]), *v = plain(args[4]);
    dash_attn_decode_params p{};
    if (!q || !k || !v || args[5] == Py_None || !decode_params(p, *q, *k, *v, args[5], args[6]) || !new_row(nk, *k) || !new_row(nv, *k)) return nothing_done();
    at::Tensor out;
    const int rc = unlocked([&] {
        out = fresh(q->sizes(), *q, q->scalar_type());
        const size_t need = lib.decode_workspace(&p);
        at::Tensor ws = scratch(need, *q);
        return lib.decode_append(&p, pointer(*q), pointer(*nk), pointer(*nv), pointer(*k), pointer(*v), pointer(out), need ? ws.data_ptr() : nullptr, need,
                                 stream_of(*q));
    });
    if (rc != DASH_ATTN_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// A Rope's tables for tensors of `dtype` with `d` features; false: not for us.
bool rope_tables(dash_rope_tables &r, Held &held, PyObject *rope, at::ScalarType dtype, int64_t d, const at::Tensor &near) {
    Ref dt(PyObject_GetAttrString(rope, "dtype")), dim(PyObject_GetAttrString(rope, "dim")), len(PyObject_GetAttrString(rope, "_len"));
    Ref oc(PyObject_GetAttrString(rope, "cos")), os(PyObject_GetAttrString(rope, "sin"));
    if (!dt.p || !dim.p || !len.p || !oc.p || !os.p || !THPDtype_Check(dt.p)) return false;
    if (reinterpret_cast<THPDtype *>(dt.p)->scalar_type != dtype) return false;
    const at::Tensor *c = plain(oc.p), *s = plain(os.p);
    int64_t features;
    if (!c || !s || !int64_of(dim.p, &features) || !int64_of(len.p, &r.len) || features > d || features > INT32_MAX) return false;
    if (c->get_device() != near.get_device() || s->get_device() != near.get_device()) return false;
    r.dtype = code_of(dtype);
    r.dim = (int32_t)features;
    held.push_back(*c);
    held.push_back(*s);
    r.cos = pointer(*c);
    r.sin = pointer(*s);
    return r.dtype >= 0;
}

// decode_append_rope(rope, query, new_key, new_value, key, value, cache_lengths, options) -> out; rotated at the lengths
PyObject *decode_append_rope(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8) return nothing_done();
    const at::Tensor *q = plain(args[1]), *nk = plain(args[2]), *nv = plain(args[3]), *k = plain(args[4]), *v = plain(args[5]);
    dash_attn_decode_params p{};
    dash_rope_tables r{};
    Held held;
    if (!q || !k || !v || args[6] == Py_None || !decode_params(p, *q, *k, *v, args[6], args[7]) || !new_row(nk, *k) || !new_row(nv, *k)) return nothing_done();
    if (q->stride(2) != 1 || !rope_tables(r, held, args[0], q->scalar_type(), q->size(2), *q)) return nothing_done();
    at::Tensor out;
    const int rc = unlocked([&] {
        out = fresh(q->sizes(), *q, q->scalar_type());
        const size_t need = lib.decode_append_rope_workspace(&p);
        at::Tensor ws = scratch(need, *q);
        return lib.decode_append_rope(&p, &r, nullptr, 0, pointer(*q), pointer(*nk), pointer(*nv), pointer(*k), pointer(*v), pointer(out),
                                      need ? ws.data_ptr() : nullptr, need, stream_of(*q));
    });
    if (rc != DASH_ATTN_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

// ---- sampling --------------------------------------------------------------------------------------
bool attr_u64(PyObject *o, const char *name, uint64_t *out) {
    Ref v(PyObject_GetAttrString(o, name));
    if (!v.p || !PyLong_Check(v.p)) return false;
    *out = PyLong_AsUnsignedLongLong(v.p);
    return !PyErr_Occurred();
}

// sample(logits, options) -> (tokens i64, logprob, tempered, sampling); no masked ids
PyObject *sample(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 2) return nothing_done();
    const at::Tensor *z = plain(args[0]);
    PyObject *options = args[1];
    if (!z || z->dim() != 2 || !fits32(*z) || z->stride(1) != 1 || code_of(z->scalar_type()) < 0 || !on_current_device(*z)) return nothing_done();
    dash_sample_params p{};
    p.dtype = code_of(z->scalar_type());
    p.b = (int32_t)z->size(0);
    p.v = (int32_t)z->size(1);
    p.row_stride = p.b > 1 ? z->stride(0) : z->size(1);
    Ref t(PyObject_GetAttrString(options, "temperature")), k(PyObject_GetAttrString(options, "top_k")), tp(PyObject_GetAttrString(options, "top_p"));
    Ref masked(PyObject_GetAttrString(options, "masked"));
    if (!t.p || !k.p || !tp.p || !masked.p || !float_of(t.p, &p.temperature) || !int64_of(k.p, &p.top_k) || !float_of(tp.p, &p.top_p)) return nothing_done();
    if (PyObject_Size(masked.p) != 0 || !attr_u64(options, "seed", &p.seed) || !attr_u64(options, "offset", &p.offset)) return nothing_done();
    const uint32_t no_ids = 0;
    p.masked = &no_ids;
    p.token_elem_bytes = 8;
    at::Tensor tokens, logprob, tempered, sampling;
    const int rc = unlocked([&] {
        tokens = fresh({p.b}, *z, at::kLong);
        logprob = fresh({p.b}, *z, at::kFloat);
        tempered = fresh({p.b}, *z, at::kFloat);
        sampling = fresh({p.b}, *z, at::kFloat);
        const size_t need = lib.sample_workspace(&p);
        at::Tensor ws = scratch(need, *z);
        return lib.sample(&p, pointer(*z), pointer(tokens), static_cast<float *>(pointer(logprob)), static_cast<float *>(pointer(tempered)),
                          static_cast<float *>(pointer(sampling)), need ? ws.data_ptr() : nullptr, need, stream_of(*z));
    });
    if (rc != DASH_ATTN_OK) return PyLong_FromLong(rc);
    return wrapped({tokens, logprob, tempered, sampling});
    END_HANDLE_TH_ERRORS
}

// use(addresses): the library's functions, in Library's order
PyObject *use(PyObject *, PyObject *const *args, Py_ssize_t n) {
    constexpr Py_ssize_t want = sizeof(Library) / sizeof(void *);
    if (n != want) return PyErr_Format(PyExc_TypeError, "use: %zd addresses, got %zd", want, n);
    void *at[want];
    for (Py_ssize_t i = 0; i < want; ++i) {
        at[i] = PyLong_AsVoidPtr(args[i]);
        if (!at[i]) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "use: address %zd is null", i);
    }
    memcpy(&lib, at, sizeof lib);
    if (!default_device_mode) {
        Ref module(PyImport_ImportModule("torch.utils._device"));
        if (module.p) default_device_mode = PyObject_GetAttrString(module.p, "DeviceContext");
        PyErr_Clear();   // (without it every mode watches)
    }
    Py_RETURN_NONE;
}

template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)> PyCFunction fast() {
    return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(F));
}

PyMethodDef methods[] = {
    {"use", fast<use>(), METH_FASTCALL, nullptr},
    {"forward", fast<forward>(), METH_FASTCALL, nullptr},
    {"backward", fast<backward>(), METH_FASTCALL, nullptr},
    {"decode", fast<decode>(), METH_FASTCALL, nullptr},
    {"decode_append", fast<decode_append>(), METH_FASTCALL, nullptr},
    {"decode_append_rope", fast<decode_append_rope>(), METH_FASTCALL, nullptr},
    {"sample", fast<sample>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// `torch`: the version this was built for.  Nothing of torch's is touched until a function is called.
PyMODINIT_FUNC PyInit__binding(void) {
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch", DASH_BUILT_FOR_TORCH) < 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
