// CPython binding of the C ABI for torch tensors: the per-call work of the Python operators (descriptors of the
// tensors, allocation of the outputs and the workspace, the call itself) in native code.
//
// A decode step is a few microseconds of GPU work per operator, so what a small call costs is its host path.  Built
// from ctypes structures, field by field, that path was 40 us for a WKV7 call (nine descriptors) and 170 us for the
// four calls around it in a decode step; here a descriptor is a handful of stores and an output one call into torch's
// caching allocator.
//
// The module links nothing of this library: it takes the path of the shared object to open from the package, so that
// another build of it (an instrumented one) can stand in.  Functions take positional arguments only; the package's
// public functions, with their names and defaults, sit on top.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include "rwkv7_b200.h"

namespace {

// ---- the C ABI, resolved at run time ---------------------------------------------------------

#define RWKV7_BOUND(X)                                                                                          \
    X(rwkv7_last_error_message) X(rwkv7_wkv7_workspace_bytes) X(rwkv7_fused_wkv7_pretrain)                       \
    X(rwkv7_fused_wkv7_statetune) X(rwkv7_fused_wkv7_statepass) X(rwkv7_fused_wkv7_statepass_noalloc)            \
    X(rwkv7_fused_wkv7_forward_saved) X(rwkv7_fused_wkv7_backward) X(rwkv7_fused_wkv7_backward_parallel)         \
    X(rwkv7_wkv7_training_saved_bytes) X(rwkv7_wkv7_training_workspace_bytes)                                    \
    X(rwkv7_fused_wkv7_training_forward) X(rwkv7_fused_wkv7_training_backward)                                   \
    X(rwkv7_wkv7_backward_workspace_bytes) X(rwkv7_fused_mix6) X(rwkv7_fused_mix6_stacked)                       \
    X(rwkv7_fused_addcmul) X(rwkv7_fused_addcmul5) X(rwkv7_fused_token_shift_diff)                               \
    X(rwkv7_fused_token_shift_diff_into)                                                                         \
    X(rwkv7_fused_weight_prepare) X(rwkv7_fused_gated_readout) X(rwkv7_channel_mixer_workspace_bytes)            \
    X(rwkv7_fused_channel_mixer) X(rwkv7_lm_head_ce_workspace_bytes) X(rwkv7_fused_lm_head_ce_partial)           \
    X(rwkv7_lm_head_ce_finalize)

struct Abi {
#define RWKV7_FIELD(name) decltype(&::name) name = nullptr;
    RWKV7_BOUND(RWKV7_FIELD)
#undef RWKV7_FIELD
} abi;

PyObject *g_error = nullptr;   // KernelInputsError

// Thrown when a Python exception is already set.
struct PythonError {};

[[noreturn]] void raise(PyObject *type, const char *what) {
    PyErr_SetString(type, what);
    throw PythonError{};
}

void check(int status) {
    if (status == 0) return;
    if (PyObject *e = PyObject_CallFunction(g_error, "is", status, abi.rwkv7_last_error_message())) {
        PyErr_SetObject(g_error, e);
        Py_DECREF(e);
    }
    throw PythonError{};
}

// ---- tensors -----------------------------------------------------------------------------------

int32_t dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return RWKV7_F32;
        case at::kBFloat16: return RWKV7_BF16;
        case at::kHalf: return RWKV7_F16;
        case at::kInt: return RWKV7_I32;
        case at::kLong: return RWKV7_I64;
        default: return -1;
    }
}

const at::Tensor &tensor(PyObject *o) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch tensor");
    return THPVariable_Unpack(o);
}

// The borrowed descriptor of a tensor (no copy); null for None.
struct Desc {
    rwkv7_tensor d;
    rwkv7_tensor *p = nullptr;
    Desc() = default;
    explicit Desc(const at::Tensor &t) { set(t); }
    explicit Desc(PyObject *o) { set(o); }
    Desc(const Desc &) = delete;
    Desc &operator=(const Desc &) = delete;
    void set(PyObject *o) {   // (None: the library says which tensor is missing)
        if (o != Py_None) set(tensor(o));
    }
    void set(const at::Tensor &t) {
        const int32_t dt = dtype_code(t.scalar_type());
        if (dt < 0) {
            PyErr_Format(PyExc_TypeError, "unsupported torch dtype torch.%s", c10::toString(t.scalar_type()));
            throw PythonError{};
        }
        const int64_t nd = t.dim();
        if (nd > RWKV7_MAX_DIMS) raise(PyExc_IndexError, "tensor has too many dimensions");
        d.data = t.numel() ? t.data_ptr() : nullptr;
        d.dtype = dt;
        d.device = t.is_cuda() ? t.get_device() : RWKV7_HOST;
        d.ndim = (int32_t)nd;
        d.reserved = 0;
        for (int64_t i = 0; i < RWKV7_MAX_DIMS; ++i) {
            d.shape[i] = i < nd ? t.size(i) : 0;
            d.stride[i] = i < nd ? t.stride(i) : 0;
        }
        p = &d;
    }
};

rwkv7_stream stream_of(const at::Tensor &t) {
    return t.is_cuda() ? (rwkv7_stream)c10::cuda::getCurrentCUDAStream(t.get_device()).stream() : nullptr;
}

at::Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, const at::Tensor &beside) {
    if (beside.is_cuda()) return at::Tensor(at::detail::empty_cuda(shape, dtype, beside.device(), std::nullopt));
    return at::empty(shape, beside.options().dtype(dtype).requires_grad(false));
}

at::Tensor like(const at::Tensor &t) {
    return t.is_contiguous() ? empty(t.sizes(), t.scalar_type(), t) : at::empty_like(t);
}

// The outputs of a call, each like its own tensor.  Small ones share one allocation (at 512-byte boundaries, as the allocator itself
// would place them): an output costs 0.9 us to allocate and wrap, and a decode step around WKV7 has thirteen.  Up to 1 MB
// in all, because up to there the caching allocator cuts blocks from shared 2 MB segments anyway; larger outputs stay
// separate, so that holding one of them holds no more memory than its own.  For outputs that a step uses up together: whoever keeps or saves a
// single one keeps the memory of all of the call's, up to that 1 MB.
template <typename... Like>
void outputs_like(at::Tensor *out, const Like &...tensors) {
    constexpr int n = sizeof...(Like);
    const at::Tensor *ts[n] = {&tensors...};
    constexpr size_t kAlign = 512, kMost = (size_t)1 << 20;
    size_t at_byte[n], total = 0;
    bool together = true;
    for (int i = 0; i < n; ++i) {
        const at::Tensor &t = *ts[i];
        together = together && t.is_cuda() && t.is_contiguous() && t.device() == ts[0]->device() && t.layout() == at::kStrided && t.numel() > 0;
        at_byte[i] = total;
        total += ((size_t)t.numel() * (size_t)t.element_size() + kAlign - 1) / kAlign * kAlign;
    }
    if (!together || total > kMost) {
        for (int i = 0; i < n; ++i) out[i] = like(*ts[i]);
        return;
    }
    const at::Tensor all = empty({(int64_t)total}, at::kByte, *ts[0]);
    for (int i = 0; i < n; ++i) {
        const at::Tensor &t = *ts[i];
        out[i] = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(all.storage()), all.key_set(), t.dtype());
        out[i].unsafeGetTensorImpl()->set_storage_offset((int64_t)(at_byte[i] / (size_t)t.element_size()));
        out[i].unsafeGetTensorImpl()->set_sizes_contiguous(t.sizes());
    }
}

// Scratch memory of a call: freed when the call has been enqueued, i.e. given back to the allocator's stream order.
struct Workspace {
    at::Tensor t;
    void *ptr = nullptr;
    size_t bytes = 0;
    void allocate(size_t n, const at::Tensor &beside) {
        if (n == 0) return;
        t = empty({(int64_t)n}, at::kByte, beside);
        ptr = t.data_ptr();
        bytes = n;
    }
    void given(PyObject *o) {
        const at::Tensor &w = tensor(o);
        ptr = w.data_ptr();
        bytes = (size_t)w.numel() * (size_t)w.element_size();
    }
};

// Calls into the library without the interpreter lock, as a foreign-function call does.
template <typename F>
void call(F &&f) {
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = f();
    Py_END_ALLOW_THREADS
    check(st);
}

PyObject *wrap(const at::Tensor &t) { return THPVariable_Wrap(t); }
PyObject *given_or_wrapped(PyObject *o, const at::Tensor &t) { return o != Py_None ? Py_NewRef(o) : wrap(t); }

PyObject *pair(PyObject *a, PyObject *b) {
    PyObject *r = a && b ? PyTuple_New(2) : nullptr;
    if (!r) {
        Py_XDECREF(a);
        Py_XDECREF(b);
        return nullptr;
    }
    PyTuple_SET_ITEM(r, 0, a);
    PyTuple_SET_ITEM(r, 1, b);
    return r;
}

PyObject *tuple_of(const at::Tensor *ts, int n) {
    PyObject *r = PyTuple_New(n);
    for (int i = 0; r && i < n; ++i) {
        PyObject *o = ts[i].defined() ? wrap(ts[i]) : Py_NewRef(Py_None);
        if (!o) { Py_DECREF(r); return nullptr; }
        PyTuple_SET_ITEM(r, i, o);
    }
    return r;
}

int64_t integer(PyObject *o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PythonError{};
    return v;
}

bool truth(PyObject *o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw PythonError{};
    return v != 0;
}

// ---- operators -----------------------------------------------------------------------------------

// wkv7(initial_state|None, r, w, k, v, a, b, chunk_len, want_state, next_state|None, output|None, workspace|None)
//   -> (output, next_state|None)
PyObject *wkv7(PyObject *const *a) {
    Desc s0(a[0]), six[6];
    for (int i = 0; i < 6; ++i) six[i].set(a[1 + i]);
    const at::Tensor &r = tensor(a[1]);
    const int64_t chunk_len = integer(a[7]);
    const bool has_state = a[0] != Py_None, want_state = has_state && truth(a[8]);
    at::Tensor y_t, s_t;
    if (a[10] == Py_None) y_t = like(r);
    const at::Tensor &y = a[10] == Py_None ? y_t : tensor(a[10]);
    Desc yd(y), sd;
    Workspace ws;
    if (a[11] != Py_None) ws.given(a[11]);
    else if (r.dim() == 4)
        ws.allocate(abi.rwkv7_wkv7_workspace_bytes(r.size(0), r.size(1), r.size(2), r.size(3), six[0].d.dtype), r);
    if (want_state) {
        if (a[9] == Py_None) s_t = like(tensor(a[0]));
        sd.set(a[9] == Py_None ? s_t : tensor(a[9]));
    }
    const rwkv7_stream st = stream_of(r);
    call([&] {
        if (!has_state)
            return abi.rwkv7_fused_wkv7_pretrain(six[0].p, six[1].p, six[2].p, six[3].p, six[4].p, six[5].p, chunk_len,
                                                 yd.p, ws.ptr, ws.bytes, st);
        if (!want_state)
            return abi.rwkv7_fused_wkv7_statetune(s0.p, six[0].p, six[1].p, six[2].p, six[3].p, six[4].p, six[5].p,
                                                  chunk_len, yd.p, ws.ptr, ws.bytes, st);
        return abi.rwkv7_fused_wkv7_statepass(s0.p, six[0].p, six[1].p, six[2].p, six[3].p, six[4].p, six[5].p,
                                              chunk_len, yd.p, sd.p, ws.ptr, ws.bytes, st);
    });
    return pair(given_or_wrapped(a[10], y_t), want_state ? given_or_wrapped(a[9], s_t) : Py_NewRef(Py_None));
}

// wkv7_noalloc(initial_state, r, w, k, v, a, b, chunk_len, output, next_state)
PyObject *wkv7_noalloc(PyObject *const *a) {
    Desc s0(a[0]), six[6];
    for (int i = 0; i < 6; ++i) six[i].set(a[1 + i]);
    const int64_t chunk_len = integer(a[7]);
    Desc yd(a[8]), sd(a[9]);
    const rwkv7_stream st = stream_of(tensor(a[1]));
    call([&] {
        return abi.rwkv7_fused_wkv7_statepass_noalloc(s0.p, six[0].p, six[1].p, six[2].p, six[3].p, six[4].p, six[5].p,
                                                      chunk_len, yd.p, sd.p, st);
    });
    return Py_NewRef(Py_None);
}

// wkv7_saved(initial_state|None, r, w, k, v, a, b, chunk_len, want_state)
//   -> (output, next_state|None, snapshots, state_replacement)
PyObject *wkv7_saved(PyObject *const *a) {
    Desc s0(a[0]), six[6];
    for (int i = 0; i < 6; ++i) six[i].set(a[1 + i]);
    const at::Tensor &r = tensor(a[1]);
    if (r.dim() != 4) raise(PyExc_ValueError, "not enough values to unpack (expected 4)");
    const int64_t B = r.size(0), T = r.size(1), H = r.size(2), N = r.size(3), chunk_len = integer(a[7]);
    if (chunk_len == 0) raise(PyExc_ZeroDivisionError, "integer division or modulo by zero");
    at::Tensor out[4] = {like(r), {}, empty({B, H, T / chunk_len, N, N}, at::kFloat, r), like(r)};
    if (truth(a[8])) out[1] = empty({B, H, N, N}, at::kFloat, r);
    Desc yd(out[0]), sd, snap(out[2]), sa(out[3]);
    if (out[1].defined()) sd.set(out[1]);
    Workspace ws;
    ws.allocate(abi.rwkv7_wkv7_workspace_bytes(B, T, H, N, six[0].d.dtype), r);
    const rwkv7_stream st = stream_of(r);
    call([&] {
        return abi.rwkv7_fused_wkv7_forward_saved(s0.p, six[0].p, six[1].p, six[2].p, six[3].p, six[4].p, six[5].p,
                                                  chunk_len, yd.p, sd.p, snap.p, sa.p, ws.ptr, ws.bytes, st);
    });
    return tuple_of(out, 4);
}

// wkv7_backward(initial_state|None, r, w, k, v, a, b, snapshots, state_replacement, chunk_len, output_grad,
//               next_state_grad|None, want_state_grad, parallel, workspace|None) -> (six gradients, state gradient|None)
PyObject *wkv7_backward(PyObject *const *a) {
    Desc s0(a[0]), six[6], snap(a[7]), sa(a[8]);
    for (int i = 0; i < 6; ++i) six[i].set(a[1 + i]);
    const at::Tensor &r = tensor(a[1]);
    if (r.dim() != 4) raise(PyExc_ValueError, "not enough values to unpack (expected 4)");
    const int64_t B = r.size(0), T = r.size(1), H = r.size(2), N = r.size(3), chunk_len = integer(a[9]);
    const at::Tensor dy_t = tensor(a[10]).contiguous();
    Desc dy(dy_t), ds(a[11]), gd[6], ds0d;
    at::Tensor grads[6], ds0;
    rwkv7_tensor *gp[6];
    for (int i = 0; i < 6; ++i) {
        grads[i] = like(r);
        gd[i].set(grads[i]);
        gp[i] = gd[i].p;
    }
    if (truth(a[12])) {
        ds0 = empty({B, H, N, N}, at::kFloat, r);
        ds0d.set(ds0);
    }
    const rwkv7_stream st = stream_of(r);
    if (truth(a[13]) && r.scalar_type() == at::kBFloat16) {
        Workspace ws;
        if (a[14] != Py_None) ws.given(a[14]);
        else {
            const size_t need = abi.rwkv7_wkv7_backward_workspace_bytes(B, T, H, N);
            ws.allocate(need ? need : 1, r);
        }
        call([&] {
            return abi.rwkv7_fused_wkv7_backward_parallel(s0.p, six[0].p, six[1].p, six[2].p, six[3].p, six[4].p, six[5].p,
                                                          snap.p, sa.p, chunk_len, dy.p, ds.p, gp, ds0d.p, ws.ptr,
                                                          ws.bytes, st);
        });
    } else {
        call([&] {
            return abi.rwkv7_fused_wkv7_backward(s0.p, six[0].p, six[1].p, six[2].p, six[3].p, six[4].p, six[5].p, snap.p,
                                                 sa.p, chunk_len, dy.p, ds.p, gp, ds0d.p, st);
        });
    }
    PyObject *list = PyList_New(6);
    for (int i = 0; list && i < 6; ++i) PyList_SET_ITEM(list, i, wrap(grads[i]));
    return pair(list, ds0.defined() ? wrap(ds0) : Py_NewRef(Py_None));
}

// The node of a training step (see rwkv7_fused_wkv7_training_forward).  In native code because a short step is bound by its host
// path: with the node in Python a step of 1 x 128 tokens x 12 heads took 140 us, now 123 (the engine is most of that).
struct TrainingStep : torch::autograd::Function<TrainingStep> {
    using Tensors = torch::autograd::variable_list;

    static Tensors forward(torch::autograd::AutogradContext *ctx, const at::Tensor &r, const at::Tensor &w, const at::Tensor &k, const at::Tensor &v,
                           const at::Tensor &a, const at::Tensor &b, const std::optional<at::Tensor> &s0, int64_t chunk_len, int64_t keep) {
        const Desc in[6] = {Desc(r), Desc(w), Desc(k), Desc(v), Desc(a), Desc(b)};
        Desc sd0;
        if (s0) sd0.set(*s0);
        Tensors out{like(r), empty({r.size(0), r.size(2), r.size(3), r.size(3)}, at::kFloat, r)};
        const at::Tensor kept = empty({keep}, at::kByte, r);
        Desc yd(out[0]), sd(out[1]);
        const rwkv7_stream st = stream_of(r);
        call([&] {
            return abi.rwkv7_fused_wkv7_training_forward(sd0.p, in[0].p, in[1].p, in[2].p, in[3].p, in[4].p, in[5].p, chunk_len, yd.p, sd.p,
                                                         kept.data_ptr(), (size_t)keep, st);
        });
        // (what the backward pass reads, and only that: the version counters catch a change in place before it)
        ctx->save_for_backward({r, w, k, v, a, b, kept});
        ctx->saved_data["chunk_len"] = chunk_len;
        ctx->saved_data["has_state"] = s0.has_value();
        ctx->set_materialize_grads(false);
        return out;
    }

    // On a thread of the autograd engine, without the interpreter lock.
    static Tensors backward(torch::autograd::AutogradContext *ctx, Tensors grad) {
        const Tensors t = ctx->get_saved_variables();
        const at::Tensor &r = t[0], &kept = t[6];
        const int64_t chunk_len = ctx->saved_data["chunk_len"].toInt();
        const Desc in[6] = {Desc(t[0]), Desc(t[1]), Desc(t[2]), Desc(t[3]), Desc(t[4]), Desc(t[5])};
        const at::Tensor dy_t = grad[0].defined() ? grad[0].contiguous() : at::zeros_like(r), ds_t = grad[1].defined() ? grad[1].contiguous() : grad[1];
        Desc dy(dy_t), ds, gd[6], ds0d;
        if (ds_t.defined()) ds.set(ds_t);
        Tensors out(9);
        rwkv7_tensor *gp[6];
        for (int i = 0; i < 6; ++i) {
            out[i] = like(r);
            gd[i].set(out[i]);
            gp[i] = gd[i].p;
        }
        if (ctx->saved_data["has_state"].toBool()) {
            out[6] = empty({r.size(0), r.size(2), r.size(3), r.size(3)}, at::kFloat, r);
            ds0d.set(out[6]);
        }
        Workspace ws;
        ws.allocate(abi.rwkv7_wkv7_training_workspace_bytes(r.size(0), r.size(1), r.size(2), r.size(3)), r);
        const int status = abi.rwkv7_fused_wkv7_training_backward(in[0].p, in[1].p, in[2].p, in[3].p, in[4].p, in[5].p, chunk_len,
                                                                  kept.data_ptr(), (size_t)kept.numel(), dy.p, ds.p, gp, ds0d.p, ws.ptr,
                                                                  ws.bytes, stream_of(r));
        if (status != 0) {
            const PyGILState_STATE gil = PyGILState_Ensure();
            python_error error;
            try {
                check(status);
            } catch (const PythonError &) {
                error.persist();
            }
            PyGILState_Release(gil);
            throw error;
        }
        return out;
    }
};

// wkv7_training_step(initial_state|None, r, w, k, v, a, b, chunk_len) -> (output, next_state), part of the autograd graph, or
// None for what the training step does not cover
PyObject *wkv7_training_step(PyObject *const *a) {
    const at::Tensor &r = tensor(a[1]);
    for (int i = 2; i < 7; ++i) tensor(a[i]);
    const int64_t chunk_len = integer(a[7]);
    const size_t keep = r.dim() != 4 || !r.is_cuda()
                            ? 0 : abi.rwkv7_wkv7_training_saved_bytes(r.size(0), r.size(1), r.size(2), r.size(3), dtype_code(r.scalar_type()), chunk_len);
    if (keep == 0) return Py_NewRef(Py_None);
    const auto out = TrainingStep::apply(r, tensor(a[2]), tensor(a[3]), tensor(a[4]), tensor(a[5]), tensor(a[6]),
                                         a[0] == Py_None ? std::nullopt : std::make_optional(tensor(a[0])), chunk_len, (int64_t)keep);
    return pair(wrap(out[0]), wrap(out[1]));
}

// mix6(x, six scales) -> six outputs
PyObject *mix6(PyObject *const *a) {
    const at::Tensor &x = tensor(a[0]);
    Desc xd(x), sd[6], od[6];
    at::Tensor out[6];
    outputs_like(out, x, x, x, x, x, x);
    const rwkv7_tensor *sp[6];
    rwkv7_tensor *op[6];
    for (int i = 0; i < 6; ++i) {
        sd[i].set(a[1 + i]);
        sp[i] = sd[i].p;
        od[i].set(out[i]);
        op[i] = od[i].p;
    }
    const rwkv7_stream st = stream_of(x);
    call([&] { return abi.rwkv7_fused_mix6(xd.p, sp, op, st); });
    return tuple_of(out, 6);
}

// mix6_stacked(x, six scales) -> [6, ...]
PyObject *mix6_stacked(PyObject *const *a) {
    const at::Tensor &x = tensor(a[0]);
    Desc xd(x), sd[6];
    const rwkv7_tensor *sp[6];
    for (int i = 0; i < 6; ++i) {
        sd[i].set(a[1 + i]);
        sp[i] = sd[i].p;
    }
    std::vector<int64_t> shape{6};
    for (int64_t n : x.sizes()) shape.push_back(n);
    const at::Tensor out = empty(shape, x.scalar_type(), x);
    Desc od(out);
    const rwkv7_stream st = stream_of(x);
    call([&] { return abi.rwkv7_fused_mix6_stacked(xd.p, sp, od.p, st); });
    return wrap(out);
}

// addcmul(base, diff, scale, inplace) -> output
PyObject *addcmul(PyObject *const *a) {
    const at::Tensor &base = tensor(a[0]);
    const bool inplace = truth(a[3]);
    Desc bd(base), dd(a[1]), sd(a[2]);
    const at::Tensor out = inplace ? base : like(base);
    Desc od(out);
    const rwkv7_stream st = stream_of(base);
    call([&] { return abi.rwkv7_fused_addcmul(bd.p, dd.p, sd.p, od.p, st); });
    return inplace ? Py_NewRef(a[0]) : wrap(out);
}

// addcmul5(base, diff, five scales) -> five outputs
PyObject *addcmul5(PyObject *const *a) {
    const at::Tensor &base = tensor(a[0]);
    Desc bd(base), dd(a[1]), sd[5], od[5];
    at::Tensor out[5];
    outputs_like(out, base, base, base, base, base);
    const rwkv7_tensor *sp[5];
    rwkv7_tensor *op[5];
    for (int i = 0; i < 5; ++i) {
        sd[i].set(a[2 + i]);
        sp[i] = sd[i].p;
        od[i].set(out[i]);
        op[i] = od[i].p;
    }
    const rwkv7_stream st = stream_of(base);
    call([&] { return abi.rwkv7_fused_addcmul5(bd.p, dd.p, sp, op, st); });
    return tuple_of(out, 5);
}

// token_shift_diff(x, state, batch_ids, inplace_state) -> (diff, next state)
PyObject *token_shift_diff(PyObject *const *a) {
    const at::Tensor &x = tensor(a[0]);
    // (Copied first, and the copy updated in place: a state the kernel does not take as it is, such as some columns of a wider
    // table, a broadcast row or rows from an odd offset on, which its copy mends; and nothing to compute, T = 0.)
    const at::Tensor &given = tensor(a[1]);
    const bool keep = !truth(a[3]);
    const bool copied = keep && (x.numel() == 0 || !given.is_contiguous() || (reinterpret_cast<uintptr_t>(given.data_ptr()) & 15u) != 0);
    const at::Tensor state = copied ? given.detach().clone() : given;
    const bool inplace = !keep || copied;
    at::Tensor out[2];   // diff, next state
    out[0] = like(x);
    if (!inplace) out[1] = like(state);   // (its own memory: a server keeps it, and must not keep the step's difference with it)
    Desc xd(x), sd(state), idd(a[2]), dd(out[0]), nd;
    if (!inplace) nd.set(out[1]);
    const rwkv7_stream st = stream_of(x);
    call([&] {
        return inplace ? abi.rwkv7_fused_token_shift_diff(xd.p, sd.p, idd.p, dd.p, st)
                       : abi.rwkv7_fused_token_shift_diff_into(xd.p, sd.p, idd.p, nd.p, dd.p, st);
    });
    return pair(wrap(out[0]), !keep ? Py_NewRef(a[1]) : wrap(copied ? state : out[1]));
}

// weight_prepare(key_precursor, learning_rate_lora, weight_decay_lora, key_removal, key_replacement,
//                value_precursor|None, value_from_first_cell|None, value_residual_lora|None, num_heads)
//   -> (weight_decay, replacement_key, removal_key_normalized, replacement, value|None)
PyObject *weight_prepare(PyObject *const *a) {
    const at::Tensor &key = tensor(a[0]);
    Desc in[8], od[5];
    for (int i = 0; i < 8; ++i) in[i].set(a[i]);
    at::Tensor out[5];
    if (a[5] == Py_None) outputs_like(out, key, key, key, key);   // (no value inputs: no value output)
    else outputs_like(out, key, key, key, key, key);
    for (int i = 0; i < 5; ++i)
        if (out[i].defined()) od[i].set(out[i]);
    const int64_t heads = integer(a[8]);
    const rwkv7_stream st = stream_of(key);
    call([&] {
        return abi.rwkv7_fused_weight_prepare(in[0].p, in[1].p, in[2].p, in[3].p, in[4].p, in[5].p, in[6].p, in[7].p, heads,
                                              od[0].p, od[1].p, od[2].p, od[3].p, od[4].p, st);
    });
    return tuple_of(out, 5);
}

// gated_readout(wkv7_output, receptance, replacement_key, value, gate, gamma, beta, bonus, num_heads, epsilon) -> output
PyObject *gated_readout(PyObject *const *a) {
    const at::Tensor &y = tensor(a[0]);
    Desc in[8];
    for (int i = 0; i < 8; ++i) in[i].set(a[i]);
    const int64_t heads = integer(a[8]);
    const double eps = PyFloat_AsDouble(a[9]);
    if (eps == -1.0 && PyErr_Occurred()) throw PythonError{};
    const at::Tensor out = like(y);
    Desc od(out);
    const rwkv7_stream st = stream_of(y);
    call([&] {
        return abi.rwkv7_fused_gated_readout(in[0].p, in[1].p, in[2].p, in[3].p, in[4].p, in[5].p, in[6].p, in[7].p, eps,
                                             heads, od.p, st);
    });
    return wrap(out);
}

// channel_mixer(x, key_scale, key_weight, value_weight, workspace|None) -> output
PyObject *channel_mixer(PyObject *const *a) {
    const at::Tensor &x = tensor(a[0]), &kw = tensor(a[2]);
    Desc xd(x), sd(a[1]), kd(kw), vd(a[3]);
    const at::Tensor out = like(x);
    Desc od(out);
    Workspace ws;
    if (x.dim() == 3 && kw.dim() == 2) {
        if (a[4] != Py_None) ws.given(a[4]);
        else ws.allocate(abi.rwkv7_channel_mixer_workspace_bytes(x.size(0), x.size(1), x.size(2), kw.size(0)), x);
    }
    const rwkv7_stream st = stream_of(x);
    call([&] { return abi.rwkv7_fused_channel_mixer(xd.p, sd.p, kd.p, vd.p, od.p, ws.ptr, ws.bytes, st); });
    return wrap(out);
}

at::Tensor lm_head_partial_of(const at::Tensor &x, const at::Tensor &w, PyObject *targets, int64_t offset) {
    if (x.dim() < 2 || w.dim() < 1) raise(PyExc_IndexError, "tuple index out of range");
    const at::Tensor partials = empty({x.size(0), 3}, at::kFloat, x);
    Workspace ws;
    const size_t need = abi.rwkv7_lm_head_ce_workspace_bytes(x.size(0), x.size(1), w.size(0));
    ws.allocate(need, x);
    Desc xd(x), wd(w), td(targets), pd(partials);
    const rwkv7_stream st = stream_of(x);
    call([&] { return abi.rwkv7_fused_lm_head_ce_partial(xd.p, wd.p, td.p, offset, pd.p, ws.ptr, ws.bytes, st); });
    return partials;
}

PyObject *lm_head_finalize_of(const at::Tensor &partials_all, PyObject *targets) {
    if (partials_all.dim() < 2) raise(PyExc_IndexError, "tuple index out of range");
    const int64_t R = partials_all.size(1);
    const at::Tensor out[2] = {empty({R}, at::kFloat, partials_all), empty({R}, at::kFloat, partials_all)};
    Desc pd(partials_all), td(targets), ld(out[0]), sd(out[1]);
    const rwkv7_stream st = stream_of(partials_all);
    call([&] { return abi.rwkv7_lm_head_ce_finalize(pd.p, td.p, ld.p, sd.p, st); });
    return tuple_of(out, 2);
}

// lm_head_ce_partial(x, weight_shard, targets, vocab_offset) -> partials
PyObject *lm_head_ce_partial(PyObject *const *a) {
    return wrap(lm_head_partial_of(tensor(a[0]), tensor(a[1]), a[2], integer(a[3])));
}
// lm_head_ce_finalize(partials_all, targets) -> (lse, loss)
PyObject *lm_head_ce_finalize(PyObject *const *a) { return lm_head_finalize_of(tensor(a[0]), a[1]); }
// lm_head_ce(x, weight, targets) -> (lse, loss)
PyObject *lm_head_ce(PyObject *const *a) {
    const at::Tensor p = lm_head_partial_of(tensor(a[0]), tensor(a[1]), a[2], 0);
    return lm_head_finalize_of(p.unsqueeze(0), a[2]);
}

// ---- module ---------------------------------------------------------------------------------------

// Checks the number of arguments and turns what is thrown below into a Python exception.
template <PyObject *(*F)(PyObject *const *), int NARGS>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != NARGS) {
        PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", NARGS, n);
        return nullptr;
    }
    if (g_error == nullptr) {
        PyErr_SetString(PyExc_RuntimeError, "the library has not been opened");
        return nullptr;
    }
    try {
        return F(args);
    } catch (const PythonError &) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// open(path of the shared library, exception class taking (status, message))
PyObject *open_library(PyObject *, PyObject *const *args, Py_ssize_t n) {
    const char *path = n == 2 ? PyUnicode_AsUTF8(args[0]) : nullptr;
    if (path == nullptr) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "open(path, error class)");
        return nullptr;
    }
    void *h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (h == nullptr) return PyErr_Format(PyExc_RuntimeError, "%s: %s", path, dlerror());
    Abi found;
#define RWKV7_RESOLVE(name)                                                              \
    found.name = reinterpret_cast<decltype(found.name)>(dlsym(h, #name));                \
    if (found.name == nullptr) return PyErr_Format(PyExc_RuntimeError, "%s lacks %s", path, #name);
    RWKV7_BOUND(RWKV7_RESOLVE)
#undef RWKV7_RESOLVE
    abi = found;
    Py_XSETREF(g_error, Py_NewRef(args[1]));
    Py_RETURN_NONE;
}

#define RWKV7_METHOD(name, nargs) \
    {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name, nargs>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"open", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&open_library)), METH_FASTCALL, nullptr},
    RWKV7_METHOD(wkv7, 12), RWKV7_METHOD(wkv7_noalloc, 10), RWKV7_METHOD(wkv7_saved, 9), RWKV7_METHOD(wkv7_backward, 15), RWKV7_METHOD(wkv7_training_step, 8),
    RWKV7_METHOD(mix6, 7), RWKV7_METHOD(mix6_stacked, 7), RWKV7_METHOD(addcmul, 4), RWKV7_METHOD(addcmul5, 7),
    RWKV7_METHOD(token_shift_diff, 4), RWKV7_METHOD(weight_prepare, 9), RWKV7_METHOD(gated_readout, 10),
    RWKV7_METHOD(channel_mixer, 5), RWKV7_METHOD(lm_head_ce_partial, 4), RWKV7_METHOD(lm_head_ce_finalize, 2),
    RWKV7_METHOD(lm_head_ce, 3),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "rwkv7_b200_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_rwkv7_b200_torch(void) { return PyModule_Create(&module); }
