// Native host path of the operator set: one call from Python validates the tensors, allocates the
// outputs, launches through the C ABI of librgd_b200.so and records the autograd node; the backward
// runs inside the autograd engine without entering Python.
//
// What bounds the small operators is this code, not their kernels (a forward + backward of a
// [4, 256, 1024] fp32 RMSNorm is 13 us of GPU time): with the marshalling in Python (ctypes, a Python
// autograd.Function, launch keys built from Python tuples) such a call took 126 us, a forward alone 15 us.
//
// Every entry returns None for arguments it does not cover: anything that is wrong (the Python path then
// raises the right exception), tensor subclasses, forward-mode tangents, views whose channel stride is not 1, empty tensors,
// caches that are not a _LaunchCache, a bias that wants a gradient; and for every call while something watches
// the operations (torch.jit.trace, dispatch modes, functorch transforms).  The Python path in functional.py
// handles those, so conditions here only have to be sufficient.
//
// Under compiled autograd a node is traced instead of run: its saved tensors are then stand-ins without
// storage, and it calls the registered operator of its backward (rgd_triton_b200/library.py) on them.
//
// The C ABI is bound at run time through the handle of the library that _lib.py has loaded, so this
// module has no link-time dependency on it and the two can never be different copies.
#include <Python.h>

#include <dlfcn.h>
#include <math.h>

#include <array>
#include <atomic>
#include <memory>
#include <mutex>
#include <vector>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>

#include "../../../include/rgd_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using torch::dynamo::autograd::CompiledNodeArgs;
using torch::dynamo::autograd::SwapSavedVariables;

// ------------------------------------------------------------------ C ABI, bound once
struct Api {
#define RGD_FN(name) decltype(&rgd_##name) name = nullptr;
#define RGD_FUNCTIONS(X)                                                                                              \
    X(device_supported) X(status_string) X(cache_create) X(cache_destroy) X(l2norm_fwd) X(l2norm_bwd) X(rmsnorm_fwd)   \
    X(rmsnorm_bwd) X(rmsnorm_bwd_workspace_bytes) X(headln_fwd) X(headln_bwd) X(rope) X(lnrope_fwd) X(lnrope_bwd)      \
    X(attn_lse_rows) X(attn_fwd) X(attn_bwd) X(attn_bwd_workspace_bytes) X(attn_bwd_single_pass_workspace_bytes)
    RGD_FUNCTIONS(RGD_FN)
#undef RGD_FN
};
Api api;
std::atomic<bool> single_pass{true};        // how the attention backward forms dQ (functional.set_attention_backward)

// Thrown by a forward whose arguments the library refuses: the call is handed back to Python, which
// raises what the entry point documents.
struct Refused {};

void launched(int code, const char *what, bool forward) {
    if (code == 0) return;
    if (forward) throw Refused{};
    TORCH_CHECK(false, what, ": ", api.status_string(code), " (status ", code, ")");
}

bool device_ok(int index) {
    static std::array<std::atomic<signed char>, 64> known{};
    if (index < 0 || index >= 64) return false;
    signed char v = known[index].load(std::memory_order_relaxed);
    if (v == 0) {
        v = api.device_supported(index) == 1 ? 1 : -1;
        known[index].store(v, std::memory_order_relaxed);
    }
    return v == 1;
}

int code_of(const Tensor &t) {
    switch (t.scalar_type()) {
        case at::kFloat: return RGD_F32;
        case at::kHalf: return RGD_F16;
        case at::kBFloat16: return RGD_BF16;
        default: return -1;
    }
}

// A tensor that only Python knows how to handle, or that carries a forward-mode tangent (the autograd
// functions have no jvp: the Python path refuses it).
bool special(const Tensor &t) { return t.unsafeGetTensorImpl()->is_python_dispatch() || t._fw_grad(0).defined(); }

// A plain CUDA tensor of a supported type with unit channel stride and at least one element.
bool plain(const Tensor &t, int64_t ndim) {
    return t.defined() && t.is_cuda() && t.dim() == ndim && t.numel() > 0 && t.stride(-1) == 1 && code_of(t) >= 0 && !special(t);
}

bool like(const Tensor &t, const Tensor &first) {
    return t.scalar_type() == first.scalar_type() && t.device() == first.device();
}

// empty_like: dense tensors keep their strides, as torch.empty_like's preserve_format does.
Tensor new_like(const Tensor &t) {
    if (t.is_non_overlapping_and_dense())
        return at::detail::empty_strided_cuda(t.sizes(), t.strides(), t.scalar_type(), t.device());
    at::AutoDispatchBelowADInplaceOrView guard;
    return at::empty_like(t);
}

Tensor new_buffer(at::IntArrayRef sizes, at::ScalarType type, c10::Device device) {
    return at::detail::empty_cuda(sizes, type, device, std::nullopt);
}

void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// ------------------------------------------------------------------ launch state behind a module's cache
// What a module's cache slots report (the shapes, strides and types last launched per kernel) and the
// library's tensor-map cache.  Shared by the module and the autograd nodes of its calls, so a backward
// after the module is gone still has it.
struct LaunchState {
    std::mutex mu;
    rgd_cache *cache = nullptr;
    std::vector<int64_t> seen[2];       // forward, backward
    ~LaunchState() {
        if (cache) api.cache_destroy(cache);
    }
    rgd_cache *native() {
        std::lock_guard<std::mutex> lock(mu);
        if (!cache) cache = api.cache_create();
        return cache;
    }
};
using State = std::shared_ptr<LaunchState>;

struct PyLaunchState {
    PyObject_HEAD
    State *state;
};
PyTypeObject *launch_state_type = nullptr;

struct Key {
    int64_t v[64];
    int n = 0;
    void add(int64_t x) { if (n < 64) v[n++] = x; }
    void add(const Tensor &t) {
        for (int64_t s : t.sizes()) add(s);
        for (int64_t s : t.strides()) add(s);
        add((int64_t)t.scalar_type());
    }
};

template <typename... Ts>
void note(const State &st, int slot, const Ts &...ts) {
    if (!st) return;
    Key k;
    (k.add(ts), ...);
    std::lock_guard<std::mutex> lock(st->mu);
    std::vector<int64_t> &s = st->seen[slot];
    if ((int)s.size() != k.n || !std::equal(s.begin(), s.end(), k.v)) s.assign(k.v, k.v + k.n);
}

PyObject *str_state = nullptr;

// The launch state of a Python cache object.  None: no state, fine.  Anything else without one: decline.
bool state_of(PyObject *cache, State &out) {
    if (cache == Py_None) return true;
    PyObject *s = PyObject_GetAttr(cache, str_state);
    if (!s) {
        PyErr_Clear();
        return false;
    }
    const bool ok = Py_TYPE(s) == launch_state_type;
    if (ok) out = *reinterpret_cast<PyLaunchState *>(s)->state;
    Py_DECREF(s);
    return ok;
}

// bool(o); what its __bool__ raises goes to the caller.
bool truth(PyObject *o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw python_error();
    return v == 1;
}

bool tensor_arg(PyObject *o, Tensor &out) {
    if (!THPVariable_CheckExact(o)) return false;
    out = THPVariable_Unpack(o);
    return true;
}

bool wants_grad(std::initializer_list<const Tensor *> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor *t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

// The kernels need a unit channel stride.
Tensor unit(const Tensor &g) {
    if (!g.defined() || g.stride(-1) == 1) return g;
    Tensor c = g.contiguous();
    return c.stride(-1) == 1 ? c : at::empty(g.sizes(), g.options()).copy_(g);
}

// The gradient the engine hands over: undefined means zero.
Tensor upstream(const Tensor &g, const Tensor &ref) {
    return g.defined() ? unit(g) : at::zeros(ref.sizes(), ref.options());
}

// What a backward unpacks may lie differently from what the forward saved: saved-tensor hooks move and copy
// (torch.autograd.graph.save_on_cpu gives back a dense copy of a slice).  Strides are therefore taken from
// the unpacked tensors, never kept from the forward; sizes and types have to be the same.
void restored(bool ok, const char *what) {
    TORCH_CHECK(ok, what, " backward: a saved tensor came back from its hooks with another shape, type or device");
}

// Something on this thread sees every operation (a tracer, a dispatch mode, a functorch transform) and would miss
// this call: the Python functions take it.
bool watched() {
    return at::tracer::impl::is_dispatch_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

// ------------------------------------------------------------------ compiled autograd
bool stand_in(const Tensor &t) { return t.defined() && t.unsafeGetTensorImpl()->is_python_dispatch(); }

// The operators are registered when their module is imported.
void register_operators() {
    PyGILState_STATE gil = PyGILState_Ensure();
    PyObject *m = PyImport_ImportModule("rgd_triton_b200.library");
    if (!m) PyErr_Clear();      // the lookup below then says what is missing
    Py_XDECREF(m);
    PyGILState_Release(gil);
}

template <typename... A>
std::vector<c10::IValue> call_operator(const char *name, A &&...args) {
    auto op = c10::Dispatcher::singleton().findSchemaOrThrow(name, "");
    torch::jit::Stack stack{c10::IValue(std::forward<A>(args))...};
    op.callBoxed(stack);
    return stack;
}

// What compiled autograd asks of a node, given its attributes in a fixed order: SAVED lists the saved variables,
// CONSTANTS what a traced backward is specialised on.
#define RGD_COMPILED(SAVED, CONSTANTS)                                                                                \
    void compiled_args(CompiledNodeArgs &args) const override {                                                       \
        register_operators();                                                                                         \
        auto collect = [&](const SavedVariable &v, bool is_output) { args.collect(v, is_output); };                  \
        auto constant = [&](auto... v) { (args.collect(v), ...); };                                                  \
        SAVED(collect)                                                                                                \
        CONSTANTS(constant)                                                                                           \
    }                                                                                                                 \
    variable_list apply_with_saved(const variable_list &grads, SwapSavedVariables &saved) override {                 \
        auto before = [&](SavedVariable &v, bool) { saved.before(v); };                                              \
        auto after = [&](SavedVariable &v, bool) { saved.after(v); };                                                \
        SAVED(before)                                                                                                 \
        variable_list out = apply(variable_list(grads));                                                              \
        SAVED(after)                                                                                                  \
        return out;                                                                                                   \
    }

template <typename N>
std::shared_ptr<N> new_node(torch::autograd::edge_list edges) {
    std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
    n->set_next_edges(std::move(edges));
    return n;
}

PyObject *wrap2(Tensor a, Tensor b) {
    PyObject *t = PyTuple_New(2);
    if (!t) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(a)));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(b)));
    return t;
}

// Allocation and launches run without the GIL, as they do through ctypes: a full launch queue or a
// first allocation then stops no other Python thread.
struct NoGil {
    PyThreadState *saved = PyEval_SaveThread();
    NoGil() = default;
    NoGil(const NoGil &) = delete;
    ~NoGil() { PyEval_RestoreThread(saved); }
};

// ------------------------------------------------------------------ row norms
rgd_rows rows(const Tensor &t) { return {t.data_ptr(), t.stride(0), t.stride(1)}; }

struct Rows {
    int n = 0;
    Tensor x[2], w[2];          // w undefined for L2
    int64_t N[2] = {0, 0}, C[2] = {0, 0}, B = 0;
    int64_t w_stride[2] = {0, 0};
    int per_batch[2] = {0, 0};
    int dtype = 0, w_dtype = 0;
    double eps = 0;
    State state;
};

// Sizes and weight forms ([C], [1,1,C] shared; [B,1,C] per batch); false: not covered here.
bool rows_ok(Rows &r) {
    const Tensor &a = r.x[0];
    if (!plain(a, 3) || !device_ok(a.get_device())) return false;
    r.B = a.size(0);
    r.dtype = code_of(a);
    for (int i = 0; i < r.n; ++i) {
        const Tensor &x = r.x[i];
        if (i > 0 && (!plain(x, 3) || !like(x, a) || x.size(0) != r.B)) return false;
        r.N[i] = x.size(1);
        r.C[i] = x.size(2);
        r.w_stride[i] = r.per_batch[i] = 0;
        const Tensor &w = r.w[i];
        if (!w.defined()) continue;
        if (!w.is_cuda() || w.device() != a.device() || code_of(w) < 0 || w.scalar_type() != r.w[0].scalar_type() ||
            special(w) || (w.dim() != 1 && w.dim() != 3) || w.stride(-1) != 1 ||
            w.size(-1) != r.C[i])
            return false;
        if (w.dim() == 3) {
            if (w.size(1) != 1 || (w.size(0) != 1 && w.size(0) != r.B)) return false;
            if (w.size(0) != 1) {
                r.w_stride[i] = w.stride(0);
                r.per_batch[i] = 1;
            }
        }
        r.w_dtype = code_of(w);
    }
    return true;
}

void rows_forward(Rows &r, Tensor (&y)[2]) {
    NoGil nogil;
    c10::cuda::OptionalCUDAGuard guard(r.x[0].device());
    rgd_rows xs[2], ys[2];
    const void *ws[2] = {nullptr, nullptr};
    for (int i = 0; i < r.n; ++i) {
        y[i] = new_like(r.x[i]);
        xs[i] = rows(r.x[i]);
        ys[i] = rows(y[i]);
        if (r.w[i].defined()) ws[i] = r.w[i].data_ptr();
    }
    void *st = stream_of(r.x[0]);
    if (r.w[0].defined())
        launched(api.rmsnorm_fwd(r.n, xs, ws, r.w_stride, ys, r.N, r.C, r.B, (float)r.eps, r.dtype, r.w_dtype, st), "rmsnorm_fwd", true);
    else
        launched(api.l2norm_fwd(r.n, xs, ys, r.N, r.C, r.B, (float)r.eps, r.dtype, st), "l2norm_fwd", true);
    if (r.n == 1) note(r.state, 0, r.x[0]);
    else note(r.state, 0, r.x[0], r.x[1]);
}

// Saves the inputs only: the row statistics are recomputed from x, which the backward reads anyway.
struct RowsBackward : public Node {
    Rows r;                     // its tensors are cleared, the saved variables stand for them
    SavedVariable x[2], w[2];
    bool affine = false;

    std::string name() const override { return affine ? "FusedRMSNormBackward" : "L2NormalizeBackward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (int i = 0; i < 2; ++i) {
            x[i].reset_data();
            w[i].reset_data();
        }
    }
#define RGD_SAVED(f)                      \
    for (int i = 0; i < r.n; ++i) {       \
        f(x[i], false);                   \
        if (affine) f(w[i], false);       \
    }
#define RGD_CONSTANTS(f) f(r.n, affine, r.eps);
    RGD_COMPILED(RGD_SAVED, RGD_CONSTANTS)
#undef RGD_SAVED
#undef RGD_CONSTANTS
    variable_list traced(const variable_list &grads, const Tensor (&xt)[2], const Tensor (&wt)[2]) const {
        c10::List<Tensor> xs, ws, dys;
        for (int i = 0; i < r.n; ++i) {
            xs.push_back(xt[i]);
            if (affine) ws.push_back(wt[i]);
            dys.push_back(grads[i].defined() ? grads[i].contiguous() : at::zeros_like(xt[i]));
        }
        const auto out = affine ? call_operator("rgd_b200::rmsnorm_bwd", xs, ws, dys, r.eps)
                                : call_operator("rgd_b200::l2norm_bwd", xs, dys, r.eps);
        return out.at(0).toTensorVector();
    }
    variable_list apply(variable_list &&grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        Tensor dy[2], dx[2], dw[2];
        rgd_rows xs[2], dys[2], dxs[2];
        const void *ws[2] = {nullptr, nullptr};
        void *dws[2] = {nullptr, nullptr};
        Rows r = this->r;       // with the unpacked tensors, and the weights' strides from them
        Tensor(&xt)[2] = r.x, (&wt)[2] = r.w;
        for (int i = 0; i < r.n; ++i) {
            xt[i] = x[i].unpack();
            if (affine) wt[i] = w[i].unpack();
        }
        if (stand_in(xt[0])) return traced(grads, xt, wt);
        c10::cuda::OptionalCUDAGuard guard(xt[0].device());
        at::AutoDispatchBelowADInplaceOrView below;
        for (int i = 0; i < r.n; ++i) {
            xt[i] = unit(xt[i]);
            wt[i] = unit(wt[i]);
        }
        restored(rows_ok(r) && r.dtype == this->r.dtype && std::equal(r.N, r.N + r.n, this->r.N) &&
                     std::equal(r.C, r.C + r.n, this->r.C) && r.B == this->r.B && (!affine || r.w_dtype == this->r.w_dtype),
                 affine ? "FusedRMSNorm" : "L2Normalize");
        for (int i = 0; i < r.n; ++i) {
            dy[i] = upstream(grads[i], xt[i]);
            dx[i] = new_like(xt[i]);
            xs[i] = rows(xt[i]);
            dys[i] = rows(dy[i]);
            dxs[i] = rows(dx[i]);
            if (affine) {       // fp32 sums over the batch (or per batch), rounded once into w's own shape
                dw[i] = new_buffer(wt[i].sizes(), wt[i].scalar_type(), wt[i].device());
                ws[i] = wt[i].data_ptr();
                dws[i] = dw[i].data_ptr();
            }
        }
        void *st = stream_of(xt[0]);
        variable_list out;
        out.reserve(4);
        for (int i = 0; i < r.n; ++i) out.push_back(dx[i]);
        if (affine) {
            const int64_t bytes = std::max<int64_t>(api.rmsnorm_bwd_workspace_bytes(r.n, r.N, r.C, r.B), 16);
            Tensor work = new_buffer({bytes}, at::kByte, xt[0].device());
            launched(api.rmsnorm_bwd(r.n, xs, ws, r.w_stride, dys, dxs, dws, r.per_batch, r.N, r.C, r.B, (float)r.eps, r.dtype,
                                     r.w_dtype, work.data_ptr(), bytes, st), "rmsnorm_bwd", false);
            for (int i = 0; i < r.n; ++i) out.push_back(dw[i]);
        } else {
            launched(api.l2norm_bwd(r.n, xs, dys, dxs, r.N, r.C, r.B, (float)r.eps, r.dtype, st), "l2norm_bwd", false);
        }
        if (r.n == 1) note(r.state, 1, xt[0], dy[0]);
        else note(r.state, 1, xt[0], xt[1], dy[0], dy[1]);
        return out;
    }
};

PyObject *rows_call(Rows &r) {
    if (!rows_ok(r)) Py_RETURN_NONE;
    Tensor y[2];
    rows_forward(r, y);
    if (wants_grad({&r.x[0], &r.x[1], &r.w[0], &r.w[1]})) {
        const bool affine = r.w[0].defined();
        auto node = new_node<RowsBackward>(
            affine ? (r.n == 1 ? torch::autograd::collect_next_edges(r.x[0], r.w[0])
                               : torch::autograd::collect_next_edges(r.x[0], r.x[1], r.w[0], r.w[1]))
                   : (r.n == 1 ? torch::autograd::collect_next_edges(r.x[0]) : torch::autograd::collect_next_edges(r.x[0], r.x[1])));
        node->affine = affine;
        for (int i = 0; i < r.n; ++i) {
            node->x[i] = SavedVariable(r.x[i], false);
            if (affine) node->w[i] = SavedVariable(r.w[i], false);
            r.x[i].reset();
            r.w[i].reset();
        }
        node->r = r;
        for (int i = 0; i < r.n; ++i) torch::autograd::set_history(y[i], node);
    }
    return r.n == 1 ? THPVariable_Wrap(std::move(y[0])) : wrap2(std::move(y[0]), std::move(y[1]));
}

// ------------------------------------------------------------------ head operators
enum HeadOp { HEAD_LN, HEAD_ROPE, HEAD_LNROPE };

struct Heads {
    HeadOp op = HEAD_LN;
    bool heads_second = true;
    int64_t B = 0, H = 0, nq = 0, nk = 0, d = 0, P = 0, R = 0, cut_q = 0, cut_k = 0, pos_s = 0, pos_n = 0;
    int dtype = 0, pos_dtype = 0;
    double eps = 0;
    State state;

    rgd_heads view(const Tensor &t) const {
        return heads_second ? rgd_heads{t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)}
                            : rgd_heads{t.data_ptr(), t.stride(0), t.stride(2), t.stride(1)};
    }
};

bool heads_ok(Heads &h, const Tensor &q, const Tensor &k) {
    if (!plain(q, 4) || !plain(k, 4) || !like(k, q) || !device_ok(q.get_device())) return false;
    const int tok = h.heads_second ? 2 : 1, head = h.heads_second ? 1 : 2;
    h.B = q.size(0); h.H = q.size(head); h.nq = q.size(tok); h.nk = k.size(tok); h.d = q.size(3);
    h.dtype = code_of(q);
    return k.size(0) == h.B && k.size(head) == h.H && k.size(3) == h.d && h.d <= (h.op == HEAD_LN ? 256 : 128);
}

bool table_ok(Heads &h, const Tensor &pos, c10::Device device) {
    if (!plain(pos, 3) || pos.device() != device || pos.size(0) != 2 || h.nq >= pos.size(1) || h.nk >= pos.size(1) ||
        (code_of(pos) != h.dtype && pos.scalar_type() != at::kFloat))
        return false;
    h.P = pos.size(1); h.R = pos.size(2); h.pos_s = pos.stride(0); h.pos_n = pos.stride(1);
    h.pos_dtype = code_of(pos);
    return true;
}

// seq_cutoff: None, an int, or a (q, k) pair.
bool cutoffs(Heads &h, PyObject *o) {
    h.cut_q = h.nq;
    h.cut_k = h.nk;
    if (o == Py_None) return true;
    if (PyLong_Check(o)) {
        h.cut_q = h.cut_k = PyLong_AsLongLong(o);
    } else if ((PyTuple_Check(o) || PyList_Check(o)) && PySequence_Fast_GET_SIZE(o) == 2) {
        PyObject *a = PySequence_Fast_GET_ITEM(o, 0), *b = PySequence_Fast_GET_ITEM(o, 1);
        if (!PyLong_Check(a) || !PyLong_Check(b)) return false;
        h.cut_q = PyLong_AsLongLong(a);
        h.cut_k = PyLong_AsLongLong(b);
    } else {
        return false;
    }
    if (PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

// dq / dk: the upstream gradients (backward; a rotation needs no q, k then)
void heads_launch(const Heads &h, bool backward, const Tensor &q, const Tensor &k, const Tensor &dqi, const Tensor &dki,
                  const Tensor &pos, const Tensor &qo, const Tensor &ko) {
    void *st = stream_of(qo);
    const rgd_heads qov = h.view(qo), kov = h.view(ko);
    if (h.op == HEAD_ROPE) {
        const rgd_heads a = h.view(backward ? dqi : q), b = h.view(backward ? dki : k);
        launched(api.rope(&a, &b, pos.data_ptr(), h.pos_s, h.pos_n, &qov, &kov, h.B, h.H, h.nq, h.nk, h.d, h.P, h.R, h.cut_q,
                          h.cut_k, backward ? 1 : 0, h.dtype, h.pos_dtype, st), "rope", !backward);
        return;
    }
    const rgd_heads qv = h.view(q), kv = h.view(k);
    rgd_heads dqv{}, dkv{};
    if (backward) {
        dqv = h.view(dqi);
        dkv = h.view(dki);
    }
    if (h.op == HEAD_LN) {
        launched(backward ? api.headln_bwd(&qv, &kv, &dqv, &dkv, &qov, &kov, h.B, h.H, h.nq, h.nk, h.d, (float)h.eps, h.dtype, st)
                          : api.headln_fwd(&qv, &kv, &qov, &kov, h.B, h.H, h.nq, h.nk, h.d, (float)h.eps, h.dtype, st),
                 backward ? "headln_bwd" : "headln_fwd", !backward);
        return;
    }
    launched(backward ? api.lnrope_bwd(&qv, &kv, &dqv, &dkv, pos.data_ptr(), h.pos_s, h.pos_n, &qov, &kov, h.B, h.H, h.nq, h.nk,
                                       h.d, h.P, h.R, h.cut_q, h.cut_k, (float)h.eps, h.dtype, h.pos_dtype, st)
                      : api.lnrope_fwd(&qv, &kv, pos.data_ptr(), h.pos_s, h.pos_n, &qov, &kov, h.B, h.H, h.nq, h.nk, h.d, h.P,
                                       h.R, h.cut_q, h.cut_k, (float)h.eps, h.dtype, h.pos_dtype, st),
             backward ? "lnrope_bwd" : "lnrope_fwd", !backward);
}

struct HeadsBackward : public Node {
    Heads h;
    SavedVariable q, k, pos;
    std::vector<int64_t> q_sizes, k_sizes;      // for upstream gradients that are undefined (zero)
    at::TensorOptions options;

    const char *operator_name() const { return h.op == HEAD_LN ? "FusedHeadLayerNorm" : h.op == HEAD_ROPE ? "RoPE" : "FusedLNRoPE"; }
    std::string name() const override { return std::string(operator_name()) + "Backward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        q.reset_data();
        k.reset_data();
        pos.reset_data();
    }
#define RGD_SAVED(f)             \
    if (h.op != HEAD_ROPE) {     \
        f(q, false);             \
        f(k, false);             \
    }                            \
    if (h.op != HEAD_LN) f(pos, false);
#define RGD_CONSTANTS(f) f((int64_t)h.op, h.heads_second, h.cut_q, h.cut_k, h.eps, options, q_sizes, k_sizes);
    RGD_COMPILED(RGD_SAVED, RGD_CONSTANTS)
#undef RGD_SAVED
#undef RGD_CONSTANTS
    variable_list traced(const variable_list &grads, const Tensor &qt, const Tensor &kt, const Tensor &pt) const {
        const Tensor dq = grads[0].defined() ? grads[0].contiguous() : at::zeros(q_sizes, options);
        const Tensor dk = grads[1].defined() ? grads[1].contiguous() : at::zeros(k_sizes, options);
        const auto out = h.op == HEAD_LN     ? call_operator("rgd_b200::headln_bwd", qt, kt, dq, dk, h.heads_second, h.eps)
                         : h.op == HEAD_ROPE ? call_operator("rgd_b200::rope", dq, dk, pt, h.cut_q, h.cut_k, h.heads_second, true)
                                             : call_operator("rgd_b200::lnrope_bwd", qt, kt, dq, dk, pt, h.cut_q, h.cut_k,
                                                             h.heads_second, h.eps);
        return {out.at(0).toTensor(), out.at(1).toTensor()};
    }
    variable_list apply(variable_list &&grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        Tensor qt, kt, pt;
        Heads h = this->h;      // with the strides of the unpacked rotary table
        if (h.op != HEAD_ROPE) {
            qt = q.unpack();
            kt = k.unpack();
        }
        if (h.op != HEAD_LN) pt = pos.unpack();
        if (stand_in(h.op == HEAD_LN ? qt : pt)) return traced(grads, qt, kt, pt);
        c10::cuda::OptionalCUDAGuard guard(options.device());
        at::AutoDispatchBelowADInplaceOrView below;
        qt = unit(qt);
        kt = unit(kt);
        pt = unit(pt);
        auto as_saved = [&](const Tensor &t, const std::vector<int64_t> &sizes) {
            return plain(t, 4) && t.sizes() == at::IntArrayRef(sizes) && t.scalar_type() == options.dtype() && t.device() == options.device();
        };
        restored((h.op == HEAD_ROPE || (as_saved(qt, q_sizes) && as_saved(kt, k_sizes))) &&
                     (h.op == HEAD_LN || (table_ok(h, pt, options.device()) && h.P == this->h.P && h.R == this->h.R &&
                                          h.pos_dtype == this->h.pos_dtype)), operator_name());
        Tensor g[2];
        for (int i = 0; i < 2; ++i) {
            if (!grads[i].defined()) g[i] = at::zeros(i ? k_sizes : q_sizes, options);
            else g[i] = upstream(grads[i], grads[i]);
        }
        Tensor dq = new_like(g[0]), dk = new_like(g[1]);
        heads_launch(h, true, qt, kt, g[0], g[1], pt, dq, dk);
        note(h.state, 1, g[0], g[1]);
        return {dq, dk};
    }
};

PyObject *heads_call(Heads &h, const Tensor &q, const Tensor &k, const Tensor &pos) {
    Tensor qo, ko;
    {
        NoGil nogil;
        c10::cuda::OptionalCUDAGuard guard(q.device());
        qo = new_like(q);
        ko = new_like(k);
        heads_launch(h, false, q, k, Tensor(), Tensor(), pos, qo, ko);
        note(h.state, 0, q, k);
    }
    if (wants_grad({&q, &k})) {
        auto node = new_node<HeadsBackward>(torch::autograd::collect_next_edges(q, k));
        node->h = h;
        if (h.op != HEAD_ROPE) {
            node->q = SavedVariable(q, false);
            node->k = SavedVariable(k, false);
        }
        if (h.op != HEAD_LN) node->pos = SavedVariable(pos, false);
        node->q_sizes = q.sizes().vec();
        node->k_sizes = k.sizes().vec();
        node->options = q.options();
        torch::autograd::set_history(qo, node);
        torch::autograd::set_history(ko, node);
    }
    return wrap2(std::move(qo), std::move(ko));
}

// ------------------------------------------------------------------ attention
struct Attn {
    int64_t B = 0, H = 0, tq = 0, tk = 0, d = 0;
    double scale = 0;
    bool causal = false;
    int dtype = 0;
    int bias_kind = RGD_BIAS_NONE, bias_dtype = RGD_F32;
    int64_t bias_sb = 0, bias_sh = 0, bias_sq = 0;
    State state;

    static rgd_heads view(const Tensor &t) { return {t.data_ptr(), t.stride(0), t.stride(2), t.stride(1)}; }
    rgd_bias bias(const Tensor &t, const Tensor &tiles) const {
        return {t.defined() ? t.data_ptr() : nullptr, bias_sb, bias_sh, bias_sq, bias_kind, bias_dtype,
                tiles.defined() ? tiles.data_ptr() : nullptr};
    }
};

bool attn_ok(Attn &a, const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &bias) {
    if (!plain(q, 4) || !plain(k, 4) || !plain(v, 4) || !like(k, q) || !like(v, q) || q.scalar_type() == at::kFloat ||
        !device_ok(q.get_device()))
        return false;
    a.B = q.size(0); a.tq = q.size(1); a.H = q.size(2); a.d = q.size(3); a.tk = k.size(1);
    a.dtype = code_of(q);
    for (const Tensor *t : {&k, &v})
        if (t->size(0) != a.B || t->size(1) != a.tk || t->size(2) != a.H || t->size(3) != a.d) return false;
    if (a.d > 128) return false;
    if (!bias.defined()) return true;
    if (!plain(bias, 4) || bias.device() != q.device() || (code_of(bias) != a.dtype && bias.scalar_type() != at::kFloat) ||
        bias.size(3) != a.tk || (bias.size(0) != 1 && bias.size(0) != a.B) || (bias.size(1) != 1 && bias.size(1) != a.H))
        return false;
    if (bias.size(2) == 1) a.bias_kind = RGD_BIAS_VECTOR;
    else if (bias.size(2) == a.tq) a.bias_kind = RGD_BIAS_MATRIX;
    else return false;
    a.bias_dtype = code_of(bias);
    a.bias_sb = bias.size(0) == a.B ? bias.stride(0) : 0;       // broadcast dimensions advance by 0
    a.bias_sh = bias.size(1) == a.H ? bias.stride(1) : 0;
    a.bias_sq = a.bias_kind == RGD_BIAS_MATRIX ? bias.stride(2) : 0;
    return true;
}

// Views that the aligned kernels take as they are, and the problems for which others are worth a dense copy
// (functional.py, _addressable and flash_attn_func, which makes those of the inputs).
bool addressable(const Tensor &t, bool zero_strides = false) {
    bool ok = t.stride(-1) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
    for (int i = 0; i < 3; ++i) ok = ok && t.stride(i) % 8 == 0 && (t.stride(i) > 0 || t.size(i) == 1 || zero_strides);
    return ok;
}
bool copies_pay(const Attn &a) {
    return a.d % 8 == 0 && a.d != 64 && a.d != 128 && a.B * a.H * a.tq * a.tk >= (int64_t)1 << 24;
}
// Outputs and gradients lie as the inputs do; those of the problems above are dense, as they were when these were
// padded (a caller may view the heads and channels of a large output as one).
Tensor attn_out(const Attn &a, const Tensor &t) {
    return copies_pay(a) ? new_buffer(t.sizes(), t.scalar_type(), t.device()) : new_like(t);
}

struct AttnBackward : public Node {
    Attn a;
    SavedVariable q, k, v, o, lse, bias;
    Tensor tiles;

    std::string name() const override { return "FlashAttentionBackward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable *s : {&q, &k, &v, &o, &lse, &bias}) s->reset_data();
        tiles.reset();
    }
#define RGD_SAVED(f)             \
    f(q, false);                 \
    f(k, false);                 \
    f(v, false);                 \
    f(o, true);                  \
    f(lse, false);               \
    if (a.bias_kind != RGD_BIAS_NONE) f(bias, false);
#define RGD_CONSTANTS(f) f(a.causal, a.scale, a.bias_kind);
    RGD_COMPILED(RGD_SAVED, RGD_CONSTANTS)
#undef RGD_SAVED
#undef RGD_CONSTANTS
    variable_list apply(variable_list &&grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        Tensor qt = q.unpack(), kt = k.unpack(), vt = v.unpack(), ot = o.unpack(shared_from_this()), lt = lse.unpack(), bt, tiles;
        if (a.bias_kind != RGD_BIAS_NONE) bt = bias.unpack();
        if (stand_in(qt)) {
            const auto out = call_operator("rgd_b200::attn_bwd", qt, kt, vt, bt.defined() ? c10::IValue(bt) : c10::IValue(), ot, lt,
                                           grads[0].defined() ? grads[0].contiguous() : at::zeros_like(qt), a.causal, a.scale, false);
            return {out.at(0).toTensor(), out.at(1).toTensor(), out.at(2).toTensor()};
        }
        c10::cuda::OptionalCUDAGuard guard(qt.device());
        at::AutoDispatchBelowADInplaceOrView below;
        for (Tensor *t : {&qt, &kt, &vt, &ot, &bt}) *t = unit(*t);
        lt = lt.contiguous();
        Attn a = this->a;       // with the strides of the unpacked bias
        a.bias_kind = RGD_BIAS_NONE;
        a.bias_dtype = RGD_F32;
        restored(attn_ok(a, qt, kt, vt, bt) && a.B == this->a.B && a.H == this->a.H && a.tq == this->a.tq && a.tk == this->a.tk &&
                     a.d == this->a.d && a.dtype == this->a.dtype && a.bias_kind == this->a.bias_kind &&
                     a.bias_dtype == this->a.bias_dtype && plain(ot, 4) && like(ot, qt) && ot.sizes() == qt.sizes() &&
                     lt.scalar_type() == at::kFloat && lt.device() == qt.device() && lt.dim() == 3 && lt.size(0) == a.B &&
                     lt.size(1) == a.H && lt.size(2) == api.attn_lse_rows(a.tq), "FlashAttention");
        // the tile lists are indexed by the bias's broadcast dimensions
        if ((a.bias_sb == 0) == (this->a.bias_sb == 0) && (a.bias_sh == 0) == (this->a.bias_sh == 0)) tiles = this->tiles;
        Tensor dot = upstream(grads[0], qt);
        if (copies_pay(a) && !addressable(dot)) dot = dot.clone(at::MemoryFormat::Contiguous);
        Tensor dq = attn_out(a, qt), dk = attn_out(a, kt), dv = attn_out(a, vt);
        int64_t bytes = std::max<int64_t>(api.attn_bwd_workspace_bytes(a.B, a.H, a.tq, a.tk, a.d, a.dtype), 16);
        if (single_pass.load(std::memory_order_relaxed) && !tiles.defined())
            bytes = std::max(bytes, api.attn_bwd_single_pass_workspace_bytes(a.B, a.H, a.tq, a.tk, a.d, a.dtype));
        Tensor work = new_buffer({bytes}, at::kByte, qt.device());
        const rgd_heads qv = Attn::view(qt), kv = Attn::view(kt), vv = Attn::view(vt), ov = Attn::view(ot), dov = Attn::view(dot),
                        dqv = Attn::view(dq), dkv = Attn::view(dk), dvv = Attn::view(dv);
        const rgd_bias b = a.bias(bt, tiles);
        launched(api.attn_bwd(&qv, &kv, &vv, &b, &ov, lt.data_ptr<float>(), &dov, &dqv, &dkv, &dvv, a.B, a.H, a.tq, a.tk, a.d,
                              (float)a.scale, a.causal ? 1 : 0, a.dtype, work.data_ptr(), bytes,
                              a.state ? a.state->native() : nullptr, stream_of(qt)), "attn_bwd", false);
        note(a.state, 1, qt, kt, vt, dot);
        return {dq, dk, dv};
    }
};

PyObject *attn_call(Attn &a, const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &bias, const Tensor &tiles,
                    bool return_lse) {
    Tensor o, lse;
    {
        NoGil nogil;
        c10::cuda::OptionalCUDAGuard guard(q.device());
        o = attn_out(a, q);
        lse = new_buffer({a.B, a.H, api.attn_lse_rows(a.tq)}, at::kFloat, q.device());
        const rgd_heads qv = Attn::view(q), kv = Attn::view(k), vv = Attn::view(v), ov = Attn::view(o);
        const rgd_bias b = a.bias(bias, tiles);
        launched(api.attn_fwd(&qv, &kv, &vv, &b, &ov, lse.data_ptr<float>(), a.B, a.H, a.tq, a.tk, a.d, (float)a.scale,
                              a.causal ? 1 : 0, a.dtype, a.state ? a.state->native() : nullptr, stream_of(q)), "attn_fwd", true);
        note(a.state, 0, q, k, v);
    }
    if (wants_grad({&q, &k, &v})) {
        auto node = new_node<AttnBackward>(torch::autograd::collect_next_edges(q, k, v));
        node->a = a;
        node->q = SavedVariable(q, false);
        node->k = SavedVariable(k, false);
        node->v = SavedVariable(v, false);
        node->lse = SavedVariable(lse, false);
        if (bias.defined()) node->bias = SavedVariable(bias, false);
        node->tiles = tiles;
        torch::autograd::set_history(o, node);
        node->o = SavedVariable(o, true);
    }
    return return_lse ? wrap2(std::move(o), std::move(lse)) : THPVariable_Wrap(std::move(o));
}

// ------------------------------------------------------------------ Python entries
// C++ exceptions become Python ones; an argument the library refuses hands the call back (None).  Saving a
// tensor runs the user's pack hooks, and what those raise has to come out as it is: torch.utils.checkpoint
// ends its recomputation with an exception of its own.
template <typename F>
PyObject *guarded(F &&f) {
    try {
        if (watched()) Py_RETURN_NONE;
        return f();
    } catch (const Refused &) {
        Py_RETURN_NONE;
    } catch (python_error &e) {
        e.restore();
    } catch (const c10::OutOfMemoryError &e) {
        PyObject *torch = PyImport_ImportModule("torch");
        PyObject *type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
        PyErr_SetString(type ? type : PyExc_RuntimeError, e.what_without_backtrace());
        Py_XDECREF(type);
        Py_XDECREF(torch);
    } catch (const c10::Error &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// rows(cache, eps, affine, x1[, x2][, w1[, w2]])
PyObject *py_rows(PyObject *, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Rows r;
        if (n < 4) Py_RETURN_NONE;
        const bool affine = args[2] == Py_True;
        r.n = (int)(n - 3) / (affine ? 2 : 1);
        if (r.n < 1 || r.n > 2 || r.n * (affine ? 2 : 1) != n - 3 || !state_of(args[0], r.state)) Py_RETURN_NONE;
        r.eps = PyFloat_AsDouble(args[1]);
        if (PyErr_Occurred()) return nullptr;
        for (int i = 0; i < r.n; ++i) {
            if (!tensor_arg(args[3 + i], r.x[i])) Py_RETURN_NONE;
            if (affine && !tensor_arg(args[3 + r.n + i], r.w[i])) Py_RETURN_NONE;
        }
        return rows_call(r);
    });
}

// headln(cache, eps, heads_second, q, k)
PyObject *py_headln(PyObject *, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Heads h;
        Tensor q, k;
        if (n != 5 || !state_of(args[0], h.state) || !tensor_arg(args[3], q) || !tensor_arg(args[4], k)) Py_RETURN_NONE;
        h.eps = PyFloat_AsDouble(args[1]);
        if (PyErr_Occurred()) return nullptr;
        h.heads_second = truth(args[2]);
        if (!heads_ok(h, q, k)) Py_RETURN_NONE;
        return heads_call(h, q, k, Tensor());
    });
}

// rotary(cache, eps or None, heads_second, q, k, pos, seq_cutoff): rotation alone without an eps, else LayerNorm first
PyObject *py_rotary(PyObject *, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Heads h;
        Tensor q, k, pos;
        if (n != 7 || !state_of(args[0], h.state) || !tensor_arg(args[3], q) || !tensor_arg(args[4], k) || !tensor_arg(args[5], pos))
            Py_RETURN_NONE;
        h.op = args[1] == Py_None ? HEAD_ROPE : HEAD_LNROPE;
        if (h.op == HEAD_LNROPE) {
            h.eps = PyFloat_AsDouble(args[1]);
            if (PyErr_Occurred()) return nullptr;
        }
        h.heads_second = truth(args[2]);
        if (!heads_ok(h, q, k) || !table_ok(h, pos, q.device()) || !cutoffs(h, args[6]) || (at::GradMode::is_enabled() && pos.requires_grad()))
            Py_RETURN_NONE;
        return heads_call(h, q, k, pos);
    });
}

// attn(cache, q, k, v, bias or None, tiles or None, causal, scale or None, return_lse)
PyObject *py_attn(PyObject *, PyObject *const *args, Py_ssize_t n) {
    return guarded([&]() -> PyObject * {
        Attn a;
        Tensor q, k, v, bias, tiles;
        if (n != 9 || !state_of(args[0], a.state) || !tensor_arg(args[1], q) || !tensor_arg(args[2], k) || !tensor_arg(args[3], v) ||
            (args[4] != Py_None && !tensor_arg(args[4], bias)) || (args[5] != Py_None && !tensor_arg(args[5], tiles)))
            Py_RETURN_NONE;
        if (!attn_ok(a, q, k, v, bias) || (bias.defined() && at::GradMode::is_enabled() && bias.requires_grad())) Py_RETURN_NONE;
        a.causal = truth(args[6]);
        if (copies_pay(a)) {
            const bool few = a.tq <= 16 && !a.causal && !wants_grad({&q, &k, &v});
            if (!addressable(q, few) || !addressable(k, few) || !addressable(v, few)) Py_RETURN_NONE;
        }
        a.scale = args[7] == Py_None ? 0.0 : PyFloat_AsDouble(args[7]);
        if (PyErr_Occurred()) return nullptr;
        if (a.scale == 0.0) a.scale = 1.0 / sqrt((double)a.d);
        return attn_call(a, q, k, v, bias, tiles, truth(args[8]));
    });
}

PyObject *py_set_single_pass(PyObject *, PyObject *on) {
    single_pass.store(PyObject_IsTrue(on));
    Py_RETURN_NONE;
}

// bind(handle): resolve the C ABI in the library that ctypes opened.
PyObject *py_bind(PyObject *, PyObject *handle) {
    void *h = PyLong_AsVoidPtr(handle);
    if (PyErr_Occurred()) return nullptr;
#define RGD_FN(name)                                                                                                  \
    if (!(api.name = reinterpret_cast<decltype(api.name)>(dlsym(h, "rgd_" #name)))) {                                 \
        PyErr_SetString(PyExc_RuntimeError, "librgd_b200.so does not export rgd_" #name);                             \
        return nullptr;                                                                                               \
    }
    RGD_FUNCTIONS(RGD_FN)
#undef RGD_FN
    Py_RETURN_NONE;
}

// ------------------------------------------------------------------ LaunchState as a Python object
PyObject *state_new(PyTypeObject *type, PyObject *, PyObject *) {
    PyObject *o = type->tp_alloc(type, 0);
    if (o) reinterpret_cast<PyLaunchState *>(o)->state = new State(std::make_shared<LaunchState>());
    return o;
}
void state_dealloc(PyObject *o) {
    delete reinterpret_cast<PyLaunchState *>(o)->state;
    PyTypeObject *t = Py_TYPE(o);
    t->tp_free(o);
    Py_DECREF(t);
}
PyObject *state_native(PyObject *o, PyObject *) {
    return PyLong_FromVoidPtr((*reinterpret_cast<PyLaunchState *>(o)->state)->native());
}
// seen(slot): shapes, strides and types last launched (0 forward, 1 backward), or None
PyObject *state_seen(PyObject *o, PyObject *slot) {
    const long i = PyLong_AsLong(slot);
    if (PyErr_Occurred()) return nullptr;
    LaunchState &s = **reinterpret_cast<PyLaunchState *>(o)->state;
    std::lock_guard<std::mutex> lock(s.mu);
    if (i < 0 || i > 1 || s.seen[i].empty()) Py_RETURN_NONE;
    PyObject *t = PyTuple_New((Py_ssize_t)s.seen[i].size());
    for (size_t j = 0; t && j < s.seen[i].size(); ++j) PyTuple_SET_ITEM(t, j, PyLong_FromLongLong(s.seen[i][j]));
    return t;
}
PyMethodDef state_methods[] = {{"native", state_native, METH_NOARGS, "handle of the library's tensor-map cache"},
                               {"seen", state_seen, METH_O, "what was launched last (0 forward, 1 backward), or None"},
                               {nullptr, nullptr, 0, nullptr}};
PyType_Slot state_slots[] = {{Py_tp_new, reinterpret_cast<void *>(state_new)},
                             {Py_tp_dealloc, reinterpret_cast<void *>(state_dealloc)},
                             {Py_tp_methods, state_methods},
                             {0, nullptr}};
PyType_Spec state_spec = {"rgd_triton_b200._host.LaunchState", sizeof(PyLaunchState), 0, Py_TPFLAGS_DEFAULT, state_slots};

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(f)), METH_FASTCALL
PyMethodDef methods[] = {{"bind", py_bind, METH_O, "bind the C ABI of an opened librgd_b200"},
                         {"set_single_pass", py_set_single_pass, METH_O, "how the attention backward forms dQ"},
                         {"rows", FAST(py_rows), "L2 / RMS norm of one or two [B, N, C] tensors"},
                         {"headln", FAST(py_headln), "LayerNorm over head_dim of q and k"},
                         {"rotary", FAST(py_rotary), "rotary embedding of q and k, LayerNorm first when an eps is given"},
                         {"attn", FAST(py_attn), "attention"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "native host path of the operator set", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    PyObject *m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    str_state = PyUnicode_InternFromString("_state");
    launch_state_type = reinterpret_cast<PyTypeObject *>(PyType_FromSpec(&state_spec));
    if (!str_state || !launch_state_type || PyModule_AddObjectRef(m, "LaunchState", reinterpret_cast<PyObject *>(launch_state_type)) < 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
