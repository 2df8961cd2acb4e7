// The operator's host path on PyTorch tensors: stage calls, autograd nodes and the argument fast path.
//
// Why native: with Python autograd functions around ctypes calls, a second-order step over a small layer
// (forward, first gradients kept in the graph, second gradients; five kernels) cost 390 us of host time
// whatever its size, on a GPU that needs a fraction of that; the nodes below run without the interpreter.
//
// PyTorch supplies device memory, streams and the autograd engine; all arithmetic is in libbob_sm100.so,
// whose entry points flashbob_b200/_native.py hands over as addresses (one library per process, wherever
// it was loaded from).  The autograd protocol is the reference's (reference: src/bob/sdpa.py:239-368):
//   * SdpaNode::apply runs only the first backward when grad mode is off, otherwise it also records a
//     SecondOrderNode over (q, k, v, dO), whose apply is the second backward;
//   * undefined incoming gradients stay undefined and switch off the products they would feed.
#include "../../include/bob_sm100.h"

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <cmath>
#include <optional>

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ---- the library ------------------------------------------------------------------------------------
struct Library {
    decltype(&bob_sm100_fwd) fwd = nullptr;
    decltype(&bob_sm100_bwd1) bwd1 = nullptr;
    decltype(&bob_sm100_bwd2) bwd2 = nullptr;
    decltype(&bob_sm100_workspace_bytes) workspace_bytes = nullptr;
    decltype(&bob_sm100_read_status) read_status = nullptr;
    decltype(&bob_sm100_last_status) last_status = nullptr;
    decltype(&bob_sm100_error_string) error_string = nullptr;
};
Library lib;
PyObject* error_class = nullptr;           // BobSm100Error

[[noreturn]] void fail(const std::string& what, int rc) {
    // the Python exception class is kept, also from the autograd engine's threads
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(error_class, (what + " failed with code " + std::to_string(rc) + ": " + lib.error_string(rc)).c_str());
    python_error e;
    e.persist();
    throw e;
}

struct Mask {
    bool causal = false;
    int window = 0;
    int64_t q_offset = 0, k_offset = 0;
    std::optional<double> scale;           // none: 1 / sqrt(D)
    bool check_status = false;             // wait for the stream after each stage and read its status word
};

// In-place addressing needs unit stride along the head dim, batch / head / row strides that are positive
// multiples of 8 elements (16 bytes) and a 16-byte aligned base; anything else is made contiguous.
Tensor tma_ready(const Tensor& t) {
    bool ok = t.stride(3) == 1 && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
    for (int i = 0; i < 3; ++i) ok = ok && t.stride(i) % 8 == 0 && (t.stride(i) > 0 || t.size(i) == 1);
    return ok ? t : t.contiguous();
}

void set_strides(int64_t (&field)[3], const Tensor& t) {
    for (int i = 0; i < 3; ++i) field[i] = t.stride(i);
}

bob_sm100_geom geometry(const Tensor& q, const Tensor& k, const Mask& m) {
    bob_sm100_geom g = {};
    g.B = static_cast<int32_t>(q.size(0)); g.Hq = static_cast<int32_t>(q.size(1)); g.Hkv = static_cast<int32_t>(k.size(1));
    g.Nq = static_cast<int32_t>(q.size(2)); g.Nk = static_cast<int32_t>(k.size(2)); g.D = static_cast<int32_t>(q.size(3));
    g.dtype = q.scalar_type() == at::kBFloat16 ? BOB_SM100_BF16 : BOB_SM100_FP16;
    g.is_causal = m.causal;
    g.window = m.window;
    g.device = q.device().index();
    g.flags = BOB_SM100_SPLIT_KEYS;        // (every workspace below is sized for its own call)
    g.q_offset = m.q_offset;
    g.k_offset = m.k_offset;
    g.scale = static_cast<float>(m.scale ? *m.scale : 1.0 / std::sqrt(static_cast<double>(g.D)));
    return g;
}

Tensor empty(at::IntArrayRef size, at::ScalarType type, const Tensor& like) {
    return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
}
Tensor workspace(int stage, const bob_sm100_geom& g, const Tensor& like) {
    return empty({static_cast<int64_t>(lib.workspace_bytes(stage, &g))}, at::kByte, like);
}
void* ptr(const Tensor& t) { return t.defined() ? const_cast<void*>(t.const_data_ptr()) : nullptr; }
float* fptr(const Tensor& t) { return static_cast<float*>(ptr(t)); }
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// Raises if a kernel on this device gave up on a bounded wait: by default a non-blocking look at the
// device's host-visible status word (a time-out of an earlier call surfaces here), with `check_status` the
// call's own status word after waiting for the stream.
void finish(int rc, const char* what, const Mask& m, const Tensor& ws) {
    if (rc) fail(what, rc);
    if (m.check_status && (rc = lib.read_status(ptr(ws), stream_of(ws)))) fail(std::string(what) + " (device status)", rc);
    if ((rc = lib.last_status(ws.device().index())))
        fail("an earlier libbob_sm100 kernel on cuda:" + std::to_string(ws.device().index()) + " (seen after " + what +
             "; its results are undefined)", rc);
}

// ---- the three stages -------------------------------------------------------------------------------
struct Forward { Tensor out, lse; };
Forward run_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Mask& m) {
    const Tensor q = tma_ready(q_), k = tma_ready(k_), v = tma_ready(v_);
    bob_sm100_geom g = geometry(q, k, m);
    set_strides(g.q_strides, q); set_strides(g.k_strides, k); set_strides(g.v_strides, v);
    Forward r{empty(q.sizes(), q.scalar_type(), q), empty(q.sizes().slice(0, 3), at::kFloat, q)};
    const Tensor ws = workspace(BOB_SM100_STAGE_FWD, g, q);
    const int rc = lib.fwd(&g, ptr(q), ptr(k), ptr(v), ptr(r.out), fptr(r.lse), ptr(ws), stream_of(q));
    finish(rc, "bob_sm100_fwd", m, ws);
    return r;
}

struct First { Tensor dQ, dK, dV, delta, pk; };
First run_first(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& out_, const Tensor& lse_,
                const Tensor& dO_, const Mask& m, bool for_second_order) {
    const Tensor q = tma_ready(q_), k = tma_ready(k_), v = tma_ready(v_), out = tma_ready(out_), dO = tma_ready(dO_);
    const Tensor lse = lse_.contiguous();
    bob_sm100_geom g = geometry(q, k, m);
    set_strides(g.q_strides, q); set_strides(g.k_strides, k); set_strides(g.v_strides, v);
    set_strides(g.out_strides, out); set_strides(g.do_strides, dO);
    First r{empty(q.sizes(), q.scalar_type(), q), empty(k.sizes(), q.scalar_type(), q), empty(k.sizes(), q.scalar_type(), q),
            empty(q.sizes().slice(0, 3), at::kFloat, q), for_second_order ? empty(q.sizes(), at::kFloat, q) : Tensor()};
    const Tensor ws = workspace(BOB_SM100_STAGE_BWD1, g, q);
    const int rc = lib.bwd1(&g, ptr(q), ptr(k), ptr(v), ptr(out), fptr(lse), ptr(dO), ptr(r.dQ), ptr(r.dK), ptr(r.dV),
                            fptr(r.delta), fptr(r.pk), ptr(ws), stream_of(q));
    finish(rc, "bob_sm100_bwd1", m, ws);
    return r;
}

struct Second { Tensor Qbar, Kbar, Vbar, dObar; };
Second run_second(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& out_, const Tensor& lse_,
                  const Tensor& delta_, const Tensor& pk_, const Tensor& dO_, const Tensor& dQ_, const Tensor& uQ_,
                  const Tensor& uK_, const Tensor& uV_, const Mask& m) {
    const Tensor q = tma_ready(q_), k = tma_ready(k_), v = tma_ready(v_), out = tma_ready(out_), dO = tma_ready(dO_), dQ = tma_ready(dQ_);
    auto tangent = [&](const Tensor& t) { return t.defined() ? tma_ready(t.scalar_type() == q.scalar_type() ? t : t.to(q.scalar_type())) : t; };
    const Tensor uQ = tangent(uQ_), uK = tangent(uK_), uV = tangent(uV_);
    const Tensor lse = lse_.contiguous(), delta = delta_.contiguous(), pk = pk_.contiguous();
    bob_sm100_geom g = geometry(q, k, m);
    set_strides(g.q_strides, q); set_strides(g.k_strides, k); set_strides(g.v_strides, v);
    set_strides(g.out_strides, out); set_strides(g.do_strides, dO); set_strides(g.dq_strides, dQ);
    if (uQ.defined()) set_strides(g.uq_strides, uQ);
    if (uK.defined()) set_strides(g.uk_strides, uK);
    if (uV.defined()) set_strides(g.uv_strides, uV);
    Second r{empty(q.sizes(), q.scalar_type(), q), empty(k.sizes(), q.scalar_type(), q), empty(k.sizes(), q.scalar_type(), q),
             empty(q.sizes(), q.scalar_type(), q)};
    const Tensor ws = workspace(BOB_SM100_STAGE_BWD2, g, q);
    const int rc = lib.bwd2(&g, ptr(q), ptr(k), ptr(v), ptr(out), fptr(lse), fptr(delta), fptr(pk), ptr(dO), ptr(dQ), ptr(uQ),
                            ptr(uK), ptr(uV), ptr(r.Qbar), ptr(r.Kbar), ptr(r.Vbar), ptr(r.dObar), ptr(ws), stream_of(q));
    finish(rc, "bob_sm100_bwd2", m, ws);
    return r;
}

// ---- autograd nodes ---------------------------------------------------------------------------------
// The nodes call the library below PyTorch's dispatcher; copies of awkwardly strided inputs must not be
// recorded on the tape either.
struct Untracked {
    at::AutoGradMode grad_off{false};
    at::AutoDispatchBelowADInplaceOrView below;
};

// deleteNode frees a graph node by node; a plain destructor would free a node's predecessors inside its own, one
// stack frame deeper for each of a chain of calls.
template <class N> std::shared_ptr<N> make_node() { return std::shared_ptr<N>(new N(), torch::autograd::deleteNode); }

// First backward as a differentiable function of (q, k, v, dO): its gradient is the second backward.
struct SecondOrderNode : Node {
    Mask mask;
    SavedVariable q, k, v, dO, out, lse, dQ, delta, pk;
    std::string name() const override { return "BoBSecondOrderBackward"; }
    variable_list apply(variable_list&& u) override {
        std::lock_guard<std::mutex> lock(mutex_);
        if (!u[0].defined() && !u[1].defined() && !u[2].defined()) return variable_list(4);
        const Tensor q_ = q.unpack(), k_ = k.unpack(), v_ = v.unpack(), dO_ = dO.unpack(), out_ = out.unpack(), lse_ = lse.unpack(),
                     dQ_ = dQ.unpack(shared_from_this()), delta_ = delta.unpack(), pk_ = pk.unpack();
        Untracked untracked;
        const c10::cuda::CUDAGuard device(q_.device());
        Second r = run_second(q_, k_, v_, out_, lse_, delta_, pk_, dO_, dQ_, u[0], u[1], u[2], mask);
        return {r.Qbar, r.Kbar, r.Vbar, r.dObar};
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* s : {&q, &k, &v, &dO, &out, &lse, &dQ, &delta, &pk}) s->reset_data();
    }
};

// Attention forward whose gradient is itself differentiable once more.
struct SdpaNode : Node {
    Mask mask;
    SavedVariable q, k, v, out, lse;
    std::string name() const override { return "SDPAWithBoBBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        const Tensor& dO = grads[0];
        if (!dO.defined()) return variable_list(3);
        const Tensor q_ = q.unpack(), k_ = k.unpack(), v_ = v.unpack(), out_ = out.unpack(shared_from_this()), lse_ = lse.unpack();
        const bool record = torch::autograd::compute_requires_grad(q_, k_, v_, dO);
        // a graph that is kept would hold a derivative from which the tangent's term is missing
        TORCH_CHECK_NOT_IMPLEMENTED(!record || !dO._fw_grad(0).defined(), "forward-mode AD is unsupported; differentiate with "
                                    "reverse mode (torch.autograd.grad twice) instead");
        First r;
        {
            Untracked untracked;
            const c10::cuda::CUDAGuard device(q_.device());
            r = run_first(q_, k_, v_, out_, lse_, dO, mask, record);
        }
        if (record) {
            auto node = make_node<SecondOrderNode>();
            node->set_next_edges(torch::autograd::collect_next_edges(q_, k_, v_, dO));
            node->mask = mask;
            node->q = SavedVariable(q_, false); node->k = SavedVariable(k_, false); node->v = SavedVariable(v_, false);
            node->dO = SavedVariable(dO, false); node->out = SavedVariable(out_.detach(), false); node->lse = SavedVariable(lse_, false);
            node->delta = SavedVariable(r.delta, false); node->pk = SavedVariable(r.pk, false);
            for (const Tensor& t : {r.dQ, r.dK, r.dV}) torch::autograd::set_history(t, node);
            node->dQ = SavedVariable(r.dQ, true);
        }
        return {r.dQ, r.dK, r.dV};
    }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        for (SavedVariable* s : {&q, &k, &v, &out, &lse}) s->reset_data();
    }
};

Tensor sdpa(const Tensor& q, const Tensor& k, const Tensor& v, const Mask& m) {
    const bool record = torch::autograd::compute_requires_grad(q, k, v);
    Forward r;
    {
        Untracked untracked;
        const c10::cuda::CUDAGuard device(q.device());
        r = run_forward(q, k, v, m);
    }
    if (record) {
        auto node = make_node<SdpaNode>();
        node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
        node->mask = m;
        node->q = SavedVariable(q, false); node->k = SavedVariable(k, false); node->v = SavedVariable(v, false);
        node->lse = SavedVariable(r.lse, false);
        torch::autograd::set_history(r.out, node);
        node->out = SavedVariable(r.out, true);
    }
    return r.out;
}

// ---- Python entry points ----------------------------------------------------------------------------
bool is_int(PyObject* o) { return PyLong_CheckExact(o); }       // a bool is a subclass: not exact

// The argument checks of sdpa_bob in their common, valid form.  Anything else - a CPU tensor, an int-like
// that is no int, a grouped call with a window, an invalid shape, a call that torch.jit.trace records - is left
// to the Python side, which raises or resolves it; its checks are the one statement of what is allowed.
bool common_call(const Tensor& q, const Tensor& k, const Tensor& v, PyObject* causal, PyObject* scale, PyObject* window,
                 PyObject* q_offset, PyObject* k_offset, Mask& m) {
    if (torch::jit::tracer::isTracing()) return false;
    const auto type = q.scalar_type();
    if (!q.is_cuda() || q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || (type != at::kHalf && type != at::kBFloat16)) return false;
    if (k.scalar_type() != type || v.scalar_type() != type || k.device() != q.device() || v.device() != q.device()) return false;
    if (k.sizes() != v.sizes() || q.numel() <= 0 || k.numel() <= 0) return false;
    const int64_t n_q = q.size(2), n_k = k.size(2), D = q.size(3), group = q.size(1) / k.size(1);
    if (k.size(0) != q.size(0) || k.size(3) != D || group * k.size(1) != q.size(1) || (D != 32 && D != 64 && D != 128)) return false;
    if (n_q > INT32_MAX || n_k > INT32_MAX || q.size(0) > INT32_MAX || q.size(1) > INT32_MAX) return false;
    for (const Tensor* t : {&q, &k, &v})
        if (t->_fw_grad(0).defined()) return false;
    if (!PyBool_Check(causal) || !is_int(window) || !is_int(k_offset) || !(q_offset == Py_None || is_int(q_offset))) return false;
    m.causal = causal == Py_True;
    auto count = [](PyObject* o, int64_t& x) {
        int overflow = 0;
        x = PyLong_AsLongLongAndOverflow(o, &overflow);
        return !overflow && x >= 0 && x < (int64_t(1) << 40);
    };
    int64_t w = 0;
    if (!count(window, w) || !count(k_offset, m.k_offset)) return false;
    if (w > 0 && !m.causal) return false;
    if (q_offset != Py_None) {
        if (!count(q_offset, m.q_offset)) return false;
    } else {                               // a causal rectangle defaults to right alignment
        m.q_offset = m.k_offset + (m.causal && n_k > n_q ? n_k - n_q : 0);
    }
    const bool rectangular = n_q != n_k || m.q_offset != m.k_offset;
    // a window that already covers every causal key is no window
    if (m.causal && w > 0 && w >= (rectangular ? m.q_offset - m.k_offset + n_q : n_q)) w = 0;
    if (w > INT32_MAX) return false;
    m.window = static_cast<int>(w);
    if (group > 1 && (rectangular || w > 0 || type != at::kBFloat16 || group > 32)) return false;
    if (scale != Py_None) {
        if (!PyFloat_CheckExact(scale)) return false;
        const float s = static_cast<float>(PyFloat_AS_DOUBLE(scale));
        if (!(s > 0) || !std::isfinite(s)) return false;
        m.scale = PyFloat_AS_DOUBLE(scale);
    }
    return true;
}

const Tensor& tensor_arg(PyObject* o) {
    if (!THPVariable_Check(o)) throw torch::TypeError("expected a torch.Tensor");
    return THPVariable_Unpack(o);
}
Tensor optional_tensor_arg(PyObject* o) { return o == Py_None ? Tensor() : tensor_arg(o); }

int64_t int_arg(PyObject* o) {
    const int64_t x = PyLong_AsLongLong(o);
    if (x == -1 && PyErr_Occurred()) throw python_error();
    return x;
}

// (is_causal, window_size, q_offset, k_offset, scale or None, check_status), all checked by the caller
Mask mask_args(PyObject* const* a) {
    Mask m;
    m.causal = PyObject_IsTrue(a[0]);
    m.window = static_cast<int>(int_arg(a[1]));
    m.q_offset = int_arg(a[2]);
    m.k_offset = int_arg(a[3]);
    if (a[4] != Py_None) {
        m.scale = PyFloat_AsDouble(a[4]);
        if (PyErr_Occurred()) throw python_error();
    }
    m.check_status = PyObject_IsTrue(a[5]);
    return m;
}

template <class F> auto without_gil(F f) {
    pybind11::gil_scoped_release released;
    return f();
}

void want(Py_ssize_t got, Py_ssize_t n) {
    if (got != n) throw torch::TypeError("expected " + std::to_string(n) + " arguments, got " + std::to_string(got));
}

PyObject* tuple_of(std::initializer_list<Tensor> ts) {
    PyObject* r = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
    Py_ssize_t i = 0;
    for (const Tensor& t : ts) PyTuple_SET_ITEM(r, i++, THPVariable_Wrap(t));     // None for an undefined tensor
    return r;
}

// try_sdpa(q, k, v, is_causal, scale, window_size, q_offset, k_offset, check_status) -> out, or None when
// the call is not in the common form
PyObject* py_try_sdpa(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want(n, 9);
    if (!THPVariable_Check(a[0]) || !THPVariable_Check(a[1]) || !THPVariable_Check(a[2])) Py_RETURN_NONE;
    const Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
    Mask m;
    if (!common_call(q, k, v, a[3], a[4], a[5], a[6], a[7], m)) Py_RETURN_NONE;
    m.check_status = PyObject_IsTrue(a[8]);
    return THPVariable_Wrap(without_gil([&] { return sdpa(q, k, v, m); }));
    END_HANDLE_TH_ERRORS
}

// sdpa(q, k, v, <mask>) -> out; arguments checked and resolved by the caller
PyObject* py_sdpa(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want(n, 9);
    const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]);
    const Mask m = mask_args(a + 3);
    return THPVariable_Wrap(without_gil([&] { return sdpa(q, k, v, m); }));
    END_HANDLE_TH_ERRORS
}

// forward(q, k, v, <mask>) -> (out, lse)
PyObject* py_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want(n, 9);
    Untracked untracked;
    const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]);
    const Mask m = mask_args(a + 3);
    const c10::cuda::CUDAGuard device(q.device());
    Forward r = without_gil([&] { return run_forward(q, k, v, m); });
    return tuple_of({r.out, r.lse});
    END_HANDLE_TH_ERRORS
}

// first_backward(q, k, v, out, lse, dO, <mask>, for_second_order) -> (dQ, dK, dV, delta, pk)
PyObject* py_first(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want(n, 13);
    Untracked untracked;
    const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]), &out = tensor_arg(a[3]), &lse = tensor_arg(a[4]),
                 &dO = tensor_arg(a[5]);
    const Mask m = mask_args(a + 6);
    const bool for_second_order = PyObject_IsTrue(a[12]);
    const c10::cuda::CUDAGuard device(q.device());
    First r = without_gil([&] { return run_first(q, k, v, out, lse, dO, m, for_second_order); });
    return tuple_of({r.dQ, r.dK, r.dV, r.delta, r.pk});
    END_HANDLE_TH_ERRORS
}

// second_backward(q, k, v, out, lse, delta, pk, dO, dQ, uQ, uK, uV, <mask>) -> (Qbar, Kbar, Vbar, dObar)
PyObject* py_second(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want(n, 18);
    Untracked untracked;
    const Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]), &out = tensor_arg(a[3]), &lse = tensor_arg(a[4]),
                 &delta = tensor_arg(a[5]), &pk = tensor_arg(a[6]), &dO = tensor_arg(a[7]), &dQ = tensor_arg(a[8]);
    const Tensor uQ = optional_tensor_arg(a[9]), uK = optional_tensor_arg(a[10]), uV = optional_tensor_arg(a[11]);
    const Mask m = mask_args(a + 12);
    const c10::cuda::CUDAGuard device(q.device());
    Second r = without_gil([&] { return run_second(q, k, v, out, lse, delta, pk, dO, dQ, uQ, uK, uV, m); });
    return tuple_of({r.Qbar, r.Kbar, r.Vbar, r.dObar});
    END_HANDLE_TH_ERRORS
}

// bind(error class, addresses of fwd, bwd1, bwd2, workspace_bytes, read_status, last_status, error_string)
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    want(n, 8);
    auto address = [&](int i) { return reinterpret_cast<void*>(int_arg(a[i])); };
    Py_INCREF(a[0]);
    error_class = a[0];
    lib.fwd = reinterpret_cast<decltype(lib.fwd)>(address(1));
    lib.bwd1 = reinterpret_cast<decltype(lib.bwd1)>(address(2));
    lib.bwd2 = reinterpret_cast<decltype(lib.bwd2)>(address(3));
    lib.workspace_bytes = reinterpret_cast<decltype(lib.workspace_bytes)>(address(4));
    lib.read_status = reinterpret_cast<decltype(lib.read_status)>(address(5));
    lib.last_status = reinterpret_cast<decltype(lib.last_status)>(address(6));
    lib.error_string = reinterpret_cast<decltype(lib.error_string)>(address(7));
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

#define BOB_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    BOB_METHOD("try_sdpa", py_try_sdpa), BOB_METHOD("sdpa", py_sdpa), BOB_METHOD("forward", py_forward),
    BOB_METHOD("first_backward", py_first), BOB_METHOD("second_backward", py_second), BOB_METHOD("bind", py_bind),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "bob_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_bob_torch() { return PyModule_Create(&module_def); }
