// The host path of the operators in native code: the CPython module `brainpylib_b200._native`.
//
// One operator call on CUDA tensors costs a few microseconds of device time for a small network, and the same call
// written in Python (argument checks one by one, a Python autograd.Function, ctypes, a descriptor, a workspace look-up)
// cost 45-60 us of host time, several times the kernels.  The functions here do the same work on the C++ tensors:
// check, allocate the output, launch; the autograd rules are C++ nodes.
//
// Contract with the Python operators: a function returns None whenever the call is not the plain case it handles
// (operands that are no CUDA tensors, anything that would raise, dtypes to convert, non-contiguous tensors, functorch
// transforms, forward-mode duals, dispatch modes, tracing).  The Python code behind it then runs as it always did and raises,
// converts or differentiates; so no check and no error message lives here twice.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <stdexcept>
#include <string>

#include "abi.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

using Target = void (*)(bpl_stream_t, void **, const char *, size_t);

// ---------------------------------------------------------------------------------------------------------
// operands
// ---------------------------------------------------------------------------------------------------------
// A plain strided CUDA tensor carries these keys only; a wrapped one (functorch, fake, functional, subclass) more.
bool plain_keys(const Tensor &t) {
    static const uint64_t allowed = c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView,
                                                         c10::DispatchKey::AutogradCUDA,
                                                         c10::DispatchKey::AutocastCUDA}).raw_repr();
    return (t.key_set().raw_repr() & ~allowed) == 0;
}

// no functorch transform and no dispatch mode is active on this thread
bool untransformed() {
    return !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
           !c10::impl::TorchDispatchModeTLS::any_modes_set();
}
// nor a tracer: torch.jit.trace records the Python autograd functions
bool plain_thread() { return untransformed() && !at::tracer::impl::is_dispatch_enabled(); }

bool plain(const Tensor &t) {
    return t.defined() && plain_keys(t) && t.is_contiguous() &&
           !(c10::isFloatingType(t.scalar_type()) && t._fw_grad(0).defined());
}

const Tensor *tensor_of(PyObject *o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const Tensor &t = THPVariable_Unpack(o);
    return plain(t) ? &t : nullptr;
}

bool int32_like(const Tensor &t) { return t.scalar_type() == at::kInt || t.scalar_type() == at::kUInt32; }
bool float_like(const Tensor &t) { return t.scalar_type() == at::kFloat || t.scalar_type() == at::kDouble; }
bool is_double(const Tensor &t) { return t.scalar_type() == at::kDouble; }

bool shape_of(PyObject *o, int64_t &a, int64_t &b) {
    if (!PyTuple_CheckExact(o) || PyTuple_GET_SIZE(o) != 2) return false;
    PyObject *x = PyTuple_GET_ITEM(o, 0), *y = PyTuple_GET_ITEM(o, 1);
    if (!PyLong_CheckExact(x) || !PyLong_CheckExact(y)) return false;
    int over_a = 0, over_b = 0;
    a = PyLong_AsLongLongAndOverflow(x, &over_a);
    b = PyLong_AsLongLongAndOverflow(y, &over_b);
    return !over_a && !over_b && a >= 0 && b >= 0 && a <= 0xffffffffll && b <= 0xffffffffll;
}

// Python numbers of the exact types only: what else converts to a number goes the Python way
bool number_of(PyObject *o, double &v) {
    if (PyFloat_CheckExact(o)) {
        v = PyFloat_AS_DOUBLE(o);
        return true;
    }
    if (PyLong_CheckExact(o)) {
        v = PyLong_AsDouble(o);
        if (v == -1.0 && PyErr_Occurred()) {
            PyErr_Clear();
            return false;
        }
        return true;
    }
    return false;
}

bool wants_grad(const Tensor &t) { return t.requires_grad() && at::GradMode::is_enabled(); }

// ---------------------------------------------------------------------------------------------------------
// calling a target
// ---------------------------------------------------------------------------------------------------------
// A launch waits where the stream's queue is full, an allocation where memory has to be freed: other Python threads run
// meanwhile.  (Backward passes come here without the lock.)
struct NoGil {
    PyThreadState *state = PyGILState_Check() ? PyEval_SaveThread() : nullptr;
    NoGil() = default;
    ~NoGil() {
        if (state) PyEval_RestoreThread(state);
    }
    NoGil(const NoGil &) = delete;
    NoGil &operator=(const NoGil &) = delete;
};

// Scratch of one call, from torch's stream-ordered allocator: taken and given back around the launches, so calls of
// several threads and streams never share it, and the memory serves other tensors in between.
struct Scratch {
    void *ptr = nullptr;
    Scratch(size_t bytes, cudaStream_t stream) {
        if (bytes) ptr = c10::cuda::CUDACachingAllocator::raw_alloc_with_stream(bytes, stream);
    }
    ~Scratch() {
        if (ptr) c10::cuda::CUDACachingAllocator::raw_delete(ptr);
    }
    Scratch(const Scratch &) = delete;
    Scratch &operator=(const Scratch &) = delete;
};

void check_status() {
    if (bpl_last_status(nullptr, 0) == 0) return;
    char message[256];
    const int code = bpl_last_status(message, sizeof(message));
    bpl_clear_status();
    if (code == BPL_ERR_OPAQUE_SIZE) throw std::runtime_error(message[0] ? message : "Invalid opaque object size");
    throw std::runtime_error("brainpylib_b200 kernel error (" + std::to_string(code) + "): " + message);
}

Tensor new_tensor(at::IntArrayRef size, at::ScalarType dtype, const c10::Device &device) {
    return Tensor(at::detail::empty_cuda(size, dtype, device, std::nullopt));
}

// the device of `t` is current while this lives
struct OnDevice {
    c10::cuda::OptionalCUDAGuard guard;
    cudaStream_t stream;
    explicit OnDevice(const Tensor &t) {
        const auto index = t.device().index();
        if (c10::cuda::current_device() != index) guard.set_index(index);
        stream = c10::cuda::getCurrentCUDAStream(index).stream();
    }
};

void *ptr(const Tensor &t) { return const_cast<void *>(t.const_data_ptr()); }

// ---------------------------------------------------------------------------------------------------------
// stored matrices
// ---------------------------------------------------------------------------------------------------------
Tensor csr_product(const Tensor &data, const Tensor &indices, const Tensor &indptr, const Tensor &vector, int64_t n_row,
                   int64_t n_col, bool transpose) {
    NoGil no_gil;
    OnDevice on(data);
    Tensor out = new_tensor({transpose ? n_col : n_row}, data.scalar_type(), data.device());
    bpl_csr_matvec(on.stream, ptr(data), ptr(indices), ptr(indptr), ptr(vector), ptr(out), static_cast<uint32_t>(n_row),
                   static_cast<uint32_t>(n_col), static_cast<uint32_t>(indices.size(0)), data.size(0) == 1, is_double(data),
                   transpose);
    check_status();
    return out;
}

Tensor event_csr_product(const Tensor &data, const Tensor &indices, const Tensor &indptr, const Tensor &events,
                         int64_t n_row, int64_t n_col, bool transpose) {
    NoGil no_gil;
    OnDevice on(data);
    Tensor out = new_tensor({transpose ? n_col : n_row}, data.scalar_type(), data.device());
    Scratch ws(bpl_event_csr_matvec_workspace(static_cast<uint32_t>(n_row), static_cast<uint32_t>(n_col),
                                              static_cast<uint32_t>(indices.size(0)), data.size(0) == 1, is_double(data), transpose),
               on.stream);
    void *buffers[6] = {ptr(data), ptr(indices), ptr(indptr), ptr(events), ptr(out), ws.ptr};
    bpl_event_csr_matvec(on.stream, buffers, static_cast<uint32_t>(n_row), static_cast<uint32_t>(n_col),
                         static_cast<uint32_t>(indices.size(0)), data.size(0) == 1, is_double(data),
                         events.scalar_type() == at::kBool, transpose);
    check_status();
    return out;
}

// ---------------------------------------------------------------------------------------------------------
// differentiation rules (the Python rules of event_ops.py and sparse_ops.py, on C++ nodes)
// ---------------------------------------------------------------------------------------------------------
// Where a cotangent is not a plain tensor (batched gradients, forward over reverse) the Python rule takes over.
PyObject *g_event_csr_backward = nullptr, *g_csr_backward = nullptr, *g_csr_outer = nullptr;

bool plain_cotangent(const Tensor &ct) { return plain_keys(ct) && plain_thread() && !ct._fw_grad(0).defined(); }

// fn(tensors..., n_row, n_col, transpose, need_a, need_b) -> (a or None, b or None)
std::pair<Tensor, Tensor> python_rule(PyObject *fn, std::initializer_list<Tensor> tensors, int64_t n_row, int64_t n_col,
                                      bool transpose, bool need_a, bool need_b) {
    pybind11::gil_scoped_acquire gil;
    const size_t n = tensors.size() + 5;
    pybind11::tuple args(n);
    size_t i = 0;
    for (const Tensor &t : tensors) args[i++] = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(t));
    args[i++] = pybind11::int_(n_row);
    args[i++] = pybind11::int_(n_col);
    args[i++] = pybind11::bool_(transpose);
    args[i++] = pybind11::bool_(need_a);
    args[i++] = pybind11::bool_(need_b);
    PyObject *r = PyObject_CallObject(fn, args.ptr());
    if (r == nullptr) throw python_error();
    const auto owned = pybind11::reinterpret_steal<pybind11::object>(r);
    auto item = [&](int k) {
        PyObject *o = PyTuple_GET_ITEM(r, k);
        return o == Py_None ? Tensor() : THPVariable_Unpack(o);
    };
    return {item(0), item(1)};
}

struct CsrFn : public torch::autograd::Function<CsrFn> {
    static Tensor forward(AutogradContext *ctx, const Tensor &data, const Tensor &indices, const Tensor &indptr,
                          const Tensor &vector, int64_t n_row, int64_t n_col, bool transpose) {
        ctx->save_for_backward({data, indices, indptr, vector});
        ctx->saved_data["r"] = n_row;
        ctx->saved_data["c"] = n_col;
        ctx->saved_data["t"] = transpose;
        return csr_product(data, indices, indptr, vector, n_row, n_col, transpose);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads);
};

Tensor csr_outer(const Tensor &row_vector, const Tensor &col_vector, const Tensor &indices, const Tensor &indptr) {
    NoGil no_gil;
    OnDevice on(indices);
    Tensor out = new_tensor({indices.size(0)}, row_vector.scalar_type(), row_vector.device());
    bpl_csr_outer(on.stream, ptr(row_vector), ptr(col_vector), ptr(indices), ptr(indptr), ptr(out),
                  static_cast<uint32_t>(indptr.size(0) - 1), static_cast<uint32_t>(col_vector.size(0)),
                  static_cast<uint32_t>(indices.size(0)), is_double(row_vector) ? 1 : 0);
    check_status();
    return out;
}

// g[e] = row_vector[row(e)] * col_vector[indices[e]] over the stored entries: the gradient of a product with respect to
// the weights.  Bilinear, and its own derivatives are products with the matrix of cotangents.
struct CsrOuterFn : public torch::autograd::Function<CsrOuterFn> {
    static Tensor forward(AutogradContext *ctx, const Tensor &row_vector, const Tensor &col_vector, const Tensor &indices,
                          const Tensor &indptr) {
        ctx->save_for_backward({row_vector, col_vector, indices, indptr});
        return csr_outer(row_vector, col_vector, indices, indptr);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &row = saved[0], &col = saved[1], &indices = saved[2], &indptr = saved[3];
        const Tensor g = grads[0].contiguous();
        const int64_t n_row = row.size(0), n_col = col.size(0);
        Tensor g_row, g_col;
        if (!plain_cotangent(g)) {
            std::tie(g_row, g_col) = python_rule(g_csr_outer, {row, col, indices, indptr, g}, n_row, n_col, false,
                                                 ctx->needs_input_grad(0), ctx->needs_input_grad(1));
        } else {
            if (ctx->needs_input_grad(0)) g_row = CsrFn::apply(g, indices, indptr, col, n_row, n_col, false);
            if (ctx->needs_input_grad(1)) g_col = CsrFn::apply(g, indices, indptr, row, n_row, n_col, true);
        }
        return {g_row, g_col, Tensor(), Tensor()};
    }
};

// In a backward pass without create_graph there is nothing to record: the kernels alone.
Tensor csr_any(const Tensor &data, const Tensor &indices, const Tensor &indptr, const Tensor &x, int64_t n_row, int64_t n_col, bool t) {
    return at::GradMode::is_enabled() ? CsrFn::apply(data, indices, indptr, x, n_row, n_col, t)
                                      : csr_product(data, indices, indptr, x, n_row, n_col, t);
}

Tensor outer_of(const Tensor &indices, const Tensor &indptr, const Tensor &x, const Tensor &ct, bool transpose) {
    const Tensor &row = transpose ? x : ct, &col = transpose ? ct : x;
    return at::GradMode::is_enabled() ? CsrOuterFn::apply(row, col, indices, indptr) : csr_outer(row, col, indices, indptr);
}

// Both gradients of a product of per-entry weights, without a graph of their own: (of the weights, of the vector)
std::pair<Tensor, Tensor> csr_gradients(const Tensor &data, const Tensor &indices, const Tensor &indptr, const Tensor &x,
                                        const Tensor &ct, int64_t n_row, int64_t n_col, bool transpose) {
    NoGil no_gil;
    OnDevice on(data);
    Tensor g_data = new_tensor({indices.size(0)}, data.scalar_type(), data.device());
    Tensor g_x = new_tensor({x.size(0)}, data.scalar_type(), data.device());
    bpl_csr_gradients(on.stream, ptr(data), ptr(indices), ptr(indptr), ptr(x), ptr(ct), ptr(g_data), ptr(g_x),
                      static_cast<uint32_t>(n_row), static_cast<uint32_t>(n_col), static_cast<uint32_t>(indices.size(0)),
                      is_double(data) ? 1 : 0, transpose ? 1 : 0);
    check_status();
    return {g_data, g_x};
}

variable_list CsrFn::backward(AutogradContext *ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &data = saved[0], &indices = saved[1], &indptr = saved[2], &x = saved[3];
    const int64_t n_row = ctx->saved_data["r"].toInt(), n_col = ctx->saved_data["c"].toInt();
    const bool t = ctx->saved_data["t"].toBool();
    const Tensor ct = grads[0].contiguous();
    Tensor g_data, g_x;
    if (!plain_cotangent(ct)) {
        std::tie(g_data, g_x) = python_rule(g_csr_backward, {data, indices, indptr, x, ct}, n_row, n_col, t,
                                            ctx->needs_input_grad(0), ctx->needs_input_grad(3));
    } else if (ctx->needs_input_grad(0) && ctx->needs_input_grad(3) && data.size(0) == indices.size(0) && data.size(0) != 1 &&
               !at::GradMode::is_enabled()) {
        std::tie(g_data, g_x) = csr_gradients(data, indices, indptr, x, ct, n_row, n_col, t);
    } else {
        if (ctx->needs_input_grad(0)) {
            if (data.size(0) == 1) {
                const Tensor ones = at::ones({1}, data.options());
                g_data = at::dot(ct, CsrFn::apply(ones, indices, indptr, x, n_row, n_col, t)).reshape({1});
            } else {
                g_data = outer_of(indices, indptr, x, ct, t);
            }
        }
        if (ctx->needs_input_grad(3)) g_x = csr_any(data, indices, indptr, ct, n_row, n_col, !t);
    }
    return {g_data, Tensor(), Tensor(), g_x, Tensor(), Tensor(), Tensor()};
}

struct EventCsrFn : public torch::autograd::Function<EventCsrFn> {
    static Tensor forward(AutogradContext *ctx, const Tensor &data, const Tensor &indices, const Tensor &indptr,
                          const Tensor &events, int64_t n_row, int64_t n_col, bool transpose) {
        ctx->save_for_backward({data, indices, indptr, events});
        ctx->saved_data["r"] = n_row;
        ctx->saved_data["c"] = n_col;
        ctx->saved_data["t"] = transpose;
        return event_csr_product(data, indices, indptr, events, n_row, n_col, transpose);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &data = saved[0], &indices = saved[1], &indptr = saved[2], &events = saved[3];
        const int64_t n_row = ctx->saved_data["r"].toInt(), n_col = ctx->saved_data["c"].toInt();
        const bool t = ctx->saved_data["t"].toBool();
        const Tensor ct = grads[0].contiguous();
        Tensor g_data, g_events;
        if (!plain_cotangent(ct)) {
            std::tie(g_data, g_events) = python_rule(g_event_csr_backward, {data, indices, indptr, events, ct}, n_row, n_col,
                                                     t, ctx->needs_input_grad(0), ctx->needs_input_grad(3));
        } else {
            if (ctx->needs_input_grad(0)) {
                if (data.size(0) == 1) {
                    const Tensor ones = at::ones({1}, data.options());
                    g_data = at::dot(ct, EventCsrFn::apply(ones, indices, indptr, events, n_row, n_col, t)).reshape({1});
                } else {
                    g_data = outer_of(indices, indptr, events.to(data.scalar_type()), ct, t);
                }
            }
            if (ctx->needs_input_grad(3)) g_events = csr_any(data, indices, indptr, ct, n_row, n_col, !t);
        }
        return {g_data, Tensor(), Tensor(), g_events, Tensor(), Tensor(), Tensor()};
    }
};

// What the checks of both CSR operators have in common.  True: the plain case.
bool csr_operands(const Tensor *data, const Tensor *indices, const Tensor *indptr, const Tensor *x, int64_t n_row,
                  int64_t n_in) {
    return data && indices && indptr && x && float_like(*data) && data->dim() == 1 && indices->dim() == 1 &&
           indptr->dim() == 1 && x->dim() == 1 && int32_like(*indices) && int32_like(*indptr) &&
           (data->size(0) == 1 || data->size(0) == indices->size(0)) && indptr->size(0) == n_row + 1 &&
           x->size(0) == n_in && indices->device() == data->device() && indptr->device() == data->device() &&
           x->device() == data->device();
}

// ---- the column-blocked storage (event_ops.ColumnBlockedCSR) ----
PyObject *g_blocked_type = nullptr;

struct Blocked {
    Tensor groups, offsets;               // (held: another thread may set the attributes while the lock is released)
    int64_t n_row = 0, n_col = 0, nse = -1;
    bool fixed = false;
    char opaque[32];
    size_t opaque_len = 0;

    static bool integer(PyObject *o, const char *name, long &v) {
        PyObject *a = PyObject_GetAttrString(o, name);
        if (a == nullptr) return PyErr_Clear(), false;
        const bool ok = PyLong_CheckExact(a);
        if (ok) v = PyLong_AsLong(a);
        Py_DECREF(a);
        return ok;
    }
    static Tensor tensor(PyObject *o, const char *name) {
        PyObject *a = PyObject_GetAttrString(o, name);
        if (a == nullptr) return PyErr_Clear(), Tensor();
        const Tensor *t = tensor_of(a);
        Tensor held = t ? *t : Tensor();
        Py_DECREF(a);
        return held;
    }
    bool read(PyObject *o) {
        if (g_blocked_type == nullptr || Py_TYPE(o) != reinterpret_cast<PyTypeObject *>(g_blocked_type)) return false;
        groups = tensor(o, "groups");
        offsets = tensor(o, "offsets");
        PyObject *shape = PyObject_GetAttrString(o, "shape");
        if (shape == nullptr) return PyErr_Clear(), false;
        const bool shaped = shape_of(shape, n_row, n_col);
        Py_DECREF(shape);
        long width = 0, lanes = 0, scale = 0, entries = -1;
        if (!groups.defined() || !offsets.defined() || !shaped || !integer(o, "block_width", width) || !integer(o, "team_lanes_log2", lanes))
            return false;
        fixed = integer(o, "scale_log2", scale);       // None: float sums
        if (integer(o, "nse", entries)) nse = entries;
        opaque_len = bpl_build_cbcsr_descriptor(static_cast<uint32_t>(n_row), static_cast<uint32_t>(n_col),
                                                static_cast<uint32_t>(width), fixed ? 1 : 0, static_cast<int>(scale),
                                                static_cast<uint32_t>(lanes), opaque, sizeof(opaque));
        return opaque_len != 0;
    }
};

#define NONE_UNLESS(condition) \
    do {                       \
        if (!(condition)) Py_RETURN_NONE; \
    } while (0)

// event_csr_matvec(data, indices, indptr, events, shape, transpose, prepared)
PyObject *py_event_csr_matvec(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    NONE_UNLESS(nargs == 7 && plain_thread());
    int64_t n_row, n_col;
    NONE_UNLESS(shape_of(args[4], n_row, n_col));
    const int t = PyObject_IsTrue(args[5]);
    if (t < 0) return nullptr;
    const Tensor *data = tensor_of(args[0]), *indices = tensor_of(args[1]), *indptr = tensor_of(args[2]),
                 *events = tensor_of(args[3]);
    NONE_UNLESS(csr_operands(data, indices, indptr, events, n_row, t ? n_row : n_col));
    NONE_UNLESS(events->scalar_type() == at::kBool || events->scalar_type() == data->scalar_type());
    const bool grad = wants_grad(*data) || wants_grad(*events);
    if (args[6] != Py_None && t && !is_double(*data) && !grad) {
        Blocked m;
        NONE_UNLESS(m.read(args[6]) && m.n_row == n_row && m.n_col == n_col && m.nse == indices->size(0) &&
                    m.groups.device() == data->device() && m.offsets.device() == data->device());
        Tensor out;
        {
            NoGil no_gil;
            OnDevice on(*data);
            out = new_tensor({n_col}, at::kFloat, data->device());
            Scratch ws(bpl_event_csr_workspace_bytes(static_cast<uint32_t>(n_row), 1), on.stream);
            void *buffers[5] = {ptr(m.groups), ptr(m.offsets), ptr(*events), ptr(out), ws.ptr};
            (events->scalar_type() == at::kBool ? event_cbcsr_matvec_heter_float_bool : event_cbcsr_matvec_heter_float_float)(
                on.stream, buffers, m.opaque, m.opaque_len);
            check_status();
        }
        return THPVariable_Wrap(std::move(out));
    }
    return THPVariable_Wrap(grad ? EventCsrFn::apply(*data, *indices, *indptr, *events, n_row, n_col, t != 0)
                                 : event_csr_product(*data, *indices, *indptr, *events, n_row, n_col, t != 0));
    END_HANDLE_TH_ERRORS
}

// csr_matvec(data, indices, indptr, vector, shape, transpose, prepared)
PyObject *py_csr_matvec(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    NONE_UNLESS(nargs == 7 && plain_thread());
    int64_t n_row, n_col;
    NONE_UNLESS(shape_of(args[4], n_row, n_col));
    const int t = PyObject_IsTrue(args[5]);
    if (t < 0) return nullptr;
    const Tensor *data = tensor_of(args[0]), *indices = tensor_of(args[1]), *indptr = tensor_of(args[2]),
                 *x = tensor_of(args[3]);
    NONE_UNLESS(csr_operands(data, indices, indptr, x, n_row, t ? n_row : n_col));
    NONE_UNLESS(x->scalar_type() == data->scalar_type());
    if (args[6] != Py_None) {
        Blocked m;
        NONE_UNLESS(!is_double(*data) && data->size(0) != 1 && !wants_grad(*x) && m.read(args[6]) && !m.fixed &&
                    m.n_row == n_row && m.n_col == n_col && m.groups.device() == data->device() &&
                    m.offsets.device() == data->device());
        Tensor out;
        {
            NoGil no_gil;
            OnDevice on(*data);
            out = new_tensor({t ? n_col : n_row}, at::kFloat, data->device());
            void *buffers[4] = {ptr(m.groups), ptr(m.offsets), ptr(*x), ptr(out)};
            (t ? cbcsr_matvec_transpose_heter_float : cbcsr_matvec_heter_float)(on.stream, buffers, m.opaque, m.opaque_len);
            check_status();
        }
        return THPVariable_Wrap(std::move(out));
    }
    return THPVariable_Wrap(wants_grad(*data) || wants_grad(*x)
                                ? CsrFn::apply(*data, *indices, *indptr, *x, n_row, n_col, t != 0)
                                : csr_product(*data, *indices, *indptr, *x, n_row, n_col, t != 0));
    END_HANDLE_TH_ERRORS
}

// event_info(events)
PyObject *py_event_info(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    // (Traced as well: neither way leaves a node in the trace, and here torch.jit.trace says so instead of keeping an empty result.)
    NONE_UNLESS(nargs == 1 && untransformed());
    const Tensor *events = tensor_of(args[0]);
    NONE_UNLESS(events && (events->dim() == 1 || events->dim() == 2));
    Target target;
    switch (events->scalar_type()) {
        case at::kBool: target = nonzero_bool; break;
        case at::kInt: target = nonzero_int; break;
        case at::kLong: target = nonzero_long; break;
        case at::kFloat: target = nonzero_float; break;
        case at::kDouble: target = nonzero_double; break;
        default: Py_RETURN_NONE;
    }
    const bool batched = events->dim() == 2;
    const int64_t batch = batched ? events->size(0) : 1, size = events->size(batched ? 1 : 0);
    Tensor ids, num;
    {
        NoGil no_gil;
        OnDevice on(*events);
        ids = new_tensor(events->sizes(), at::kInt, events->device());
        num = batched ? new_tensor({batch}, at::kInt, events->device()) : new_tensor({}, at::kInt, events->device());
        const bpl::DoubleSizeDescriptor d{static_cast<unsigned>(size), static_cast<unsigned>(batch)};
        Scratch ws(bpl_nonzero_workspace_bytes(static_cast<uint32_t>(batch)), on.stream);
        void *buffers[4] = {ptr(*events), ptr(ids), ptr(num), ws.ptr};
        target(on.stream, buffers, reinterpret_cast<const char *>(&d), sizeof(d));
        check_status();
    }
    PyObject *r = PyTuple_New(2);
    if (r == nullptr) return nullptr;
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(ids)));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(num)));
    return r;
    END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------------------
// just-in-time connectivity
// ---------------------------------------------------------------------------------------------------------
struct JitArgs {
    int64_t kind;               // 0 homogeneous, 1 uniform, 2 normal
    double weight;              // homogeneous: the factor of the result
    double w1, w2, log_p;
    int64_t n_out, n_in, seed;
    bool rows;                  // one stream per output (outdim_parallel) or per input

    // the transposed product walks the same streams from the other side
    JitArgs transposed() const {
        JitArgs t = *this;
        std::swap(t.n_out, t.n_in);
        t.rows = !rows;
        return t;
    }
};

// The descriptor's real fields are float32-rounded, here as in bpl_build_jitconn_prob_*_descriptor.
Tensor jit_product(const Tensor &x, const JitArgs &a, const bool events) {
    NoGil no_gil;
    OnDevice on(x);
    const bool b = x.scalar_type() == at::kBool;
    Tensor out = new_tensor({a.n_out}, b ? at::kFloat : x.scalar_type(), x.device());
    bpl_jit_matvec(on.stream, ptr(x), ptr(out), b ? 0 : is_double(x) ? 2 : 1, events, static_cast<int>(a.kind), a.rows,
                   static_cast<uint32_t>(a.n_out), static_cast<uint32_t>(a.n_in), static_cast<uint32_t>(a.seed),
                   static_cast<float>(a.log_p), static_cast<float>(a.w1), static_cast<float>(a.w2), a.weight);
    check_status();
    // homogeneous event sums over columns are counts: scaled once, like the counts of rows
    if (events && !a.rows && a.kind == 0) out.mul_(a.weight);
    return out;
}

PyObject *g_jit_backward = nullptr;     // jitconn_ops.backward_rule

struct JitFn : public torch::autograd::Function<JitFn> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x, const JitArgs &a, bool events) {
        ctx->saved_data["i"] = std::vector<int64_t>{a.kind, a.n_out, a.n_in, a.seed, a.rows ? 1 : 0};
        ctx->saved_data["f"] = std::vector<double>{a.weight, a.w1, a.w2, a.log_p};
        return jit_product(x, a, events);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const auto i = ctx->saved_data["i"].toIntVector();
        const auto f = ctx->saved_data["f"].toDoubleVector();
        const JitArgs a{i[0], f[0], f[1], f[2], f[3], i[1], i[2], i[3], i[4] != 0};
        const JitArgs t = a.transposed();
        const Tensor ct = grads[0].contiguous();
        Tensor g;
        if (plain_cotangent(ct)) g = at::GradMode::is_enabled() ? JitFn::apply(ct, t, false) : jit_product(ct, t, false);
        else g = python_jit_rule(ct, t);
        return {g, Tensor(), Tensor()};
    }
    // backward_rule(ct, kind, weight, w1, w2, log_p, n_out, n_in, seed, rows)
    static Tensor python_jit_rule(const Tensor &ct, const JitArgs &t) {
        pybind11::gil_scoped_acquire gil;
        const auto c = pybind11::reinterpret_steal<pybind11::object>(THPVariable_Wrap(ct));
        const auto r = pybind11::reinterpret_borrow<pybind11::object>(g_jit_backward)(
            c, t.kind, t.weight, t.w1, t.w2, t.log_p, t.n_out, t.n_in, t.seed, t.rows);
        return THPVariable_Unpack(r.ptr());
    }
};

// jit_matvec(vector, events, kind, weight, w1, w2, log_p, shape, seed, transpose, outdim_parallel)
//   events: whether `vector` is an event vector
PyObject *py_jit_matvec(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    NONE_UNLESS(nargs == 11 && plain_thread());
    const Tensor *x = tensor_of(args[0]);
    const bool events = args[1] == Py_True;
    JitArgs a;
    int64_t s0, s1;
    double kind;
    NONE_UNLESS(x && x->dim() == 1 && (float_like(*x) || (events && x->scalar_type() == at::kBool)));
    NONE_UNLESS(number_of(args[2], kind) && number_of(args[3], a.weight) && number_of(args[4], a.w1) &&
                number_of(args[5], a.w2) && number_of(args[6], a.log_p) && shape_of(args[7], s0, s1) &&
                PyLong_CheckExact(args[8]));
    const int t = PyObject_IsTrue(args[9]), rows = PyObject_IsTrue(args[10]);
    if (t < 0 || rows < 0) return nullptr;
    a.kind = static_cast<int64_t>(kind);
    a.seed = static_cast<int64_t>(PyLong_AsUnsignedLongMask(args[8]) & 0xffffffffull);
    a.n_out = t ? s1 : s0;
    a.n_in = t ? s0 : s1;
    a.rows = rows != 0;
    NONE_UNLESS(x->size(0) == a.n_in);
    return THPVariable_Wrap(wants_grad(*x) ? JitFn::apply(*x, a, events) : jit_product(*x, a, events));
    END_HANDLE_TH_ERRORS
}

// jit_matmat(matrix, kind, w1, w2, log_p, shape, seed): version v1, lists in a workspace
PyObject *py_jit_matmat(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    static const Target targets[2][2] = {   // [kind - 1][double]
        {gpu_matmat_prob_prob_uniform_float_v1_ws, gpu_matmat_prob_prob_uniform_double_v1_ws},
        {gpu_matmat_prob_prob_normal_float_v1_ws, gpu_matmat_prob_prob_normal_double_v1_ws}};
    NONE_UNLESS(nargs == 7 && plain_thread());
    const Tensor *x = tensor_of(args[0]);
    double kind, w1, w2, log_p;
    int64_t k, n;
    NONE_UNLESS(x && x->dim() == 2 && float_like(*x) && !wants_grad(*x) && number_of(args[1], kind) &&
                number_of(args[2], w1) && number_of(args[3], w2) && number_of(args[4], log_p) && shape_of(args[5], k, n) &&
                x->size(1) == k && x->size(0) <= 0xffffffffll && PyLong_CheckExact(args[6]));
    const uint32_t seed = static_cast<uint32_t>(PyLong_AsUnsignedLongMask(args[6]));
    Tensor out;
    {
        NoGil no_gil;
        OnDevice on(*x);
        out = new_tensor({x->size(0), n}, x->scalar_type(), x->device());
        char opaque[64];
        const size_t len = bpl_build_matmat_jit_prob_descriptor1(
            static_cast<uint32_t>(x->size(0)), static_cast<uint32_t>(k), static_cast<uint32_t>(n), seed, static_cast<float>(log_p),
            static_cast<float>(w1), static_cast<float>(w2), opaque, sizeof(opaque));
        Scratch ws(bpl_workspace_bytes(is_double(*x) ? "gpu_matmat_prob_prob_normal_double_v1_ws"
                                                     : "gpu_matmat_prob_prob_normal_float_v1_ws", opaque, len), on.stream);
        void *buffers[3] = {ptr(*x), ptr(out), ws.ptr};
        targets[kind > 1.5][is_double(*x)](on.stream, buffers, opaque, len);
        check_status();
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------------------
// the caller's neuron step
// ---------------------------------------------------------------------------------------------------------
bool float_attr(PyObject *o, const char *name, float &v) {
    PyObject *a = PyObject_GetAttrString(o, name);
    if (a == nullptr) return PyErr_Clear(), false;
    const double d = PyFloat_AsDouble(a);
    Py_DECREF(a);
    if (d == -1.0 && PyErr_Occurred()) return PyErr_Clear(), false;
    v = static_cast<float>(d);
    return true;
}

// up to four floats of a sequence attribute; their number, or -1
int floats_attr(PyObject *o, const char *name, float (&v)[4]) {
    PyObject *a = PyObject_GetAttrString(o, name);
    if (a == nullptr) return PyErr_Clear(), -1;
    int n = -1;
    Py_buffer view;
    if (PyObject_CheckBuffer(a)) {
        if (PyObject_GetBuffer(a, &view, PyBUF_ND | PyBUF_FORMAT) == 0) {
            if (view.ndim == 1 && view.itemsize == 4 && view.format && std::strcmp(view.format, "f") == 0 && view.shape[0] >= 1 &&
                view.shape[0] <= 4) {
                n = static_cast<int>(view.shape[0]);
                std::memcpy(v, view.buf, 4 * static_cast<size_t>(n));
            }
            PyBuffer_Release(&view);
        } else {
            PyErr_Clear();
        }
    } else if (PyList_CheckExact(a) || PyTuple_CheckExact(a)) {
        const Py_ssize_t len = PySequence_Fast_GET_SIZE(a);
        if (len >= 1 && len <= 4) {
            n = static_cast<int>(len);
            for (int i = 0; i < n; ++i) {
                const double d = PyFloat_AsDouble(PySequence_Fast_GET_ITEM(a, i));
                if (d == -1.0 && PyErr_Occurred()) {
                    PyErr_Clear();
                    n = -1;
                    break;
                }
                v[i] = static_cast<float>(d);
            }
        }
    }
    Py_DECREF(a);
    return n;
}

bool step_vector(const Tensor *t, const Tensor &v, int64_t k) {
    if (!t || t->scalar_type() != at::kFloat || t->device() != v.device()) return false;
    const int64_t n = v.size(0);
    return k == 0 ? (t->dim() == 1 && t->size(0) == n)
                  : ((t->dim() == 2 && t->size(0) == k && t->size(1) == n) || (k == 1 && t->dim() == 1 && t->size(0) == n));
}

// lif_exp_step(y, g, V, t_last, params, t, spikes | None, spike_list | None)
PyObject *py_lif_exp_step(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    NONE_UNLESS(nargs == 8 && plain_thread());
    const Tensor *y = tensor_of(args[0]), *g = tensor_of(args[1]), *V = tensor_of(args[2]), *t_last = tensor_of(args[3]);
    NONE_UNLESS(V && V->dim() == 1 && V->scalar_type() == at::kFloat);
    float decay[4], e_rev[4], ext, v_rest, v_th, v_reset, r, lif, tau_ref;
    double t;
    const int k = floats_attr(args[4], "syn_decay", decay);
    NONE_UNLESS(k >= 1 && floats_attr(args[4], "E_rev", e_rev) == k && number_of(args[5], t));
    NONE_UNLESS(float_attr(args[4], "ext_input", ext) && float_attr(args[4], "V_rest", v_rest) &&
                float_attr(args[4], "V_th", v_th) && float_attr(args[4], "V_reset", v_reset) && float_attr(args[4], "R", r) &&
                float_attr(args[4], "lif_decay", lif) && float_attr(args[4], "tau_ref", tau_ref));
    NONE_UNLESS(step_vector(y, *V, k) && step_vector(g, *V, k) && step_vector(t_last, *V, 0));
    const int64_t n = V->size(0);
    NONE_UNLESS(n <= 0xffffffffll);
    const size_t list_bytes = bpl_event_csr_workspace_bytes(static_cast<uint32_t>(n), 1);
    OnDevice on(*V);
    Tensor spikes, list;
    if (args[6] != Py_None) {
        const Tensor *s = tensor_of(args[6]);
        NONE_UNLESS(step_vector(s, *V, 0));
        spikes = *s;
    } else {
        spikes = new_tensor({n}, at::kFloat, V->device());
    }
    if (args[7] != Py_None) {
        const Tensor *s = tensor_of(args[7]);
        NONE_UNLESS(s && s->nbytes() >= list_bytes && s->device() == V->device());
        list = *s;
    } else {
        list = new_tensor({static_cast<int64_t>(list_bytes)}, at::kByte, V->device());
    }
    char opaque[128];
    const size_t len = bpl_build_lif_exp_descriptor(static_cast<uint32_t>(n), static_cast<uint32_t>(k), static_cast<float>(t),
                                                    decay, e_rev, ext, v_rest, v_th, v_reset, r, lif, tau_ref, opaque,
                                                    sizeof(opaque));
    NONE_UNLESS(len != 0);
    {
        NoGil no_gil;
        void *buffers[6] = {ptr(*y), ptr(*g), ptr(*V), ptr(*t_last), ptr(spikes), ptr(list)};
        lif_exp_step_float(on.stream, buffers, opaque, len);
        check_status();
    }
    PyObject *res = PyTuple_New(2);
    if (res == nullptr) return nullptr;
    PyTuple_SET_ITEM(res, 0, THPVariable_Wrap(std::move(spikes)));
    PyTuple_SET_ITEM(res, 1, THPVariable_Wrap(std::move(list)));
    return res;
    END_HANDLE_TH_ERRORS
}

// list_matvec(data, indices, indptr, spike_list, y, shape, prepared) -> True when done
PyObject *py_list_matvec(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    NONE_UNLESS(nargs == 7 && plain_thread());
    int64_t n_row, n_col;
    const Tensor *list = tensor_of(args[3]), *y = tensor_of(args[4]);
    NONE_UNLESS(shape_of(args[5], n_row, n_col) && list && y && y->scalar_type() == at::kFloat && y->numel() == n_col &&
                list->nbytes() >= bpl_event_csr_workspace_bytes(static_cast<uint32_t>(n_row), 1) &&
                list->device() == y->device());
    if (args[6] != Py_None) {
        Blocked m;
        NONE_UNLESS(m.read(args[6]) && m.n_row == n_row && m.n_col == n_col && m.groups.device() == y->device());
        NoGil no_gil;
        OnDevice on(*y);
        void *buffers[4] = {ptr(m.groups), ptr(m.offsets), ptr(*list), ptr(*y)};
        event_cbcsr_matvec_list_heter_float(on.stream, buffers, m.opaque, m.opaque_len);
        check_status();
    } else {
        const Tensor *data = tensor_of(args[0]), *indices = tensor_of(args[1]), *indptr = tensor_of(args[2]);
        NONE_UNLESS(data && indices && indptr && data->scalar_type() == at::kFloat && int32_like(*indices) &&
                    int32_like(*indptr) && data->numel() == indices->numel() && indptr->numel() == n_row + 1 &&
                    n_row <= 1024 * 4096 && data->device() == y->device() && indices->device() == y->device() &&
                    indptr->device() == y->device());
        char opaque[16];
        const size_t len = bpl_build_triple_size_descriptor(static_cast<uint32_t>(n_row), static_cast<uint32_t>(n_col),
                                                            static_cast<uint32_t>((n_row + 4095) / 4096), opaque, sizeof(opaque));
        NoGil no_gil;
        OnDevice on(*y);
        void *buffers[5] = {ptr(*data), ptr(*indices), ptr(*indptr), ptr(*list), ptr(*y)};
        event_csr_matvec_list_heter_float(on.stream, buffers, opaque, len);
        check_status();
    }
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// csr_outer(row_vector, col_vector, indices, indptr): the Python rule's forward, on checked tensors
PyObject *py_csr_outer(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    NONE_UNLESS(nargs == 4);
    for (int i = 0; i < 4; ++i) NONE_UNLESS(THPVariable_Check(args[i]));
    const Tensor row = THPVariable_Unpack(args[0]).contiguous(), col = THPVariable_Unpack(args[1]).contiguous();
    const Tensor &indices = THPVariable_Unpack(args[2]), &indptr = THPVariable_Unpack(args[3]);
    Tensor out = csr_outer(row, col, indices, indptr);
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// register(blocked_type, event_csr_backward, csr_backward, csr_outer_backward, jit_backward)
PyObject *py_register(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 5) {
        PyErr_SetString(PyExc_TypeError, "register takes 5 arguments");
        return nullptr;
    }
    PyObject **slots[5] = {&g_blocked_type, &g_event_csr_backward, &g_csr_backward, &g_csr_outer, &g_jit_backward};
    for (int i = 0; i < 5; ++i) {
        Py_INCREF(args[i]);
        Py_XSETREF(*slots[i], args[i]);
    }
    Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(event_csr_matvec), FAST(csr_matvec), FAST(event_info), FAST(jit_matvec), FAST(jit_matmat),
                         FAST(lif_exp_step), FAST(list_matvec), FAST(csr_outer), FAST(register), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Native host path of the operators.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
