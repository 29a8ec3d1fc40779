// The Python binding's hot calls on torch tensors, and the cutespmm torch operators, as native code.
//
// A product on a small matrix is 5-10 us of GPU time; argument checks, the output's allocation, the stream lookup and a
// ctypes call in Python took 10 us of host time in front of it, and an operator registered from Python 50-60 us per call
// (forward, backward and the dispatch of both).  Here a call is one CPython fast call, an ATen allocation and the C ABI
// (2-3 us), and the operators' forward and backward run without the interpreter.
//
// The plans themselves stay with the Python objects (Plan, SparseOperator); this file holds handles only.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>
#include <ATen/ops/empty.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/cuda/CUDAStream.h>

#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <unordered_map>

#include "../../include/cutespmm.h"

namespace {

using at::Tensor;

PyObject *g_error_class = nullptr;  // CuteSpmmError(status, message)

// The GIL is held.
void set_status_error(int status)
{
    const char *msg = cutespmm_last_error();
    if (!msg || !*msg) msg = cutespmm_status_string(status);
    PyObject *e = g_error_class ? PyObject_CallFunction(g_error_class, "is", status, msg) : nullptr;
    if (e) {
        PyErr_SetObject(reinterpret_cast<PyObject *>(Py_TYPE(e)), e);
        Py_DECREF(e);
    } else if (!PyErr_Occurred()) {
        PyErr_SetString(PyExc_RuntimeError, msg);
    }
}

void check_status(int status)  // with or without the GIL
{
    if (status == CUTESPMM_OK) return;
    PyGILState_STATE g = PyGILState_Ensure();
    set_status_error(status);
    python_error err;
    err.persist();
    PyGILState_Release(g);
    throw err;
}

bool dense2d(const Tensor &t) { return t.is_cuda() && t.scalar_type() == at::kFloat && t.dim() == 2 && t.stride(1) == 1; }
uint64_t ld(const Tensor &t, int64_t rows) { return rows > 1 ? (uint64_t)t.stride(0) : (uint64_t)std::max<int64_t>(t.size(1), 1); }
void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
const float *in(const Tensor &t) { return static_cast<const float *>(t.const_data_ptr()); }
float *out(const Tensor &t) { return static_cast<float *>(t.mutable_data_ptr()); }
Tensor new_dense(int64_t rows, int64_t cols, const Tensor &like) { return at::empty({rows, cols}, like.options().requires_grad(false)); }

Tensor run_spmm(const cutespmm_plan_t *plan, int64_t M, int64_t K, const Tensor &B, Tensor C, void *stream)
{
    TORCH_CHECK_VALUE(dense2d(B), "B must be a 2-D CUDA fp32 tensor with unit column stride");
    TORCH_CHECK_VALUE(B.size(0) == K, "B has ", B.size(0), " rows, A has ", K, " columns");
    const int64_t N = B.size(1);
    if (!C.defined()) C = new_dense(M, N, B);
    else TORCH_CHECK_VALUE(dense2d(C) && C.size(0) == M && C.size(1) == N, "C must be an M x N CUDA fp32 tensor with unit column stride");
    check_status(cutespmm_spmm(plan, in(B), ld(B, K), out(C), ld(C, M), (uint32_t)N, stream ? stream : stream_of(B)));
    return C;
}

Tensor run_sddmm(const cutespmm_plan_t *plan, int64_t M, int64_t K, int64_t nnz, const Tensor &X, const Tensor &Y, Tensor o, bool scale, void *stream)
{
    TORCH_CHECK_VALUE(dense2d(X) && X.size(0) == M, "X must be a ", M, " x N CUDA fp32 tensor with unit column stride");
    TORCH_CHECK_VALUE(dense2d(Y) && Y.size(0) == K, "Y must be a ", K, " x N CUDA fp32 tensor with unit column stride");
    TORCH_CHECK_VALUE(X.size(1) == Y.size(1), "X and Y must have the same number of columns");
    if (!o.defined()) o = at::empty({nnz}, X.options().requires_grad(false));
    else
        TORCH_CHECK_VALUE(o.is_cuda() && o.scalar_type() == at::kFloat && o.numel() == nnz && o.is_contiguous(),
                          "out must be a contiguous CUDA fp32 tensor with one element per nonzero");
    check_status(cutespmm_sddmm(plan, in(X), ld(X, M), in(Y), ld(Y, K), (uint32_t)X.size(1), scale ? 1 : 0, out(o), stream ? stream : stream_of(X)));
    return o;
}

void run_set_values(cutespmm_plan_t *plan, int64_t nnz, const Tensor &vals, const Tensor &order, void *stream)
{
    TORCH_CHECK_VALUE(vals.is_cuda() && vals.scalar_type() == at::kFloat && vals.numel() == nnz && vals.is_contiguous(),
                      "vals must be a contiguous CUDA fp32 tensor with one element per nonzero");
    void *s = stream ? stream : stream_of(vals);
    if (order.defined())
        check_status(cutespmm_plan_set_values_gathered(plan, in(vals), static_cast<const uint32_t *>(order.const_data_ptr()), s));
    else check_status(cutespmm_plan_set_values(plan, in(vals), s));
}

// ---- operators -------------------------------------------------------------------------------------------------------

// What an operator needs to know of a registered SparseOperator.
struct OpState {
    cutespmm_plan_t *plan = nullptr, *transposed = nullptr;
    int64_t M = 0, K = 0, nnz = 0;
    Tensor order;              // storage position in A of every stored position of A^T (int32)
    PyObject *build = nullptr;  // build(need_order): makes the plan of A^T (and `order`) and calls set_transposed
    ~OpState()
    {
        if (build && Py_IsInitialized()) {
            PyGILState_STATE g = PyGILState_Ensure();
            Py_DECREF(build);
            PyGILState_Release(g);
        }
    }
};
std::mutex g_ops_mutex;
// never destroyed: the interpreter may be gone when static destructors run
std::unordered_map<int64_t, std::shared_ptr<OpState>> &ops()
{
    static auto *m = new std::unordered_map<int64_t, std::shared_ptr<OpState>>();
    return *m;
}

std::shared_ptr<OpState> get_op(int64_t id)
{
    std::lock_guard<std::mutex> lock(g_ops_mutex);
    auto it = ops().find(id);
    TORCH_CHECK(it != ops().end(), "cutespmm: no plan registered under id ", id);
    return it->second;
}

// The plan of A^T (and the order), built through the Python object on first use; two threads that ask at once get the same one
// (the object's lock).
struct Transposed {
    cutespmm_plan_t *plan;
    Tensor order;
};
Transposed need_transposed(OpState &op, bool with_order)
{
    {
        std::lock_guard<std::mutex> lock(g_ops_mutex);
        if (op.transposed && (!with_order || op.order.defined())) return {op.transposed, op.order};
    }
    PyGILState_STATE g = PyGILState_Ensure();
    PyObject *r = PyObject_CallFunction(op.build, "i", with_order ? 1 : 0);
    if (!r) {
        python_error err;
        err.persist();
        PyGILState_Release(g);
        throw err;
    }
    Py_DECREF(r);
    PyGILState_Release(g);
    std::lock_guard<std::mutex> lock(g_ops_mutex);
    TORCH_CHECK(op.transposed && (!with_order || op.order.defined()), "cutespmm: the plan of A^T could not be built");
    return {op.transposed, op.order};
}

Tensor unit_stride(const Tensor &t) { return t.dim() > 0 && t.stride(-1) == 1 ? t : t.contiguous(); }

Tensor op_spmm(int64_t id, const Tensor &B)
{
    auto op = get_op(id);
    return run_spmm(op->plan, op->M, op->K, unit_stride(B), Tensor(), nullptr);
}
Tensor op_spmm_transposed(int64_t id, const Tensor &G)
{
    auto op = get_op(id);
    return run_spmm(need_transposed(*op, false).plan, op->K, op->M, unit_stride(G), Tensor(), nullptr);
}
Tensor op_spmm_weighted(int64_t id, const Tensor &w, const Tensor &B)
{
    auto op = get_op(id);
    run_set_values(op->plan, op->nnz, w.contiguous(), Tensor(), nullptr);
    return run_spmm(op->plan, op->M, op->K, unit_stride(B), Tensor(), nullptr);
}
Tensor op_spmm_weighted_transposed(int64_t id, const Tensor &w, const Tensor &G)
{
    auto op = get_op(id);
    const Transposed t = need_transposed(*op, true);
    run_set_values(t.plan, op->nnz, w.contiguous(), t.order, nullptr);
    return run_spmm(t.plan, op->K, op->M, unit_stride(G), Tensor(), nullptr);
}
Tensor op_sddmm(int64_t id, const Tensor &X, const Tensor &Y, bool scale)
{
    auto op = get_op(id);
    return run_sddmm(op->plan, op->M, op->K, op->nnz, unit_stride(X), unit_stride(Y), Tensor(), scale, nullptr);
}

template <class Sig> c10::TypedOperatorHandle<Sig> handle(const char *name)
{
    return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<Sig>();
}
using Unary = Tensor(int64_t, const Tensor &);
using Weighted = Tensor(int64_t, const Tensor &, const Tensor &);
Tensor call_spmm(int64_t id, const Tensor &B)
{
    static auto h = handle<Unary>("cutespmm::spmm");
    return h.call(id, B);
}
Tensor call_spmm_transposed(int64_t id, const Tensor &G)
{
    static auto h = handle<Unary>("cutespmm::spmm_transposed");
    return h.call(id, G);
}
Tensor call_spmm_weighted(int64_t id, const Tensor &w, const Tensor &B)
{
    static auto h = handle<Weighted>("cutespmm::spmm_weighted");
    return h.call(id, w, B);
}
Tensor call_spmm_weighted_transposed(int64_t id, const Tensor &w, const Tensor &G)
{
    static auto h = handle<Weighted>("cutespmm::spmm_weighted_transposed");
    return h.call(id, w, G);
}
Tensor call_sddmm(int64_t id, const Tensor &X, const Tensor &Y, bool scale)
{
    static auto h = handle<Tensor(int64_t, const Tensor &, const Tensor &, bool)>("cutespmm::sddmm");
    return h.call(id, X, Y, scale);
}

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// d(A B)/dB = A^T dC, and the other way round
template <bool TRANSPOSED> struct SpmmGrad : torch::autograd::Function<SpmmGrad<TRANSPOSED>> {
    static Tensor forward(AutogradContext *ctx, int64_t id, const Tensor &B)
    {
        at::AutoDispatchBelowADInplaceOrView guard;
        ctx->saved_data["id"] = id;
        return TRANSPOSED ? call_spmm_transposed(id, B) : call_spmm(id, B);
    }
    static variable_list backward(AutogradContext *ctx, const variable_list &g)
    {
        const int64_t id = ctx->saved_data["id"].toInt();
        return {Tensor(), TRANSPOSED ? call_spmm(id, g[0]) : call_spmm_transposed(id, g[0])};
    }
};
// C = A_w B: dw = SDDMM(dC, B), dB = A_w^T dC
struct WeightedGrad : torch::autograd::Function<WeightedGrad> {
    static Tensor forward(AutogradContext *ctx, int64_t id, const Tensor &w, const Tensor &B)
    {
        at::AutoDispatchBelowADInplaceOrView guard;
        ctx->saved_data["id"] = id;
        ctx->save_for_backward({w, B});
        return call_spmm_weighted(id, w, B);
    }
    static variable_list backward(AutogradContext *ctx, const variable_list &g)
    {
        const int64_t id = ctx->saved_data["id"].toInt();
        const variable_list saved = ctx->get_saved_variables();
        // the two have no gradients of their own: unless a graph of this pass is asked for (and has to name them), go past the
        // kernels that say so
        std::optional<at::AutoDispatchBelowADInplaceOrView> guard;
        if (!c10::GradMode::is_enabled()) guard.emplace();
        return {Tensor(), ctx->needs_input_grad(0) ? call_sddmm(id, g[0], saved[1], false) : Tensor(),
                ctx->needs_input_grad(1) ? call_spmm_weighted_transposed(id, saved[0], g[0]) : Tensor()};
    }
};

TORCH_LIBRARY(cutespmm, m)
{
    m.def("spmm(int plan_id, Tensor B) -> Tensor");
    m.def("spmm_transposed(int plan_id, Tensor G) -> Tensor");
    m.def("spmm_weighted(int plan_id, Tensor w, Tensor B) -> Tensor");
    m.def("spmm_weighted_transposed(int plan_id, Tensor w, Tensor G) -> Tensor");
    m.def("sddmm(int plan_id, Tensor X, Tensor Y, bool scale_by_values) -> Tensor");
}
TORCH_LIBRARY_IMPL(cutespmm, CompositeExplicitAutograd, m)
{
    m.impl("spmm", op_spmm);
    m.impl("spmm_transposed", op_spmm_transposed);
    m.impl("spmm_weighted", op_spmm_weighted);
    m.impl("spmm_weighted_transposed", op_spmm_weighted_transposed);
    m.impl("sddmm", op_sddmm);
}
TORCH_LIBRARY_IMPL(cutespmm, Autograd, m)
{
    m.impl("spmm", [](int64_t id, const Tensor &B) { return SpmmGrad<false>::apply(id, B); });
    m.impl("spmm_transposed", [](int64_t id, const Tensor &G) { return SpmmGrad<true>::apply(id, G); });
    m.impl("spmm_weighted", [](int64_t id, const Tensor &w, const Tensor &B) { return WeightedGrad::apply(id, w, B); });
    // without one of these a backward pass through them would go on with zeros and a warning
    m.impl("spmm_weighted_transposed", torch::autograd::autogradNotImplementedFallback());
    m.impl("sddmm", torch::autograd::autogradNotImplementedFallback());
}

// ---- the Python module -----------------------------------------------------------------------------------------------

const Tensor &tensor(PyObject *o, const char *what)
{
    TORCH_CHECK_TYPE(THPVariable_Check(o), what, " must be a torch tensor");
    return THPVariable_Unpack(o);
}
Tensor tensor_or_none(PyObject *o, const char *what) { return o == Py_None ? Tensor() : tensor(o, what); }
int64_t integer(PyObject *o)
{
    const int64_t v = o == Py_None ? 0 : (int64_t)PyLong_AsUnsignedLongLong(o);
    if (PyErr_Occurred()) throw python_error();
    return v;
}
void *pointer(PyObject *o) { return reinterpret_cast<void *>(integer(o)); }
void want_args(Py_ssize_t n, Py_ssize_t want) { TORCH_CHECK_TYPE(n == want, "expected ", want, " arguments, got ", n); }
// a stream the caller named: its handle (the default stream's is 0, which the calls above read as "the current one")
void *named_stream(PyObject *o)
{
    if (o == Py_None) return nullptr;
    void *s = pointer(o);
    return s ? s : reinterpret_cast<void *>(0x1);  // cudaStreamLegacy
}

// fn without the interpreter lock, as ctypes makes its calls: a launch that waits for room in its stream's queue must not hold
// up other threads, and threads that drive a stream each run side by side.  The calls below take their arguments out of
// Python first and hold references of their own to the tensors.
template <class Fn> auto without_gil(Fn &&fn)
{
    struct Released {
        PyThreadState *state = PyEval_SaveThread();
        ~Released() { PyEval_RestoreThread(state); }
    } released;
    return fn();
}

PyObject *py_spmm(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 6);  // plan, M, K, B, C or None, stream or None
    auto *plan = static_cast<cutespmm_plan_t *>(pointer(a[0]));
    const int64_t M = integer(a[1]), K = integer(a[2]);
    const Tensor B = tensor(a[3], "B"), C = tensor_or_none(a[4], "C");
    void *s = named_stream(a[5]);
    return THPVariable_Wrap(without_gil([&] { return run_spmm(plan, M, K, B, C, s); }));
    END_HANDLE_TH_ERRORS
}
PyObject *py_sddmm(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 9);  // plan, M, K, nnz, X, Y, out or None, scale, stream or None
    auto *plan = static_cast<cutespmm_plan_t *>(pointer(a[0]));
    const int64_t M = integer(a[1]), K = integer(a[2]), nnz = integer(a[3]);
    const Tensor X = tensor(a[4], "X"), Y = tensor(a[5], "Y"), o = tensor_or_none(a[6], "out");
    const bool scale = PyObject_IsTrue(a[7]) == 1;
    void *s = named_stream(a[8]);
    return THPVariable_Wrap(without_gil([&] { return run_sddmm(plan, M, K, nnz, X, Y, o, scale, s); }));
    END_HANDLE_TH_ERRORS
}
PyObject *py_set_values(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 4);  // plan, nnz, vals, stream or None
    auto *plan = static_cast<cutespmm_plan_t *>(pointer(a[0]));
    const int64_t nnz = integer(a[1]);
    const Tensor vals = tensor(a[2], "vals");
    void *s = named_stream(a[3]);
    without_gil([&] { run_set_values(plan, nnz, vals, Tensor(), s); });
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}
PyObject *py_noalloc(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 8);  // M, K, row_ptr, cols, vals, B, C, stream or None
    const int64_t M = integer(a[0]), K = integer(a[1]);
    const Tensor rp = tensor(a[2], "row_ptr"), cols = tensor(a[3], "cols"), vals = tensor(a[4], "vals"), B = tensor(a[5], "B"), C = tensor(a[6], "C");
    auto is = [](const Tensor &t, at::ScalarType dt) { return t.is_cuda() && t.scalar_type() == dt; };
    TORCH_CHECK_VALUE(is(rp, at::kInt) && is(cols, at::kInt) && is(vals, at::kFloat) && is(B, at::kFloat) && is(C, at::kFloat),
                      "all operands must be CUDA tensors: row_ptr/cols int32, vals/B/C float32");
    TORCH_CHECK_VALUE(B.dim() == 2 && C.dim() == 2, "B and C must be 2-D");
    TORCH_CHECK_VALUE(rp.is_contiguous() && cols.is_contiguous() && vals.is_contiguous() && B.stride(1) == 1 && C.stride(1) == 1,
                      "CSR arrays must be contiguous; B and C need unit column stride");
    const int64_t N = B.size(1);
    // the call itself cannot see the sizes of the buffers behind the pointers: check them here, as run_spmm does
    TORCH_CHECK_VALUE(rp.numel() == M + 1 && cols.numel() == vals.numel(), "row_ptr must have M+1 entries; cols and vals the same length");
    TORCH_CHECK_VALUE(B.size(0) == K, "B has ", B.size(0), " rows, A has ", K, " columns");
    TORCH_CHECK_VALUE(C.size(0) == M && C.size(1) == N, "C must be ", M, " x ", N, ", got ", C.sizes());
    TORCH_CHECK_VALUE(rp.device() == B.device() && cols.device() == B.device() && vals.device() == B.device() && C.device() == B.device(),
                      "all operands must live on one device");
    void *s = named_stream(a[7]);
    without_gil([&] {
        check_status(cutespmm_spmm_csr_noalloc((uint32_t)M, (uint32_t)K, (uint32_t)cols.numel(), static_cast<const uint32_t *>(rp.const_data_ptr()),
                                               static_cast<const uint32_t *>(cols.const_data_ptr()), in(vals), in(B), ld(B, K), out(C), ld(C, M),
                                               (uint32_t)N, s ? s : stream_of(B)));
    });
    Py_INCREF(a[6]);
    return a[6];
    END_HANDLE_TH_ERRORS
}

// Operators called without the packet lookup of torch.ops.
PyObject *py_op_spmm(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 2);
    const int64_t id = integer(a[0]);
    const Tensor B = tensor(a[1], "B");
    return THPVariable_Wrap(without_gil([&] { return call_spmm(id, B); }));
    END_HANDLE_TH_ERRORS
}
PyObject *py_op_weighted(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 3);
    const int64_t id = integer(a[0]);
    const Tensor w = tensor(a[1], "w"), B = tensor(a[2], "B");
    return THPVariable_Wrap(without_gil([&] { return call_spmm_weighted(id, w, B); }));
    END_HANDLE_TH_ERRORS
}
PyObject *py_op_sddmm(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 4);
    const int64_t id = integer(a[0]);
    const Tensor X = tensor(a[1], "X"), Y = tensor(a[2], "Y");
    const bool scale = PyObject_IsTrue(a[3]) == 1;
    return THPVariable_Wrap(without_gil([&] { return call_sddmm(id, X, Y, scale); }));
    END_HANDLE_TH_ERRORS
}

PyObject *py_register(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 6);  // id, plan, M, K, nnz, build
    auto op = std::make_shared<OpState>();
    op->plan = static_cast<cutespmm_plan_t *>(pointer(a[1]));
    op->M = integer(a[2]); op->K = integer(a[3]); op->nnz = integer(a[4]);
    Py_INCREF(a[5]);
    op->build = a[5];
    std::lock_guard<std::mutex> lock(g_ops_mutex);
    ops()[integer(a[0])] = op;
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}
PyObject *py_unregister(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 1);
    std::shared_ptr<OpState> gone;  // dropped outside the lock
    {
        std::lock_guard<std::mutex> lock(g_ops_mutex);
        auto it = ops().find(integer(a[0]));
        if (it != ops().end()) {
            gone = it->second;
            ops().erase(it);
        }
    }
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}
PyObject *py_set_transposed(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    want_args(n, 3);  // id, plan of A^T or None, order or None
    auto op = get_op(integer(a[0]));
    Tensor order = tensor_or_none(a[2], "order");
    std::lock_guard<std::mutex> lock(g_ops_mutex);
    op->transposed = static_cast<cutespmm_plan_t *>(pointer(a[1]));
    op->order = order;
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}
PyObject *py_set_error_class(PyObject *, PyObject *cls)
{
    Py_INCREF(cls);
    Py_XDECREF(g_error_class);
    g_error_class = cls;
    Py_RETURN_NONE;
}

#define FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FAST("spmm", py_spmm), FAST("sddmm", py_sddmm), FAST("set_values", py_set_values), FAST("spmm_csr_noalloc", py_noalloc),
                           FAST("op_spmm", py_op_spmm), FAST("op_weighted", py_op_weighted), FAST("op_sddmm", py_op_sddmm),
                           FAST("register_op", py_register), FAST("unregister_op", py_unregister), FAST("set_transposed", py_set_transposed),
                           {"set_error_class", py_set_error_class, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_torch_bind", "Hot calls of cutespmm_ae_b200 on torch tensors.", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_bind(void) { return PyModule_Create(&g_module); }
