// Calls of the C API with torch tensors, for hccl_b200/_calls.py: checks, output allocation, the current stream and the call
// itself without Python or ctypes objects in between.  A decode step's operators take 4 .. 10 us on the device; with Python-level
// allocations and ctypes a call of one took 10 .. 18 us of the host.
//
// Every function takes only what is plain: dense CUDA tensors that no transform, subclass, dispatch or function mode,
// forward-mode gradient or tracer looks at, and (but for those of the second part) that no gradient is recorded for.  For
// anything else it returns None and the caller goes the general way (torch.autograd.Function, ctypes), which also words the
// errors.  An int is the HcclResult of a failed call.
//
// The second part (add_rms_norm_grad, swiglu_grad, rope_grad, linear, embedding) records gradients: nodes of autograd's graph in the place of
// Python functions, whose passes through the interpreter took 100 us of the host for a norm forward and backward and 250 for the
// FFN half of a layer, several times what the kernels of a small one take.
//
// The functions of the C API come as addresses (`bind`), so that this module and the ctypes binding always use the same library.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/PyInterpreter.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/accumulate_grad.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/library.h>
#include <atomic>
#include <cstdint>
#include "hccl/hccl.h"
#include "hccl/hccl_fused_ops.h"
#include "hccl/hccl_mc2.h"
#include "hccl/hccl_moe.h"

namespace {

using at::Tensor;

struct Api {
    decltype(&HcclFusedAddRmsNormFwd) addRmsNormFwd;
    decltype(&HcclFusedRmsNormBwdPartials) rmsNormBwdPartials;
    decltype(&HcclFusedRmsNormBwdCopy) rmsNormBwd;
    decltype(&HcclFusedSwigluFwd) swigluFwd;
    decltype(&HcclFusedSwigluBwd) swigluBwd;
    decltype(&HcclFusedRope) rope;
    decltype(&HcclMc2Matmul) matmul;
    decltype(&HcclFusedEmbeddingGrad) embeddingGrad;
    decltype(&HcclMoeExpertOffsets) expertOffsets;
    decltype(&HcclAllReduce) allReduce;
    decltype(&HcclReduceScatter) reduceScatter;
    decltype(&HcclAllGather) allGather;
    decltype(&HcclAlltoAll) alltoAll;
};
Api api;
struct Slot { const char* name; void** at; };
const Slot kSlots[] = {
    {"HcclFusedAddRmsNormFwd", (void**)&api.addRmsNormFwd}, {"HcclFusedRmsNormBwdPartials", (void**)&api.rmsNormBwdPartials},
    {"HcclFusedRmsNormBwdCopy", (void**)&api.rmsNormBwd},   {"HcclFusedSwigluFwd", (void**)&api.swigluFwd},
    {"HcclFusedSwigluBwd", (void**)&api.swigluBwd},         {"HcclFusedRope", (void**)&api.rope},
    {"HcclMc2Matmul", (void**)&api.matmul},                 {"HcclMoeExpertOffsets", (void**)&api.expertOffsets},
    {"HcclAllReduce", (void**)&api.allReduce},              {"HcclReduceScatter", (void**)&api.reduceScatter},
    {"HcclAllGather", (void**)&api.allGather},              {"HcclAlltoAll", (void**)&api.alltoAll},
};

// Functions that only the backward passes of recorded calls use.
const Slot kBackwardSlots[] = {{"HcclFusedEmbeddingGrad", (void**)&api.embeddingGrad}};

// The function mode behind torch.set_default_device and `with torch.device(...)`.  It gives a device to factory calls that name
// none; these calls name theirs, so that it has nothing to see here.
PyTypeObject* defaultDeviceMode = nullptr;
bool FunctionModes()
{
    if (!at::impl::torch_function_mode_enabled()) return false;
    for (int64_t i = 0; i < at::impl::PythonTorchFunctionTLS::stack_len(); ++i)
        if (Py_TYPE(at::impl::PythonTorchFunctionTLS::get_stack_at(i)->ptr(getPyInterpreter())) != defaultDeviceMode) return true;
    return false;
}
bool HasModes()
{
    return c10::impl::TorchDispatchModeTLS::any_modes_set() || c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}
// A call that nothing but its own arithmetic is asked of: no tracer, no mode, no functional transform around it.
bool PlainCall() { return !FunctionModes() && !torch::jit::tracer::isTracing() && !HasModes(); }
// A dense CUDA tensor that nothing looks at and nothing is recorded for.
bool Plain(const Tensor& t)
{
    return t.is_cuda() && t.layout() == at::kStrided && !(t.requires_grad() && c10::GradMode::is_enabled()) && !at::isTensorSubclassLike(t) &&
           !t._fw_grad(0).defined();
}
// Tensors and parameters themselves: a subclass may have a __torch_function__ of its own.
const Tensor* Get(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
const Tensor* GetPlain(PyObject* o)
{
    const Tensor* t = Get(o);
    return t != nullptr && Plain(*t) ? t : nullptr;
}
const Tensor* GetPlainBf16(PyObject* o)
{
    const Tensor* t = GetPlain(o);
    return t != nullptr && t->scalar_type() == at::kBFloat16 && t->is_contiguous() ? t : nullptr;
}
void* Stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
void* StreamOf(PyObject* o) { return o == Py_None ? Stream() : PyLong_AsVoidPtr(o); }
PyObject* None() { Py_RETURN_NONE; }
// An argument that is not what it is here (a float where an int is meant, say): the general way makes of it what it can.
bool Odd()
{
    const bool odd = PyErr_Occurred() != nullptr;
    if (odd) PyErr_Clear();
    return odd;
}
PyObject* Wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
template <class... T> PyObject* WrapAll(T... t)
{
    PyObject* all[] = {Wrap(std::move(t))...};
    PyObject* out = PyTuple_New(sizeof...(T));
    for (size_t i = 0; i < sizeof...(T); ++i) PyTuple_SET_ITEM(out, i, all[i]);
    return out;
}
// Errors of torch (out of memory among them) become the Python exceptions that torch's own functions raise.
template <class F> PyObject* Guarded(F f)
{
    HANDLE_TH_ERRORS
    return f();
    END_HANDLE_TH_ERRORS
}
// The interpreter's lock is not held while memory is allocated and the C API is called, as with torch's own functions and ctypes:
// both may wait (a full launch queue, a kernel's first load, the allocator) for what another Python thread has yet to issue.
class Unlocked {
public:
    Unlocked() : state_(PyEval_SaveThread()) {}
    ~Unlocked() { PyEval_RestoreThread(state_); }
    Unlocked(const Unlocked&) = delete;
    Unlocked& operator=(const Unlocked&) = delete;
private:
    PyThreadState* state_;
};
#define HCCL_ARGS(n) \
    if (nargs != (n)) { PyErr_SetString(PyExc_TypeError, "wrong number of arguments"); return nullptr; }

// (x, delta or None, weight, eps) -> (x_out or x, h, rstd)
PyObject* AddRmsNorm(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(4)
    return Guarded([&]() -> PyObject* {
        const Tensor *x = GetPlainBf16(a[0]), *w = GetPlainBf16(a[2]), *delta = a[1] == Py_None ? nullptr : GetPlainBf16(a[1]);
        if (!x || !w || (a[1] != Py_None && !delta) || !PyFloat_Check(a[3]) || !PlainCall()) return None();
        if (x->dim() == 0 || x->numel() == 0 || w->numel() != x->size(-1) || (delta && delta->sizes() != x->sizes())) return None();
        const uint64_t hidden = (uint64_t)x->size(-1), rows = (uint64_t)x->numel() / hidden;
        if (hidden % 8 != 0 || hidden > 8192) return None();
        const float eps = (float)PyFloat_AS_DOUBLE(a[3]);
        Tensor h, xOut, rstd;
        const int r = [&] {
            Unlocked unlocked;
            h = at::empty_like(*x);
            xOut = delta ? at::empty_like(*x) : *x;
            rstd = at::empty({(int64_t)rows}, x->options().dtype(at::kFloat));
            return api.addRmsNormFwd(x->const_data_ptr(), delta ? delta->const_data_ptr() : nullptr, w->const_data_ptr(),
                                     delta ? xOut.mutable_data_ptr() : nullptr, h.mutable_data_ptr(), rstd.mutable_data_ptr(), rows, (uint32_t)hidden, eps,
                                     Stream());
        }();
        if (r != 0) return PyLong_FromLong(r);
        return WrapAll(std::move(xOut), std::move(h), std::move(rstd));
    });
}

// (dh, x_out, weight, rstd, extra or None, a second copy of dx) -> (dx, dw, that copy or dx)
PyObject* RmsNormBwd(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(6)
    return Guarded([&]() -> PyObject* {
        const Tensor *dh = GetPlainBf16(a[0]), *x = GetPlainBf16(a[1]), *w = GetPlainBf16(a[2]), *rstd = GetPlain(a[3]);
        const Tensor* extra = a[4] == Py_None ? nullptr : GetPlainBf16(a[4]);
        if (!dh || !x || !w || !rstd || (a[4] != Py_None && !extra) || rstd->scalar_type() != at::kFloat || !rstd->is_contiguous() || !PlainCall()) return None();
        if (x->numel() == 0 || dh->sizes() != x->sizes() || (extra && extra->sizes() != x->sizes())) return None();
        const uint64_t hidden = (uint64_t)x->size(-1), rows = (uint64_t)x->numel() / hidden;
        if (w->numel() != x->size(-1) || (uint64_t)rstd->numel() != rows) return None();
        const bool twice = PyObject_IsTrue(a[5]);
        if (Odd()) return None();
        Tensor dx, dw, copy;
        const int r = [&] {
            Unlocked unlocked;
            dx = at::empty_like(*x);
            dw = at::empty_like(*w);
            copy = twice ? at::empty_like(*x) : dx;
            Tensor partial = at::empty({(int64_t)api.rmsNormBwdPartials(rows), (int64_t)hidden}, x->options().dtype(at::kFloat));
            return api.rmsNormBwd(dh->const_data_ptr(), x->const_data_ptr(), w->const_data_ptr(), rstd->const_data_ptr(),
                                  extra ? extra->const_data_ptr() : nullptr, dx.mutable_data_ptr(), twice ? copy.mutable_data_ptr() : nullptr,
                                  partial.mutable_data_ptr(), dw.mutable_data_ptr(), rows, (uint32_t)hidden, Stream());
        }();
        if (r != 0) return PyLong_FromLong(r);
        return WrapAll(std::move(dx), std::move(dw), std::move(copy));
    });
}

// (gate_up) -> out
PyObject* SwigluFwd(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(1)
    return Guarded([&]() -> PyObject* {
        const Tensor* x = GetPlainBf16(a[0]);
        if (!x || !PlainCall() || x->dim() == 0 || x->numel() == 0 || x->size(-1) % 16 != 0) return None();
        const int64_t f = x->size(-1) / 2;
        auto sizes = x->sizes().vec();
        sizes.back() = f;
        Tensor out;
        const int r = [&] {
            Unlocked unlocked;
            out = at::empty(sizes, x->options());
            return api.swigluFwd(x->const_data_ptr(), out.mutable_data_ptr(), (uint64_t)(x->numel() / (2 * f)), (uint32_t)f, Stream());
        }();
        return r != 0 ? PyLong_FromLong(r) : Wrap(std::move(out));
    });
}

// (gate_up, dout) -> dgate_up
PyObject* SwigluBwd(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(2)
    return Guarded([&]() -> PyObject* {
        const Tensor *x = GetPlainBf16(a[0]), *dout = GetPlainBf16(a[1]);
        if (!x || !dout || !PlainCall() || x->numel() == 0 || x->size(-1) % 16 != 0 || dout->numel() * 2 != x->numel()) return None();
        const int64_t f = x->size(-1) / 2;
        Tensor dx;
        const int r = [&] {
            Unlocked unlocked;
            dx = at::empty_like(*x);
            return api.swigluBwd(x->const_data_ptr(), dout->const_data_ptr(), dx.mutable_data_ptr(), (uint64_t)(x->numel() / (2 * f)), (uint32_t)f, Stream());
        }();
        return r != 0 ? PyLong_FromLong(r) : Wrap(std::move(dx));
    });
}

// (x [S, heads, D], cos, sin, backward) -> rotated x; rows of x may lie further apart than heads * D
PyObject* Rope(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(4)
    return Guarded([&]() -> PyObject* {
        const Tensor *x = GetPlain(a[0]), *c = GetPlain(a[1]), *s = GetPlain(a[2]);
        if (!x || !c || !s || !PlainCall() || x->scalar_type() != at::kBFloat16 || x->dim() != 3 || x->numel() == 0) return None();
        const int64_t rows = x->size(0), heads = x->size(1), d = x->size(2);
        if (d % 16 != 0 || x->stride(2) != 1 || x->stride(1) != d || x->stride(0) < 0 || x->stride(0) % 8 != 0 || (uintptr_t)x->const_data_ptr() % 16 != 0)
            return None();
        for (const Tensor* t : {c, s})
            if (t->scalar_type() != at::kFloat || !t->is_contiguous() || t->numel() < rows * (d / 2)) return None();
        const int backward = PyObject_IsTrue(a[3]);
        if (Odd()) return None();
        Tensor out;
        const int r = [&] {
            Unlocked unlocked;
            out = at::empty({rows, heads, d}, x->options());
            return api.rope(x->const_data_ptr(), (uint64_t)x->stride(0), out.mutable_data_ptr(), (uint64_t)(heads * d), c->const_data_ptr(),
                            s->const_data_ptr(), (uint64_t)rows, (uint32_t)heads, (uint32_t)d, backward, Stream());
        }();
        return r != 0 ? PyLong_FromLong(r) : Wrap(std::move(out));
    });
}

// (a, b, trans_a, trans_b, out or None, stream or None) -> out
PyObject* Matmul(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    HCCL_ARGS(6)
    return Guarded([&]() -> PyObject* {
        // operands that record gradients are taken as before: the product itself is not recorded
        const Tensor *a = Get(args[0]), *b = Get(args[1]), *given = args[4] == Py_None ? nullptr : Get(args[4]);
        if (!a || !b || (args[4] != Py_None && !given) || !PlainCall()) return None();
        for (const Tensor* t : {a, b, given})
            if (t && (!t->is_cuda() || t->layout() != at::kStrided || t->scalar_type() != at::kBFloat16 || t->dim() != 2 || at::isTensorSubclassLike(*t))) return None();
        if (!a->is_contiguous() || !b->is_contiguous()) return None();
        const bool ta = PyObject_IsTrue(args[2]), tb = PyObject_IsTrue(args[3]);
        void* stream = StreamOf(args[5]);
        if (Odd()) return None();
        const int64_t m = a->size(ta ? 1 : 0), k = a->size(ta ? 0 : 1), n = b->size(tb ? 0 : 1);
        if (b->size(tb ? 1 : 0) != k) return None();
        Tensor out;
        const int r = [&] {
            Unlocked unlocked;
            out = given ? *given : at::empty({m, n}, a->options());
            return api.matmul(a->const_data_ptr(), b->const_data_ptr(), out.data_ptr(), (uint64_t)m, (uint64_t)n, (uint64_t)k, ta, tb, stream);
        }();
        return r != 0 ? PyLong_FromLong(r) : Wrap(std::move(out));
    });
}

// (topk_idx, n_experts, stream or None) -> offsets
PyObject* ExpertOffsets(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(3)
    return Guarded([&]() -> PyObject* {
        const Tensor* idx = GetPlain(a[0]);
        if (!idx || !PlainCall() || idx->scalar_type() != at::kInt || !idx->is_contiguous() || !PyLong_Check(a[1])) return None();
        const long n = PyLong_AsLong(a[1]);
        void* stream = StreamOf(a[2]);
        if (Odd() || n <= 0 || n > 0x7FFFFFFFL) return None();
        Tensor out;
        const int r = [&] {
            Unlocked unlocked;
            out = at::empty({n + 1}, idx->options());
            return api.expertOffsets(idx->const_data_ptr<int32_t>(), (uint64_t)idx->numel(), (uint32_t)n, (uint32_t*)out.mutable_data_ptr(), stream);
        }();
        return r != 0 ? PyLong_FromLong(r) : Wrap(std::move(out));
    });
}

// HcclDataType of a tensor's elements, HCCL_DATA_TYPE_RESERVED where the general way has to look
HcclDataType TypeOf(const Tensor& t)
{
    switch (t.scalar_type()) {
        case at::kFloat: return HCCL_DATA_TYPE_FP32;
        case at::kBFloat16: return HCCL_DATA_TYPE_BFP16;
        default: return HCCL_DATA_TYPE_RESERVED;
    }
}
enum Which { ALL_REDUCE, REDUCE_SCATTER, ALL_GATHER, ALL_TO_ALL };
// (which, communicator, send, recv, reduction, ranks, stream or None) -> HcclResult
PyObject* Collective(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(7)
    return Guarded([&]() -> PyObject* {
        const Tensor *send = Get(a[2]), *recv = Get(a[3]);
        if (!send || !recv || !PlainCall()) return None();
        for (const Tensor* t : {send, recv})
            if (!t->is_cuda() || t->layout() != at::kStrided || !t->is_contiguous() || at::isTensorSubclassLike(*t)) return None();
        const HcclDataType type = TypeOf(*send);
        const int which = (int)PyLong_AsLong(a[0]), ranks = (int)PyLong_AsLong(a[5]);
        const HcclReduceOp op = (HcclReduceOp)PyLong_AsLong(a[4]);
        void *comm = PyLong_AsVoidPtr(a[1]), *stream = StreamOf(a[6]);
        if (Odd() || type == HCCL_DATA_TYPE_RESERVED || TypeOf(*recv) != type || comm == nullptr || ranks < 1) return None();
        void *s = const_cast<void*>(send->const_data_ptr()), *r = recv->data_ptr();
        const uint64_t nSend = (uint64_t)send->numel(), nRecv = (uint64_t)recv->numel();
        const int code = [&] {
            Unlocked unlocked;          // a first call may wait for the other ranks' threads
            switch (which) {
                case ALL_REDUCE: return api.allReduce(s, r, nSend, type, op, comm, stream);
                case REDUCE_SCATTER: return api.reduceScatter(s, r, nRecv, type, op, comm, stream);
                case ALL_GATHER: return api.allGather(s, r, nSend, type, comm, stream);
                default: return api.alltoAll(s, nSend / (uint64_t)ranks, type, r, nSend / (uint64_t)ranks, type, comm, stream);
            }
        }();
        return PyLong_FromLong(code);
    });
}

// ----------------------------------------------------------------------------- calls that record gradients
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

std::atomic<int64_t> launches{0};                  // kernels of the nodes' backward passes (benchmark accounting)
PyObject* errorClass = nullptr;                    // what a failed call raises, (code, function)

// In a backward pass, which runs on a thread of its own without the interpreter's lock.
void CheckBackward(int code, const char* what)
{
    if (code == 0) return;
    const PyGILState_STATE lock = PyGILState_Ensure();
    PyObject* error = errorClass ? PyObject_CallFunction(errorClass, "is", code, what) : nullptr;
    if (error != nullptr) {
        PyErr_SetObject(reinterpret_cast<PyObject*>(Py_TYPE(error)), error);
        Py_DECREF(error);
    } else if (!PyErr_Occurred()) {
        PyErr_Format(PyExc_RuntimeError, "%s failed (%d)", what, code);
    }
    python_error e;
    e.persist();
    PyGILState_Release(lock);
    throw e;
}
// A dense bf16 CUDA tensor that nothing but the recording of gradients looks at.
const Tensor* GetRecordable(PyObject* o, bool contiguous = true)
{
    const Tensor* t = Get(o);
    if (t == nullptr || !t->is_cuda() || t->layout() != at::kStrided || t->scalar_type() != at::kBFloat16 || at::isTensorSubclassLike(*t) ||
        t->_fw_grad(0).defined() || (contiguous && !t->is_contiguous()))
        return nullptr;
    return t;
}
bool Records(std::initializer_list<const Tensor*> inputs)
{
    if (!c10::GradMode::is_enabled()) return false;
    for (const Tensor* t : inputs)
        if (t != nullptr && t->requires_grad()) return true;
    return false;
}
// Owned as autograd owns its own nodes: long chains of them are freed one by one, not in each other's destructors.
template <class T> std::shared_ptr<T> NewNode() { return std::shared_ptr<T>(new T(), torch::autograd::deleteNode); }
template <class... T> void TakeInputs(const std::shared_ptr<Node>& node, const T&... inputs) { node->set_next_edges(torch::autograd::collect_next_edges(inputs...)); }
void GiveOutput(const std::shared_ptr<Node>& node, const Tensor& out)
{
    const uint32_t nr = node->add_input_metadata(out);
    torch::autograd::impl::set_gradient_edge(out, {node, nr});
}
// The gradient of a node's only output; zeros where what used that output gave none, as functions in Python get them.
Tensor GradientOf(const torch::autograd::InputMetadata& output, const Tensor& given) { return given.defined() ? given : output.zeros_like(); }
// The gradient of an input ends in a leaf that holds none yet: the leaf keeps the tensor it is given if nobody else has it, and
// copies it otherwise.  (Under autograd.grad the leaves keep nothing.)
torch::autograd::AccumulateGrad* EmptyLeaf(const torch::autograd::Edge& edge)
{
    auto* leaf = dynamic_cast<torch::autograd::AccumulateGrad*>(edge.function.get());
    if (leaf == nullptr || leaf->variable.grad().defined()) return nullptr;
    const auto* executed = torch::autograd::get_current_graph_task_exec_info();
    if (executed == nullptr) return nullptr;
    if (executed->empty()) return leaf;
    const auto it = executed->find(leaf);
    return it != executed->end() && it->second.needed_ && !it->second.captures_ ? leaf : nullptr;
}

// ---- gradients of plain tensors: what the nodes' backward passes launch
// (dx, dw, dx or, if that is asked for, a second copy of it)
std::tuple<Tensor, Tensor, Tensor> NormGradient(const Tensor& dh, const Tensor& x, const Tensor& w, const Tensor& rstd, const Tensor& extra, bool twice)
{
    const int64_t hidden = x.size(-1);
    const uint64_t rows = (uint64_t)(x.numel() / hidden);
    Tensor dx = at::empty_like(x), copy = twice ? at::empty_like(x) : dx, dw = at::empty_like(w);
    Tensor partial = at::empty({(int64_t)api.rmsNormBwdPartials(rows), hidden}, x.options().dtype(at::kFloat));
    CheckBackward(api.rmsNormBwd(dh.const_data_ptr(), x.const_data_ptr(), w.const_data_ptr(), rstd.const_data_ptr(), extra.defined() ? extra.const_data_ptr() : nullptr,
                                 dx.mutable_data_ptr(), twice ? copy.mutable_data_ptr() : nullptr, partial.mutable_data_ptr(), dw.mutable_data_ptr(), rows,
                                 (uint32_t)hidden, Stream()),
                  "HcclFusedRmsNormBwdCopy");
    launches += 2;
    return {std::move(dx), std::move(dw), std::move(copy)};
}
Tensor SwigluGradient(const Tensor& dout, const Tensor& x)
{
    const int64_t f = x.size(-1) / 2;
    Tensor dx = at::empty_like(x);
    CheckBackward(api.swigluBwd(x.const_data_ptr(), dout.const_data_ptr(), dx.mutable_data_ptr(), (uint64_t)(x.numel() / (2 * f)), (uint32_t)f, Stream()),
                  "HcclFusedSwigluBwd");
    launches += 1;
    return dx;
}
Tensor RopeGradient(const Tensor& dout, const Tensor& cos, const Tensor& sin)
{
    const int64_t rows = dout.size(0), heads = dout.size(1), d = dout.size(2);
    Tensor dx = at::empty_like(dout);
    CheckBackward(api.rope(dout.const_data_ptr(), (uint64_t)(heads * d), dx.mutable_data_ptr(), (uint64_t)(heads * d), cos.const_data_ptr(), sin.const_data_ptr(),
                           (uint64_t)rows, (uint32_t)heads, (uint32_t)d, 1, Stream()),
                  "HcclFusedRope");
    launches += 1;
    return dx;
}
// (dx, dw)
std::tuple<Tensor, Tensor> LinearGradient(const Tensor& dy, const Tensor& x, const Tensor& w)
{
    const uint64_t rows = (uint64_t)dy.size(0), n = (uint64_t)dy.size(1), k = (uint64_t)x.size(1);
    Tensor dw = at::empty({(int64_t)n, (int64_t)k}, dy.options()), dx = at::empty({(int64_t)rows, (int64_t)k}, dy.options());
    CheckBackward(api.matmul(dy.const_data_ptr(), x.const_data_ptr(), dw.mutable_data_ptr(), n, k, rows, 1, 0, Stream()), "HcclMc2Matmul");
    CheckBackward(api.matmul(dy.const_data_ptr(), w.const_data_ptr(), dx.mutable_data_ptr(), rows, k, n, 0, 0, Stream()), "HcclMc2Matmul");
    return {std::move(dx), std::move(dw)};
}

// ---- the same as operators of torch, for compiled backward passes (compiled autograd): its graph traces the nodes with tensors that have
// no memory, holds these operators and launches when it runs
using torch::dynamo::autograd::CompiledNodeArgs;
using torch::dynamo::autograd::SwapSavedVariables;
namespace ops {
// Anyone can call an operator: what the nodes know of their tensors is checked here.
template <class... T> bool Bf16(const T&... t) { return ((t.scalar_type() == at::kBFloat16) && ...); }
std::tuple<Tensor, Tensor> Norm(const Tensor& dh, const Tensor& x, const Tensor& w, const Tensor& rstd, const std::optional<Tensor>& extra)
{
    TORCH_CHECK(Bf16(dh, x, w) && rstd.scalar_type() == at::kFloat && x.dim() > 0 && x.numel() > 0 && x.size(-1) % 8 == 0 && x.size(-1) <= 8192 &&
                    dh.sizes() == x.sizes() && w.numel() == x.size(-1) && rstd.numel() == x.numel() / x.size(-1) && (!extra || (Bf16(*extra) && extra->sizes() == x.sizes())),
                "norm_backward: tensors of other types or sizes than a norm has");
    auto [dx, dw, copy] = NormGradient(dh.contiguous(), x.contiguous(), w.contiguous(), rstd.contiguous(), extra ? extra->contiguous() : Tensor(), false);
    return {std::move(dx), std::move(dw)};
}
Tensor Swiglu(const Tensor& dout, const Tensor& x)
{
    TORCH_CHECK(Bf16(dout, x) && x.dim() > 0 && x.numel() > 0 && x.size(-1) % 16 == 0 && dout.numel() * 2 == x.numel(), "swiglu_backward: tensors of other types or sizes than SwiGLU has");
    return SwigluGradient(dout.contiguous(), x.contiguous());
}
Tensor Rope(const Tensor& dout, const Tensor& cos, const Tensor& sin)
{
    TORCH_CHECK(Bf16(dout) && dout.dim() == 3 && dout.numel() > 0 && dout.size(2) % 16 == 0, "rope_backward: no bf16 gradient [rows, heads, a multiple of 16]");
    for (const Tensor* t : {&cos, &sin})
        TORCH_CHECK(t->scalar_type() == at::kFloat && t->numel() >= dout.size(0) * (dout.size(2) / 2), "rope_backward: no fp32 table that holds every row");
    return RopeGradient(dout.contiguous(), cos.contiguous(), sin.contiguous());
}
std::tuple<Tensor, Tensor> Linear(const Tensor& dy, const Tensor& x, const Tensor& w)
{
    TORCH_CHECK(Bf16(dy, x, w) && dy.dim() == 2 && x.dim() == 2 && w.dim() == 2 && dy.size(0) == x.size(0) && dy.size(1) == w.size(0) && x.size(1) == w.size(1),
                "linear_backward: tensors of other types or sizes than a linear layer has");
    auto out = LinearGradient(dy.contiguous(), x.contiguous(), w.contiguous());
    launches += 2;
    return out;
}
Tensor PackedLike(const Tensor& t) { return at::empty_symint(t.sym_sizes(), t.options()); }
void Define()
{
    if (c10::Dispatcher::singleton().findSchema({"hccl_b200::linear_backward", ""})) return;       // by another copy of this module
    static torch::Library lib(torch::Library::FRAGMENT, "hccl_b200", std::nullopt, __FILE__, __LINE__);
    lib.def("norm_backward(Tensor dh, Tensor x, Tensor weight, Tensor rstd, Tensor? extra) -> (Tensor, Tensor)");
    lib.def("swiglu_backward(Tensor dout, Tensor gate_up) -> Tensor");
    lib.def("rope_backward(Tensor dout, Tensor cos, Tensor sin) -> Tensor");
    lib.def("linear_backward(Tensor dy, Tensor x, Tensor weight) -> (Tensor, Tensor)");
    lib.impl("norm_backward", torch::dispatch(c10::DispatchKey::CUDA, Norm));
    lib.impl("swiglu_backward", torch::dispatch(c10::DispatchKey::CUDA, Swiglu));
    lib.impl("rope_backward", torch::dispatch(c10::DispatchKey::CUDA, Rope));
    lib.impl("linear_backward", torch::dispatch(c10::DispatchKey::CUDA, Linear));
    lib.impl("norm_backward", torch::dispatch(c10::DispatchKey::Meta, [](const Tensor&, const Tensor& x, const Tensor& w, const Tensor&, const std::optional<Tensor>&) {
                 return std::tuple<Tensor, Tensor>(PackedLike(x), PackedLike(w));
             }));
    lib.impl("swiglu_backward", torch::dispatch(c10::DispatchKey::Meta, [](const Tensor&, const Tensor& x) { return PackedLike(x); }));
    lib.impl("rope_backward", torch::dispatch(c10::DispatchKey::Meta, [](const Tensor& dout, const Tensor&, const Tensor&) { return PackedLike(dout); }));
    lib.impl("linear_backward", torch::dispatch(c10::DispatchKey::Meta, [](const Tensor&, const Tensor& x, const Tensor& w) {
                 return std::tuple<Tensor, Tensor>(PackedLike(x), PackedLike(w));
             }));
}
template <class F> c10::TypedOperatorHandle<F> Find(const char* name) { return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<F>(); }
}  // namespace ops
using torch::autograd::InputMetadata;
using torch::dynamo::autograd::IValuePacker;
using torch::dynamo::autograd::PackedArgs;
// A node's backward pass as a call in the graph of a compiled one: `apply` gets the gradients and what is read from `saved`, in the place of
// which stands what the trace has given for it.
template <class... T> class Traced {
public:
    Traced(SwapSavedVariables& trace, T&... saved) : trace_(trace), saved_(saved...) { std::apply([&](auto&... s) { (trace_.before(s), ...); }, saved_); }
    ~Traced() { std::apply([&](auto&... s) { (trace_.after(s), ...); }, saved_); }
    Traced(const Traced&) = delete;
    Traced& operator=(const Traced&) = delete;
    template <class... A> variable_list Call(const Node& node, const variable_list& grads, variable_list (*apply)(const variable_list&, const std::vector<c10::IValue>&),
                                             const A&... args) const
    {
        const auto& compiler = torch::dynamo::autograd::getPyCompilerInterface();
        const std::string name = compiler->bind_function(trace_.get_py_compiler(), node.name(), apply, {IValuePacker<A>::packed_type()...}, true, true);
        PackedArgs packed;
        (packed.pack(args), ...);
        return compiler->call_function(trace_.get_py_compiler(), "apply_functional", name, grads, packed.vec(),
                                       IValuePacker<std::vector<std::optional<InputMetadata>>>::pack(torch::dynamo::autograd::get_input_metadata(node.next_edges())));
    }
private:
    SwapSavedVariables& trace_;
    std::tuple<T&...> saved_;
};

struct AddRmsNormNode : Node {
    SavedVariable xOut, weight, rstd;
    bool hasDelta = false;
    std::string name() const override { return "_AddRmsNormBackward"; }
    void release_variables() override
    {
        std::lock_guard<std::mutex> lock(mutex_);
        xOut.reset_data();
        weight.reset_data();
        rstd.reset_data();
    }
    variable_list apply(variable_list&& grads) override
    {
        Tensor x, w, r;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            x = xOut.unpack(hasDelta ? shared_from_this() : nullptr);
            w = weight.unpack();
            r = rstd.unpack();
        }
        c10::AutoGradMode off(false);
        const Tensor extra = hasDelta && grads[0].defined() ? grads[0].contiguous() : Tensor();
        const Tensor& given = grads[hasDelta ? 1 : 0];
        const Tensor dh = given.defined() ? given.contiguous() : at::zeros_like(x);
        const torch::autograd::AccumulateGrad* first = hasDelta ? EmptyLeaf(next_edge(0)) : nullptr;
        const torch::autograd::AccumulateGrad* second = first ? EmptyLeaf(next_edge(1)) : nullptr;
        auto [dx, dw, copy] = NormGradient(dh, x, w, r, extra, second != nullptr && first != second);
        if (!hasDelta) return {std::move(dx), std::move(dw)};
        return {std::move(dx), std::move(copy), std::move(dw)};
    }
    void compiled_args(CompiledNodeArgs& args) const override
    {
        args.collect(hasDelta);
        args.collect(xOut, hasDelta);
        args.collect(weight, false);
        args.collect(rstd, false);
    }
    variable_list apply_with_saved(const variable_list& grads, SwapSavedVariables& saved) override
    {
        const Traced traced(saved, xOut, weight, rstd);
        return traced.Call(*this, grads, Compiled, xOut.unpack(hasDelta ? shared_from_this() : nullptr), weight.unpack(), rstd.unpack(), hasDelta);
    }
    static variable_list Compiled(const variable_list& grads, const std::vector<c10::IValue>& args)
    {
        PackedArgs packed(args);
        const Tensor x = packed.unpack<Tensor>(), w = packed.unpack<Tensor>(), r = packed.unpack<Tensor>();
        const bool hasDelta = packed.unpack<bool>();
        const Tensor& dh = grads[hasDelta ? 1 : 0];
        const std::optional<Tensor> extra = hasDelta && grads[0].defined() ? std::optional<Tensor>(grads[0]) : std::nullopt;
        static const auto op = ops::Find<decltype(ops::Norm)>("hccl_b200::norm_backward");
        auto [dx, dw] = op.call(dh.defined() ? dh : at::zeros_like(x), x, w, r, extra);
        if (!hasDelta) return {std::move(dx), std::move(dw)};
        Tensor copy = dx.clone();
        return {std::move(dx), std::move(copy), std::move(dw)};
    }
};
// (x, delta or None, weight, eps) -> (x_out or x, h)
PyObject* AddRmsNormGrad(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(4)
    return Guarded([&]() -> PyObject* {
        const Tensor *x = GetRecordable(a[0]), *w = GetRecordable(a[2]), *delta = a[1] == Py_None ? nullptr : GetRecordable(a[1]);
        if (!x || !w || (a[1] != Py_None && !delta) || !PyFloat_Check(a[3]) || !Records({x, w, delta}) || !PlainCall()) return None();
        if (x->dim() == 0 || x->numel() == 0 || w->numel() != x->size(-1) || (delta && delta->sizes() != x->sizes())) return None();
        const uint64_t hidden = (uint64_t)x->size(-1), rows = (uint64_t)x->numel() / hidden;
        if (hidden % 8 != 0 || hidden > 8192) return None();
        const float eps = (float)PyFloat_AS_DOUBLE(a[3]);
        Tensor h, xOut;
        const int r = [&] {
            Unlocked unlocked;
            c10::AutoGradMode off(false);
            h = at::empty_like(*x);
            xOut = delta ? at::empty_like(*x) : *x;
            Tensor rstd = at::empty({(int64_t)rows}, x->options().dtype(at::kFloat));
            const int code = api.addRmsNormFwd(x->const_data_ptr(), delta ? delta->const_data_ptr() : nullptr, w->const_data_ptr(),
                                               delta ? xOut.mutable_data_ptr() : nullptr, h.mutable_data_ptr(), rstd.mutable_data_ptr(), rows, (uint32_t)hidden, eps,
                                               Stream());
            if (code != 0) return code;
            auto node = NewNode<AddRmsNormNode>();
            node->hasDelta = delta != nullptr;
            if (delta) TakeInputs(node, *x, *delta, *w);
            else TakeInputs(node, *x, *w);
            if (delta) GiveOutput(node, xOut);
            GiveOutput(node, h);
            node->xOut = SavedVariable(xOut, delta != nullptr);
            node->weight = SavedVariable(*w, false);
            node->rstd = SavedVariable(rstd, false);
            return 0;
        }();
        if (r != 0) return PyLong_FromLong(r);
        return WrapAll(std::move(xOut), std::move(h));
    });
}

struct SwigluNode : Node {
    SavedVariable gateUp;
    std::string name() const override { return "_SwigluBackward"; }
    void release_variables() override
    {
        std::lock_guard<std::mutex> lock(mutex_);
        gateUp.reset_data();
    }
    variable_list apply(variable_list&& grads) override
    {
        Tensor x;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            x = gateUp.unpack();
        }
        c10::AutoGradMode off(false);
        return {SwigluGradient(GradientOf(input_metadata(0), grads[0]).contiguous(), x)};
    }
    void compiled_args(CompiledNodeArgs& args) const override
    {
        args.collect(gateUp, false);
        args.collect(input_metadata(0));
    }
    variable_list apply_with_saved(const variable_list& grads, SwapSavedVariables& saved) override
    {
        const Traced traced(saved, gateUp, mutable_input_metadata(0));
        return traced.Call(*this, grads, Compiled, gateUp.unpack(), input_metadata(0));
    }
    static variable_list Compiled(const variable_list& grads, const std::vector<c10::IValue>& args)
    {
        PackedArgs packed(args);
        const Tensor x = packed.unpack<Tensor>();
        static const auto op = ops::Find<decltype(ops::Swiglu)>("hccl_b200::swiglu_backward");
        return {op.call(GradientOf(packed.unpack<InputMetadata>(), grads[0]), x)};
    }
};
// (gate_up) -> out
PyObject* SwigluGrad(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(1)
    return Guarded([&]() -> PyObject* {
        const Tensor* x = GetRecordable(a[0]);
        if (!x || !Records({x}) || !PlainCall() || x->dim() == 0 || x->numel() == 0 || x->size(-1) % 16 != 0) return None();
        const int64_t f = x->size(-1) / 2;
        auto sizes = x->sizes().vec();
        sizes.back() = f;
        Tensor out;
        const int r = [&] {
            Unlocked unlocked;
            c10::AutoGradMode off(false);
            out = at::empty(sizes, x->options());
            const int code = api.swigluFwd(x->const_data_ptr(), out.mutable_data_ptr(), (uint64_t)(x->numel() / (2 * f)), (uint32_t)f, Stream());
            if (code != 0) return code;
            auto node = NewNode<SwigluNode>();
            TakeInputs(node, *x);
            GiveOutput(node, out);
            node->gateUp = SavedVariable(*x, false);
            return 0;
        }();
        return r != 0 ? PyLong_FromLong(r) : Wrap(std::move(out));
    });
}

struct RopeNode : Node {
    SavedVariable cos, sin;
    std::string name() const override { return "_RopeBackward"; }
    void release_variables() override
    {
        std::lock_guard<std::mutex> lock(mutex_);
        cos.reset_data();
        sin.reset_data();
    }
    variable_list apply(variable_list&& grads) override
    {
        Tensor c, s;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            c = cos.unpack();
            s = sin.unpack();
        }
        c10::AutoGradMode off(false);
        return {RopeGradient(GradientOf(input_metadata(0), grads[0]).contiguous(), c, s)};
    }
    void compiled_args(CompiledNodeArgs& args) const override
    {
        args.collect(cos, false);
        args.collect(sin, false);
        args.collect(input_metadata(0));
    }
    variable_list apply_with_saved(const variable_list& grads, SwapSavedVariables& saved) override
    {
        const Traced traced(saved, cos, sin, mutable_input_metadata(0));
        return traced.Call(*this, grads, Compiled, cos.unpack(), sin.unpack(), input_metadata(0));
    }
    static variable_list Compiled(const variable_list& grads, const std::vector<c10::IValue>& args)
    {
        PackedArgs packed(args);
        const Tensor c = packed.unpack<Tensor>(), s = packed.unpack<Tensor>();
        static const auto op = ops::Find<decltype(ops::Rope)>("hccl_b200::rope_backward");
        return {op.call(GradientOf(packed.unpack<InputMetadata>(), grads[0]), c, s)};
    }
};
// (x [S, heads, D], cos, sin) -> rotated x
PyObject* RopeGrad(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(3)
    return Guarded([&]() -> PyObject* {
        const Tensor *x = GetRecordable(a[0], false), *c = GetPlain(a[1]), *s = GetPlain(a[2]);
        if (!x || !c || !s || !Records({x}) || !PlainCall() || x->dim() != 3 || x->numel() == 0) return None();
        const int64_t rows = x->size(0), heads = x->size(1), d = x->size(2);
        if (d % 16 != 0 || x->stride(2) != 1 || x->stride(1) != d || x->stride(0) < 0 || x->stride(0) % 8 != 0 || (uintptr_t)x->const_data_ptr() % 16 != 0)
            return None();
        for (const Tensor* t : {c, s})
            if (t->scalar_type() != at::kFloat || !t->is_contiguous() || t->numel() < rows * (d / 2)) return None();
        Tensor out;
        const int r = [&] {
            Unlocked unlocked;
            c10::AutoGradMode off(false);
            out = at::empty({rows, heads, d}, x->options());
            const int code = api.rope(x->const_data_ptr(), (uint64_t)x->stride(0), out.mutable_data_ptr(), (uint64_t)(heads * d), c->const_data_ptr(),
                                      s->const_data_ptr(), (uint64_t)rows, (uint32_t)heads, (uint32_t)d, 0, Stream());
            if (code != 0) return code;
            auto node = NewNode<RopeNode>();
            TakeInputs(node, *x);
            GiveOutput(node, out);
            node->cos = SavedVariable(*c, false);
            node->sin = SavedVariable(*s, false);
            return 0;
        }();
        return r != 0 ? PyLong_FromLong(r) : Wrap(std::move(out));
    });
}

struct LinearNode : Node {
    SavedVariable x, weight;
    Tensor counter;                                // int64 on the host: kernels launched
    std::string name() const override { return "_LinearBackward"; }
    void release_variables() override
    {
        std::lock_guard<std::mutex> lock(mutex_);
        x.reset_data();
        weight.reset_data();
    }
    variable_list apply(variable_list&& grads) override
    {
        Tensor in, w;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            in = x.unpack();
            w = weight.unpack();
        }
        c10::AutoGradMode off(false);
        auto [dx, dw] = LinearGradient(GradientOf(input_metadata(0), grads[0]).contiguous(), in, w);
        __atomic_fetch_add(counter.mutable_data_ptr<int64_t>(), 2, __ATOMIC_RELAXED);
        return {std::move(dx), std::move(dw)};
    }
    void compiled_args(CompiledNodeArgs& args) const override
    {
        args.collect(x, false);
        args.collect(weight, false);
        args.collect(input_metadata(0));
    }
    variable_list apply_with_saved(const variable_list& grads, SwapSavedVariables& saved) override
    {
        const Traced traced(saved, x, weight, mutable_input_metadata(0));
        return traced.Call(*this, grads, Compiled, x.unpack(), weight.unpack(), input_metadata(0));
    }
    static variable_list Compiled(const variable_list& grads, const std::vector<c10::IValue>& args)
    {
        PackedArgs packed(args);
        const Tensor in = packed.unpack<Tensor>(), w = packed.unpack<Tensor>();
        static const auto op = ops::Find<decltype(ops::Linear)>("hccl_b200::linear_backward");
        auto [dx, dw] = op.call(GradientOf(packed.unpack<InputMetadata>(), grads[0]), in, w);
        return {std::move(dx), std::move(dw)};
    }
};
// (x [rows, k], weight [n, k], counter of launches) -> x @ weight^T
PyObject* Linear(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(3)
    return Guarded([&]() -> PyObject* {
        const Tensor *x = GetRecordable(a[0]), *w = GetRecordable(a[1]), *counter = Get(a[2]);
        if (!x || !w || !counter || counter->scalar_type() != at::kLong || counter->numel() != 1 || !counter->is_cpu() || !PlainCall()) return None();
        if (x->dim() != 2 || w->dim() != 2 || x->numel() == 0 || w->numel() == 0 || x->size(1) != w->size(1)) return None();
        const bool record = Records({x, w});
        Tensor out;
        const int r = [&] {
            Unlocked unlocked;
            c10::AutoGradMode off(false);
            out = at::empty({x->size(0), w->size(0)}, x->options());
            const int code = api.matmul(x->const_data_ptr(), w->const_data_ptr(), out.mutable_data_ptr(), (uint64_t)x->size(0), (uint64_t)w->size(0),
                                        (uint64_t)x->size(1), 0, 1, Stream());
            if (code != 0) return code;
            if (!record) return 0;
            auto node = NewNode<LinearNode>();
            TakeInputs(node, *x, *w);
            GiveOutput(node, out);
            node->x = SavedVariable(*x, false);
            node->weight = SavedVariable(*w, false);
            node->counter = *counter;
            return 0;
        }();
        return r != 0 ? PyLong_FromLong(r) : Wrap(std::move(out));
    });
}
struct EmbeddingNode : Node {
    SavedVariable ids;
    int64_t vocab = 0;
    std::string name() const override { return "_EmbeddingBackward"; }
    void release_variables() override
    {
        std::lock_guard<std::mutex> lock(mutex_);
        ids.reset_data();
    }
    variable_list apply(variable_list&& grads) override
    {
        if (!grads[0].defined()) return {Tensor()};
        Tensor i;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            i = ids.unpack();
        }
        // A gradient that is recorded itself (create_graph), batched, dual, a subclass or seen by a mode takes PyTorch's operator, which
        // all of these look into; ids that a hook has given back in another form too.
        if (!Plain(grads[0]) || !Plain(i) || i.scalar_type() != at::kLong || !i.is_contiguous() || HasModes()) return {at::embedding_dense_backward(grads[0], i, vocab, -1, false)};
        c10::AutoGradMode off(false);
        Tensor dy = grads[0].contiguous();
        if ((uintptr_t)dy.const_data_ptr() % 16 != 0) dy = dy.clone();      // a packed view that does not begin on 16 bytes
        Tensor dTable = at::empty({vocab, dy.size(1)}, dy.options()), scratch = at::empty({8 * dy.size(0)}, dy.options().dtype(at::kByte));
        CheckBackward(api.embeddingGrad(i.const_data_ptr<int64_t>(), dy.const_data_ptr(), dTable.mutable_data_ptr(), scratch.mutable_data_ptr(), (uint64_t)dy.size(0),
                                        (uint64_t)vocab, (uint32_t)dy.size(1), Stream()),
                      "HcclFusedEmbeddingGrad");
        launches += 2;
        return {std::move(dTable)};
    }
    void compiled_args(CompiledNodeArgs& args) const override
    {
        args.collect(ids, false);
        args.collect(vocab);
    }
    variable_list apply_with_saved(const variable_list& grads, SwapSavedVariables& saved) override
    {
        const Traced traced(saved, ids);
        return traced.Call(*this, grads, Compiled, ids.unpack(), vocab);
    }
    static variable_list Compiled(const variable_list& grads, const std::vector<c10::IValue>& args)
    {
        if (!grads[0].defined()) return {Tensor()};
        PackedArgs packed(args);
        const Tensor i = packed.unpack<Tensor>();
        return {at::embedding_dense_backward(grads[0], i, packed.unpack<int64_t>(), -1, false)};
    }
};
// (ids [tokens], table [vocab, hidden]) -> the rows
PyObject* Embedding(PyObject*, PyObject* const* a, Py_ssize_t nargs)
{
    HCCL_ARGS(2)
    return Guarded([&]() -> PyObject* {
        const Tensor *ids = GetPlain(a[0]), *table = GetRecordable(a[1]);
        if (api.embeddingGrad == nullptr || !ids || !table || !Records({table}) || !PlainCall() || ids->scalar_type() != at::kLong || ids->dim() != 1 || !ids->is_contiguous()) return None();
        if (table->dim() != 2 || table->numel() == 0 || ids->numel() == 0 || ids->numel() > 8192 || table->size(1) % 8 != 0 || table->size(0) > (1 << 24)) return None();
        Tensor out;
        {
            Unlocked unlocked;
            c10::AutoGradMode off(false);
            out = at::embedding(*table, *ids);
            auto node = NewNode<EmbeddingNode>();
            TakeInputs(node, *table);
            GiveOutput(node, out);
            node->ids = SavedVariable(*ids, false);
            node->vocab = table->size(0);
        }
        return Wrap(std::move(out));
    });
}
PyObject* Launches(PyObject*, PyObject*) { return PyLong_FromLongLong(launches.load()); }
PyObject* Raises(PyObject*, PyObject* error)
{
    Py_INCREF(error);
    Py_XSETREF(errorClass, error);
    Py_RETURN_NONE;
}

PyObject* BindSlots(const Slot* slots, size_t n, PyObject* addresses)
{
    for (size_t i = 0; i < n; ++i) {
        PyObject* v = PyDict_GetItemString(addresses, slots[i].name);
        void* p = v ? PyLong_AsVoidPtr(v) : nullptr;
        if (p == nullptr) {
            if (!PyErr_Occurred()) PyErr_Format(PyExc_KeyError, "no address of %s", slots[i].name);
            return nullptr;
        }
        *slots[i].at = p;
    }
    Py_RETURN_NONE;
}
PyObject* Bind(PyObject*, PyObject* addresses)
{
    if (Guarded([]() -> PyObject* { ops::Define(); return Py_None; }) == nullptr) return nullptr;
    if (defaultDeviceMode == nullptr) {
        PyObject* devices = PyImport_ImportModule("torch.utils._device");
        PyObject* mode = devices ? PyObject_GetAttrString(devices, "DeviceContext") : nullptr;
        if (mode && PyType_Check(mode)) defaultDeviceMode = reinterpret_cast<PyTypeObject*>(mode);          // kept
        else Py_XDECREF(mode);
        Py_XDECREF(devices);
        PyErr_Clear();                 // another torch without it: its default devices go the general way
    }
    return BindSlots(kSlots, sizeof(kSlots) / sizeof(kSlots[0]), addresses);
}
PyObject* BindBackward(PyObject*, PyObject* addresses) { return BindSlots(kBackwardSlots, sizeof(kBackwardSlots) / sizeof(kBackwardSlots[0]), addresses); }
PyObject* NamesOf(const Slot* slots, size_t n)
{
    PyObject* out = PyList_New(0);
    for (size_t i = 0; i < n; ++i) {
        PyObject* name = PyUnicode_FromString(slots[i].name);
        PyList_Append(out, name);
        Py_DECREF(name);
    }
    return out;
}
PyObject* Names(PyObject*, PyObject*) { return NamesOf(kSlots, sizeof(kSlots) / sizeof(kSlots[0])); }
PyObject* BackwardNames(PyObject*, PyObject*) { return NamesOf(kBackwardSlots, sizeof(kBackwardSlots) / sizeof(kBackwardSlots[0])); }

#define HCCL_FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr
PyMethodDef methods[] = {
    {"bind", Bind, METH_O, nullptr},           {"names", Names, METH_NOARGS, nullptr},      {"add_rms_norm", HCCL_FAST(AddRmsNorm)},
    {"rms_norm_bwd", HCCL_FAST(RmsNormBwd)},   {"swiglu_fwd", HCCL_FAST(SwigluFwd)},        {"swiglu_bwd", HCCL_FAST(SwigluBwd)},
    {"rope", HCCL_FAST(Rope)},                 {"matmul", HCCL_FAST(Matmul)},               {"expert_offsets", HCCL_FAST(ExpertOffsets)},
    {"collective", HCCL_FAST(Collective)},     {"add_rms_norm_grad", HCCL_FAST(AddRmsNormGrad)},
    {"swiglu_grad", HCCL_FAST(SwigluGrad)},    {"rope_grad", HCCL_FAST(RopeGrad)},          {"linear", HCCL_FAST(Linear)},
    {"embedding", HCCL_FAST(Embedding)},
    {"bind_backward", BindBackward, METH_O, nullptr}, {"backward_names", BackwardNames, METH_NOARGS, nullptr},
    {"launches", Launches, METH_NOARGS, nullptr}, {"raises", Raises, METH_O, nullptr},      {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "hccl_b200_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_hccl_b200_torch() { return PyModule_Create(&module); }
