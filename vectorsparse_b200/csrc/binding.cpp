// CPython extension module `_binding`: the fast way from torch tensors to the C ABI.
//
// A call of one small product costs the host more than the GPU: through ctypes and Python-side checks the operators took
// 17-28 us per call on a B200 host, against 13-16 us of GPU time.  Each function here takes the operator's arguments as
// they stand, checks them without creating Python objects, finds the current stream and calls the library.  It answers
//     an int   the library's return code (0, VS_ERR_* or a cudaError_t)
//     None     some argument is not what the fast path takes (wrong type, device, layout or size): the Python operator
//              then makes its own checks, which raise the error that belongs to the argument
// so there is one set of error messages.  The library's functions are handed over by address (bind), so that the library
// that vectorsparse_b200._lib has loaded is the one that is called.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <ATen/record_function.h>
#include <c10/core/SafePyObject.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/PyInterpreter.h>
#include <torch/csrc/Exceptions.h>

#include <climits>
#include <cstdint>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "vsparse_b200.h"

namespace {

struct Library {
    decltype(&vs_spmm_batched) spmm;
    decltype(&vs_spmm_t_batched) spmm_t;
    decltype(&vs_sddmm_batched) sddmm;
    decltype(&vs_softmax_cvse) softmax;
    decltype(&vs_softmax_cvse_backward) softmax_backward;
    decltype(&vs_attention_cvse) attention;
    decltype(&vs_attention_cvse_backward) attention_backward;
} g_lib;

// The arguments of one call: `ok` turns false at the first one the fast path does not take.
struct Args {
    PyObject *const *argv;
    bool ok = true;
    int device = -1;

    explicit Args(PyObject *const *a) : argv(a) {}

    int64_t integer64(int i) {
        const long long v = PyLong_CheckExact(argv[i]) ? PyLong_AsLongLong(argv[i]) : -1;
        if (!PyLong_CheckExact(argv[i]) || (v == -1 && PyErr_Occurred())) {
            PyErr_Clear();
            ok = false;
        }
        return v;
    }
    int integer(int i) {
        const int64_t v = integer64(i);
        if (v < INT_MIN || v > INT_MAX) ok = false;
        return (int)v;
    }
    double number(int i) {
        if (PyFloat_CheckExact(argv[i])) return PyFloat_AS_DOUBLE(argv[i]);
        if (PyLong_CheckExact(argv[i])) return (double)integer64(i);
        ok = false;
        return 0.0;
    }
    bool none(int i) const { return argv[i] == Py_None; }
    // a contiguous CUDA tensor on the device of the others
    const at::Tensor *tensor(int i) {
        if (!ok || !THPVariable_Check(argv[i])) {
            ok = false;
            return nullptr;
        }
        const at::Tensor &t = THPVariable_Unpack(argv[i]);
        if (!t.is_cuda() || !t.is_contiguous()) {
            ok = false;
            return nullptr;
        }
        const int dev = t.get_device();
        if (device < 0) device = dev;
        if (dev != device) ok = false;
        return &t;
    }
    void need(const at::Tensor *t, int64_t numel) {
        if (!ok || t->numel() < numel) ok = false;
    }
    void type(const at::Tensor *t, at::ScalarType want) {
        if (!ok || t->scalar_type() != want) ok = false;
    }
    const int32_t *index(int i, int64_t numel) {
        const at::Tensor *t = tensor(i);
        need(t, numel);
        type(t, at::kInt);
        return ok ? static_cast<const int32_t *>(t->const_data_ptr()) : nullptr;
    }
    int dtype(const at::Tensor *t) {
        if (ok && t->scalar_type() == at::kHalf) return VS_F16;
        if (ok && t->scalar_type() == at::kFloat) return VS_F32;
        ok = false;
        return -1;
    }
};

// Element stride between the problems of a batch; 0 for one problem or a shared operand.
int64_t batch_stride(const at::Tensor *t, int batched_dims, int batch) {
    return batch > 1 && t->dim() == batched_dims ? t->stride(0) : 0;
}
int64_t lead(const at::Tensor *t, int batched_dims, int batch) { return t->dim() == batched_dims ? batch : 1; }

// Makes `device` current for the call (a look at the current one when it already is) and names its current stream.  Other
// Python threads run while the library is in the call: it can block (a full launch queue, an allocation, a kernel's first
// load), and what it waits for may be a callback of one of them.  `enqueue` therefore holds addresses and numbers only: a
// tensor's may change as soon as other threads run, and reading them may throw.
template <typename F> PyObject *call(const Args &a, F &&enqueue) {
    c10::cuda::OptionalCUDAGuard guard;
    if (c10::cuda::current_device() != a.device) guard.set_index((c10::DeviceIndex)a.device);
    void *stream = (void *)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)a.device).stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = enqueue(stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

#define VS_FAST_CALL(name, count)                                                       \
    PyObject *name##_impl(Args &a);                                                     \
    PyObject *name(PyObject *, PyObject *const *argv, Py_ssize_t n) {                   \
        if (n != count) {                                                               \
            PyErr_SetString(PyExc_TypeError, #name ": wrong number of arguments");      \
            return nullptr;                                                             \
        }                                                                               \
        Args a(argv);                                                                   \
        try {                                                                           \
            return name##_impl(a);                                                      \
        } catch (const std::exception &e) {                                             \
            PyErr_SetString(PyExc_RuntimeError, e.what());                              \
            return nullptr;                                                             \
        }                                                                               \
    }                                                                                   \
    PyObject *name##_impl(Args &a)

// spmm(path, m_vec, V, k, n, row_indices, row_offsets, column_indices, values, rhs, out, batch, nonzeros_vec | None)
VS_FAST_CALL(spmm, 13) {
    const int path = a.integer(0), m_vec = a.integer(1), V = a.integer(2), k = a.integer(3), n = a.integer(4), batch = a.integer(11);
    const int64_t nnz = a.none(12) ? 0 : a.integer64(12);
    const int32_t *ri = a.index(5, m_vec), *ro = a.index(6, (int64_t)m_vec + 1), *ci = a.index(7, nnz);
    const at::Tensor *values = a.tensor(8), *rhs = a.tensor(9), *out = a.tensor(10);
    if (!a.ok) Py_RETURN_NONE;
    a.need(values, lead(values, 2, batch) * nnz * V);
    a.need(rhs, lead(rhs, 3, batch) * (int64_t)n * k);
    a.need(out, (int64_t)batch * m_vec * V * k);
    a.type(rhs, values->scalar_type());
    const int in_t = a.dtype(values), out_t = a.dtype(out);
    if (!a.ok) Py_RETURN_NONE;
    const void *pv = values->const_data_ptr(), *pr = rhs->const_data_ptr();
    void *po = out->mutable_data_ptr();
    int64_t sv = batch_stride(values, 2, batch);
    const int64_t sr = batch_stride(rhs, 3, batch), so = batch_stride(out, 3, batch);
    if (batch == 1) sv = (values->numel() + 7) / 8 * 8;   // no stride: how many values there are at most
    return call(a, [&](void *s) {
        return g_lib.spmm(path, in_t, out_t, m_vec, V, k, n, ri, ro, ci, pv, pr, po, batch, sv, sr, so, s);
    });
}

// spmm_t(m_vec, V, k, n, t_offsets, t_rows, t_src, values, rhs, out, nonzeros_vec | None)
VS_FAST_CALL(spmm_t, 11) {
    const int m_vec = a.integer(0), V = a.integer(1), k = a.integer(2), n = a.integer(3);
    const int64_t nnz = a.none(10) ? 0 : a.integer64(10);
    const int32_t *off = a.index(4, (int64_t)n + 1), *rows = a.index(5, nnz), *src = a.index(6, nnz);
    const at::Tensor *values = a.tensor(7), *rhs = a.tensor(8), *out = a.tensor(9);
    if (!a.ok || THPVariable_Unpack(a.argv[5]).numel() != THPVariable_Unpack(a.argv[6]).numel()) Py_RETURN_NONE;
    const int64_t lead_out = out->dim() == 3 ? out->size(0) : 1;
    if (lead_out > INT_MAX) Py_RETURN_NONE;
    const int batch = (int)lead_out;
    a.need(values, lead(values, 2, batch) * nnz * V);
    a.need(rhs, lead(rhs, 3, batch) * (int64_t)m_vec * V * k);
    a.need(out, (int64_t)batch * n * k);
    a.type(rhs, values->scalar_type());
    const int in_t = a.dtype(values), out_t = a.dtype(out);
    if (!a.ok) Py_RETURN_NONE;
    const void *pv = values->const_data_ptr(), *pr = rhs->const_data_ptr();
    void *po = out->mutable_data_ptr();
    const int64_t sv = batch_stride(values, 2, batch), sr = batch_stride(rhs, 3, batch), so = batch_stride(out, 3, batch);
    return call(a, [&](void *s) {
        return g_lib.spmm_t(in_t, out_t, m_vec, V, k, n, off, rows, src, pv, pr, po, batch, sv, sr, so, s);
    });
}

// sddmm(path, m_vec, k, n, nonzeros_vec, row_indices, row_offsets, col_indices, lhs, rhs, out, V, algorithm, batch)
VS_FAST_CALL(sddmm, 14) {
    const int path = a.integer(0), m_vec = a.integer(1), k = a.integer(2), n = a.integer(3), nnz = a.integer(4);
    const int V = a.integer(11), algorithm = a.integer(12), batch = a.integer(13);
    const int32_t *ri = a.index(5, m_vec), *ro = a.index(6, (int64_t)m_vec + 1), *ci = a.index(7, nnz);
    const at::Tensor *lhs = a.tensor(8), *rhs = a.tensor(9), *out = a.tensor(10);
    if (!a.ok) Py_RETURN_NONE;
    a.need(lhs, lead(lhs, 3, batch) * (int64_t)m_vec * V * k);
    a.need(rhs, lead(rhs, 3, batch) * (int64_t)n * k);
    a.need(out, (int64_t)batch * nnz * V);
    a.type(rhs, lhs->scalar_type());
    const int in_t = a.dtype(lhs), out_t = a.dtype(out);
    if (!a.ok) Py_RETURN_NONE;
    const void *pl = lhs->const_data_ptr(), *pr = rhs->const_data_ptr();
    void *po = out->mutable_data_ptr();
    const int64_t sl = batch_stride(lhs, 3, batch), sr = batch_stride(rhs, 3, batch), so = batch_stride(out, 2, batch);
    return call(a, [&](void *s) {
        return g_lib.sddmm(path, in_t, out_t, m_vec, k, n, nnz, ri, ro, ci, pl, pr, po, V, batch, sl, sr, so, s, algorithm);
    });
}

// Number of problems in a score array: [nnz] or [batch, nnz].  False if it cannot be a batch.
bool score_batch(const at::Tensor *t, int *batch) {
    const int64_t b = t->dim() == 2 ? t->size(0) : 1;
    *batch = (int)b;
    return b <= INT_MAX;
}

// softmax(m_vec, V, row_indices, row_offsets, scores, probs, scale)
VS_FAST_CALL(softmax, 7) {
    const int m_vec = a.integer(0), V = a.integer(1);
    const double scale = a.number(6);
    const int32_t *ri = a.index(2, 0), *ro = a.index(3, 0);
    const at::Tensor *scores = a.tensor(4), *probs = a.tensor(5);
    int batch = 1;
    if (!a.ok || !score_batch(scores, &batch)) Py_RETURN_NONE;
    a.type(probs, scores->scalar_type());
    const int t = a.dtype(scores);
    if (!a.ok) Py_RETURN_NONE;
    const void *in = scores->const_data_ptr();
    void *out = probs->mutable_data_ptr();
    const int64_t stride = batch_stride(scores, 2, batch);
    return call(a, [&](void *s) {
        return g_lib.softmax(t, m_vec, V, ri, ro, in, out, (float)scale, batch, stride, s);
    });
}

// softmax_backward(m_vec, V, row_offsets, probs, grad_probs, grad_scores, scale)
VS_FAST_CALL(softmax_backward, 7) {
    const int m_vec = a.integer(0), V = a.integer(1);
    const double scale = a.number(6);
    const int32_t *ro = a.index(2, 0);
    const at::Tensor *probs = a.tensor(3), *gp = a.tensor(4), *gs = a.tensor(5);
    int batch = 1;
    if (!a.ok || !score_batch(probs, &batch)) Py_RETURN_NONE;
    a.type(gp, probs->scalar_type());
    a.type(gs, probs->scalar_type());
    const int t = a.dtype(probs);
    if (!a.ok) Py_RETURN_NONE;
    const void *pp = probs->const_data_ptr(), *pg = gp->const_data_ptr();
    void *po = gs->mutable_data_ptr();
    const int64_t stride = batch_stride(probs, 2, batch);
    return call(a, [&](void *s) {
        return g_lib.softmax_backward(t, m_vec, V, ro, pp, pg, po, (float)scale, batch, stride, s);
    });
}

// attention(path, m_vec, V, n, d, nonzeros_vec, row_indices, row_offsets, col_indices, q, k, v, out, workspace, scale)
VS_FAST_CALL(attention, 15) {
    const int path = a.integer(0), m_vec = a.integer(1), V = a.integer(2), n = a.integer(3), d = a.integer(4), nnz = a.integer(5);
    const double scale = a.number(14);
    const int32_t *ri = a.index(6, 0), *ro = a.index(7, 0), *ci = a.index(8, nnz);
    const at::Tensor *t[5];
    for (int i = 0; i < 5; ++i) {
        t[i] = a.tensor(9 + i);
        a.type(t[i], at::kHalf);
    }
    if (!a.ok) Py_RETURN_NONE;
    const int64_t batch = t[0]->dim() == 3 ? t[0]->size(0) : 1;
    if (batch > INT_MAX) Py_RETURN_NONE;
    a.need(t[4], batch * nnz * V);
    if (!a.ok) Py_RETURN_NONE;
    const void *in[3];
    void *out[2];
    for (int i = 0; i < 3; ++i) in[i] = t[i]->const_data_ptr();
    for (int i = 0; i < 2; ++i) out[i] = t[3 + i]->mutable_data_ptr();
    return call(a, [&](void *s) {
        return g_lib.attention(path, m_vec, V, n, d, nnz, ri, ro, ci, in[0], in[1], in[2], out[0], out[1], (float)scale, (int)batch, s);
    });
}

// attention_backward(path, m_vec, V, n, d, nonzeros_vec, row_indices, row_offsets, col_indices, t_offsets, t_rows, t_src,
//                    q, k, v, grad_out, grad_q, grad_k, grad_v, probs_workspace, grad_workspace, scale)
VS_FAST_CALL(attention_backward, 22) {
    const int path = a.integer(0), m_vec = a.integer(1), V = a.integer(2), n = a.integer(3), d = a.integer(4), nnz = a.integer(5);
    const double scale = a.number(21);
    const int32_t *ri = a.index(6, 0), *ro = a.index(7, 0), *ci = a.index(8, nnz);
    const int32_t *off = a.index(9, 0), *rows = a.index(10, nnz), *src = a.index(11, nnz);
    const at::Tensor *t[9];
    for (int i = 0; i < 9; ++i) {
        t[i] = a.tensor(12 + i);
        a.type(t[i], at::kHalf);
    }
    if (!a.ok) Py_RETURN_NONE;
    const int64_t batch = t[0]->dim() == 3 ? t[0]->size(0) : 1;
    if (batch > INT_MAX) Py_RETURN_NONE;
    a.need(t[7], batch * nnz * V);
    a.need(t[8], batch * nnz * V);
    if (!a.ok) Py_RETURN_NONE;
    const void *in[4];
    void *out[5];
    for (int i = 0; i < 4; ++i) in[i] = t[i]->const_data_ptr();
    for (int i = 0; i < 5; ++i) out[i] = t[4 + i]->mutable_data_ptr();
    return call(a, [&](void *s) {
        return g_lib.attention_backward(path, m_vec, V, n, d, nnz, ri, ro, ci, off, rows, src, in[0], in[1], in[2], in[3], out[0],
                                        out[1], out[2], out[3], out[4], (float)scale, (int)batch, s);
    });
}

// ---- autograd -------------------------------------------------------------------------------------------------
// The two differentiable operators of torch_ops.py as nodes of torch's own graph.  An empty torch.autograd.Function costs the host 56 us of a
// forward and backward pass; with the Python around the operators a training step of a small layer took 101 us, of which the GPU
// worked 24; with these nodes 67, an attention layer's 111 -> 83.
// A node keeps what the Python function keeps (saved variables, so hooks on saved tensors, version checks and freeing a graph work as there) and the mask.
// Where something listens or a derivative of the backward pass is wanted, the node calls the Python function's backward instead.

PyObject *g_backward;   // torch_ops: (which, mask, path, scale, saved tensors, gradient, wanted) -> gradients

bool plain(const at::Tensor &t) {
    return t.defined() && t.is_cuda() && t.scalar_type() == at::kHalf && t.layout() == at::kStrided && t.has_storage() &&
           !t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                                     c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative}));
}
// Whether modes of either kind, a tracer or a profiler listen to this thread's operators (torch_ops._through asks the same).
bool heard() {
    return c10::impl::TorchDispatchModeTLS::stack_len() != 0 || at::impl::PythonTorchFunctionTLS::stack_len() != 0 || torch::jit::tracer::isTracing() ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::PreDispatch) || at::hasCallbacks();
}
template <typename F> int enqueue_on(const at::Tensor &t, F &&f) { return f((void *)c10::cuda::getCurrentCUDAStream(t.get_device()).stream()); }

struct MaskNode : torch::autograd::Node {
    int which = 0;   // 0: the product, 1: attention
    int path = 0, m_vec = 0, V = 0, n = 0, nnz = 0;
    double scale = 0.0;
    at::Tensor ri, ro, ci, off, rows, src;
    std::vector<torch::autograd::SavedVariable> saved;
    std::unique_ptr<c10::SafePyObject> mask;
    std::mutex lock;

    std::string name() const override { return which ? "FixedMaskAttentionBackward" : "SparseDenseProductBackward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> guard(lock);
        for (auto &x : saved) x.reset_data();
    }

    // As torch_ops does it, for everything that is not a plain pass over plain tensors.
    torch::autograd::variable_list in_python(const std::vector<at::Tensor> &kept, const at::Tensor &grad) {
        PyGILState_STATE gil = PyGILState_Ensure();
        torch::autograd::variable_list grads(num_outputs());
        PyObject *k = PyTuple_New((Py_ssize_t)kept.size()), *wanted = PyTuple_New((Py_ssize_t)kept.size()), *g = THPVariable_Wrap(grad);
        for (size_t i = 0; i < kept.size(); ++i) {
            PyTuple_SET_ITEM(k, (Py_ssize_t)i, THPVariable_Wrap(kept[i]));
            PyTuple_SET_ITEM(wanted, (Py_ssize_t)i, PyBool_FromLong(task_should_compute_output(i)));
        }
        PyObject *r = PyObject_CallFunction(g_backward, "iOidOOO", which, mask->ptr(getPyInterpreter()), path, scale, k, g, wanted);
        Py_DECREF(k);
        Py_DECREF(wanted);
        Py_DECREF(g);
        bool ok = r && PyTuple_Check(r) && PyTuple_GET_SIZE(r) == (Py_ssize_t)kept.size();
        for (size_t i = 0; ok && i < kept.size(); ++i) {
            PyObject *x = PyTuple_GET_ITEM(r, (Py_ssize_t)i);
            if (x != Py_None) {
                if (THPVariable_Check(x)) grads[i] = THPVariable_Unpack(x);
                else ok = false;
            }
        }
        Py_XDECREF(r);
        if (!ok) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "a gradient is not a tensor");
            python_error e;
            e.persist();   // keeps the Python error, of the same type, for the thread that asked for the gradients
            PyGILState_Release(gil);
            throw std::move(e);
        }
        PyGILState_Release(gil);
        return grads;
    }

    torch::autograd::variable_list apply(torch::autograd::variable_list &&in) override {
        std::vector<at::Tensor> kept;
        {
            std::lock_guard<std::mutex> guard(lock);
            for (auto &x : saved) kept.push_back(x.unpack(shared_from_this()));
        }
        const at::Tensor given = in[0].defined() ? in[0] : input_metadata(0).zeros_like();   // no gradient counts as zeros, as in the Python function
        bool fast = !c10::GradMode::is_enabled() && !heard() && plain(given);
        for (const at::Tensor &t : kept) fast = fast && plain(t) && t.is_contiguous() && t.device() == given.device();
        if (!fast) return in_python(kept, given);
        c10::cuda::CUDAGuard guard(given.device());
        const at::Tensor grad = given.contiguous();
        torch::autograd::variable_list out(num_outputs());
        return (which ? attention(kept, grad, out) : product(kept, grad, out)) == 0 ? out : in_python(kept, given);
    }

    int product(const std::vector<at::Tensor> &kept, const at::Tensor &grad, torch::autograd::variable_list &out) {
        const at::Tensor &values = kept[0], &b = kept[1];
        const int batch = b.dim() == 3 ? (int)b.size(0) : 1, k = (int)b.size(-1);
        const int64_t sg = batch > 1 ? grad.stride(0) : 0, sb = batch > 1 ? b.stride(0) : 0, sv = batch > 1 && values.dim() == 2 ? values.stride(0) : 0;
        int rc = 0;
        if (task_should_compute_output(1)) {
            out[1] = at::empty_like(b);
            rc = enqueue_on(b, [&](void *s) {
                return g_lib.spmm_t(VS_F16, VS_F16, m_vec, V, k, n, off.const_data_ptr<int32_t>(), rows.const_data_ptr<int32_t>(), src.const_data_ptr<int32_t>(),
                                    values.const_data_ptr(), grad.const_data_ptr(), out[1].mutable_data_ptr(), batch, sv, sg, sb, s);
            });
        }
        if (rc == 0 && task_should_compute_output(0)) {
            const int64_t per = (int64_t)nnz * V;
            at::Tensor g = b.dim() == 3 ? at::empty({batch, per}, b.options()) : at::empty({per}, b.options());
            rc = enqueue_on(b, [&](void *s) {
                return g_lib.sddmm(path, VS_F16, VS_F16, m_vec, k, n, nnz, ri.const_data_ptr<int32_t>(), ro.const_data_ptr<int32_t>(), ci.const_data_ptr<int32_t>(),
                                   grad.const_data_ptr(), b.const_data_ptr(), g.mutable_data_ptr(), V, batch, sg, sb, batch > 1 ? per : 0, s, 1);
            });
            out[0] = g.dim() == 2 && values.dim() == 1 ? g.sum(0) : g;
        }
        return rc;
    }

    int attention(const std::vector<at::Tensor> &kept, const at::Tensor &grad, torch::autograd::variable_list &out) {
        const at::Tensor &q = kept[0], &k = kept[1], &v = kept[2];
        const int batch = q.dim() == 3 ? (int)q.size(0) : 1;
        at::Tensor p = at::empty({batch, (int64_t)nnz * V}, q.options()), g = at::empty({batch, (int64_t)nnz * V}, q.options());
        out = {at::empty_like(q), at::empty_like(k), at::empty_like(v)};
        return enqueue_on(q, [&](void *s) {
            return g_lib.attention_backward(path, m_vec, V, n, (int)k.size(-1), nnz, ri.const_data_ptr<int32_t>(), ro.const_data_ptr<int32_t>(),
                                            ci.const_data_ptr<int32_t>(), off.const_data_ptr<int32_t>(), rows.const_data_ptr<int32_t>(), src.const_data_ptr<int32_t>(),
                                            q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), grad.const_data_ptr(), out[0].mutable_data_ptr(),
                                            out[1].mutable_data_ptr(), out[2].mutable_data_ptr(), p.mutable_data_ptr(), g.mutable_data_ptr(), (float)scale, batch, s);
        });
    }
};

// differentiable(which, path, m_vec, V, n, nonzeros_vec, scale, row_indices, row_offsets, col_indices, t_offsets, t_rows, t_src, mask, operands ...):
// the operator on plain contiguous fp16 CUDA tensors, recorded in torch's graph; None where something is not as it takes it, and where
// the library refuses the call.
PyObject *differentiable(PyObject *, PyObject *const *argv, Py_ssize_t n_args) {
    Args a(argv);
    try {
        const int which = n_args > 0 ? a.integer(0) : 0;
        if (n_args != (which ? 17 : 16) || !g_backward) Py_RETURN_NONE;
        const int path = a.integer(1), m_vec = a.integer(2), V = a.integer(3), n = a.integer(4), nnz = a.integer(5), operands = which ? 3 : 2;
        const double scale = a.number(6);
        const int32_t *ri = a.index(7, m_vec), *ro = a.index(8, (int64_t)m_vec + 1), *ci = a.index(9, nnz);
        a.index(10, (int64_t)n + 1), a.index(11, nnz), a.index(12, nnz);
        const at::Tensor *t[3];
        for (int i = 0; i < operands; ++i) {
            t[i] = a.tensor(14 + i);
            if (!a.ok || !plain(*t[i]) || t[i]->_fw_grad(0).defined()) Py_RETURN_NONE;
        }
        if (!a.ok || m_vec < 1 || n < 1 || nnz < 1 || V < 1 || t[1]->dim() < 2 || t[1]->dim() > 3) Py_RETURN_NONE;
        const int64_t k = t[1]->size(-1), batch = t[1]->dim() == 3 ? t[1]->size(0) : 1, m = (int64_t)m_vec * V;
        if (batch < 1 || batch > INT_MAX || k < 1 || k > INT_MAX || m > INT_MAX || t[1]->size(-2) != n) Py_RETURN_NONE;
        if (which) {
            for (int i = 0; i < 3; ++i)
                if (t[i]->dim() != t[1]->dim() || t[i]->size(-1) != k || t[i]->size(-2) != (i ? n : m) || (t[i]->dim() == 3 && t[i]->size(0) != batch)) Py_RETURN_NONE;
        } else if (!(t[0]->dim() == 1 || (t[0]->dim() == 2 && t[1]->dim() == 3 && t[0]->size(0) == batch)) || t[0]->size(-1) != (int64_t)nnz * V) {
            Py_RETURN_NONE;
        }
        c10::cuda::OptionalCUDAGuard guard;
        if (c10::cuda::current_device() != a.device) guard.set_index((c10::DeviceIndex)a.device);
        void *stream = (void *)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)a.device).stream();
        at::Tensor out;
        int rc;
        if (which) {
            out = at::empty(t[0]->sizes(), t[0]->options());
            at::Tensor ws = at::empty({batch, (int64_t)nnz * V}, t[0]->options());
            const void *pq = t[0]->const_data_ptr(), *pk = t[1]->const_data_ptr(), *pv = t[2]->const_data_ptr();
            void *po = out.mutable_data_ptr(), *pw = ws.mutable_data_ptr();
            Py_BEGIN_ALLOW_THREADS
            rc = g_lib.attention(path, m_vec, V, n, (int)k, nnz, ri, ro, ci, pq, pk, pv, po, pw, (float)scale, (int)batch, stream);
            Py_END_ALLOW_THREADS
        } else {
            out = t[1]->dim() == 3 ? at::empty({batch, m, k}, t[1]->options()) : at::empty({m, k}, t[1]->options());
            const void *pv = t[0]->const_data_ptr(), *pb = t[1]->const_data_ptr();
            void *po = out.mutable_data_ptr();
            const int64_t sv = batch == 1 ? (t[0]->numel() + 7) / 8 * 8 : t[0]->dim() == 2 ? t[0]->stride(0) : 0;
            const int64_t sb = batch > 1 ? t[1]->stride(0) : 0, so = batch > 1 ? m * k : 0;
            Py_BEGIN_ALLOW_THREADS
            rc = g_lib.spmm(path, VS_F16, VS_F16, m_vec, V, (int)k, n, ri, ro, ci, pv, pb, po, (int)batch, sv, sb, so, stream);
            Py_END_ALLOW_THREADS
        }
        if (rc != 0) Py_RETURN_NONE;
        bool wanted = false;
        for (int i = 0; i < operands; ++i) wanted = wanted || t[i]->requires_grad();
        if (wanted && c10::GradMode::is_enabled()) {
            auto node = std::shared_ptr<MaskNode>(new MaskNode(), torch::autograd::deleteNode);
            if (which) node->set_next_edges(torch::autograd::collect_next_edges(*t[0], *t[1], *t[2]));
            else node->set_next_edges(torch::autograd::collect_next_edges(*t[0], *t[1]));
            node->which = which; node->path = path; node->m_vec = m_vec; node->V = V; node->n = n; node->nnz = nnz; node->scale = scale;
            at::Tensor *const kept[6] = {&node->ri, &node->ro, &node->ci, &node->off, &node->rows, &node->src};
            for (int i = 0; i < 6; ++i) *kept[i] = THPVariable_Unpack(argv[7 + i]);
            for (int i = 0; i < operands; ++i) node->saved.emplace_back(*t[i], false);
            Py_INCREF(argv[13]);
            node->mask = std::make_unique<c10::SafePyObject>(argv[13], getPyInterpreter());
            torch::autograd::set_history(out, node);
        }
        return THPVariable_Wrap(std::move(out));
    } catch (python_error &e) {
        e.restore();
        return nullptr;
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyObject *bind_backward(PyObject *, PyObject *const *argv, Py_ssize_t n) {
    if (n != 1 || !PyCallable_Check(argv[0])) {
        PyErr_SetString(PyExc_TypeError, "bind_backward: a function");
        return nullptr;
    }
    Py_INCREF(argv[0]);
    Py_XSETREF(g_backward, argv[0]);
    Py_RETURN_NONE;
}

// bind(addresses): the library's functions in the order of struct Library
PyObject *bind(PyObject *, PyObject *const *argv, Py_ssize_t n) {
    constexpr Py_ssize_t kCount = sizeof(Library) / sizeof(void *);
    if (n != kCount) {
        PyErr_SetString(PyExc_TypeError, "bind: wrong number of addresses");
        return nullptr;
    }
    void **slot = reinterpret_cast<void **>(&g_lib);
    for (Py_ssize_t i = 0; i < n; ++i) {
        slot[i] = PyLong_AsVoidPtr(argv[i]);
        if (!slot[i]) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: null address");
            return nullptr;
        }
    }
    Py_RETURN_NONE;
}

#define VS_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(&name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {
    VS_METHOD(bind), VS_METHOD(spmm), VS_METHOD(spmm_t), VS_METHOD(sddmm), VS_METHOD(softmax), VS_METHOD(softmax_backward),
    VS_METHOD(attention), VS_METHOD(attention_backward), VS_METHOD(differentiable), VS_METHOD(bind_backward), {nullptr, nullptr, 0, nullptr},
};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_binding", "torch tensors to the C ABI of libvsparse_b200", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() { return PyModule_Create(&g_module); }
