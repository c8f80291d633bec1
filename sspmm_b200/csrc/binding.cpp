// The calls of ops.py that a program makes once per product, without the interpreter's share of them: checking four to six
// tensors, allocating the result, asking for device and stream and marshalling eighteen arguments took ops.sspmm 14.5 us a call,
// for a kernel of 5.2 (512 x 512, N = 256); with one extension call it is 6.6, launch included.
//
// Each function takes the ordinary case and nothing else.  None means that the operands are not plain (other types or layouts, host
// tensors, subclasses, wrapped tensors of a function transform, an active torch mode, ...); the caller then goes through the checks
// in Python, which accept or refuse as they always have.  An int is an error code of the library.
#define PY_SSIZE_T_CLEAN
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContextLight.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "../../include/sspmm_b200.h"

namespace {

bool modes_active() {
    return at::impl::PythonTorchFunctionTLS::stack_len() > 0 || c10::impl::TorchDispatchModeTLS::any_modes_set();
}

// A dense CUDA tensor of this type with nothing on it but autograd's keys, contiguous; null: not one.
const at::Tensor* plain(PyObject* o, at::ScalarType type) {
    static const c10::DispatchKeySet allowed =
        c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
        c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) | c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA);
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.scalar_type() != type || !t.has_storage() || !allowed.isSupersetOf(t.key_set()) || !t.is_contiguous())
        return nullptr;
    return &t;
}

bool small_int(PyObject* o, long lo, long hi, long* v) {
    if (!PyLong_CheckExact(o)) return false;
    int over = 0;
    *v = PyLong_AsLongAndOverflow(o, &over);
    return over == 0 && *v >= lo && *v <= hi;
}

void* stream_of(c10::DeviceIndex device) { return static_cast<void*>(at::cuda::getCurrentCUDAStream(device).stream()); }

// f(stream) on the device and its current stream, without the interpreter lock.
template <typename F>
int launch(c10::DeviceIndex device, F&& f) {
    int rc;
    const c10::cuda::OptionalCUDAGuard guard(device);
    void* const stream = stream_of(device);
    Py_BEGIN_ALLOW_THREADS
    rc = f(stream);
    Py_END_ALLOW_THREADS
    return rc;
}

PyObject* result(int rc, const at::Tensor& out) {
    if (rc != 0) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
}

// Runs a body that may throw (allocation, device guard): the exception becomes the Python one torch would raise.
template <typename F>
PyObject* guarded(F&& f) {
    HANDLE_TH_ERRORS
    return f();
    END_HANDLE_TH_ERRORS
}

// sspmm(row_offsets, column_indices, values, rhs, vec_length, bias, row_indices, out_dtype)
PyObject* py_sspmm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long V;
        if (n != 8 || modes_active() || !small_int(a[4], 1, 1 << 20, &V) || !THPDtype_Check(a[7])) Py_RETURN_NONE;
        const at::ScalarType type = reinterpret_cast<THPDtype*>(a[7])->scalar_type;
        if (type != at::kHalf && type != at::kFloat) Py_RETURN_NONE;
        const at::Tensor *ptr = plain(a[0], at::kInt), *col = plain(a[1], at::kInt), *val = plain(a[2], at::kHalf), *rhs = plain(a[3], at::kHalf);
        const at::Tensor* bias = a[5] == Py_None ? nullptr : plain(a[5], at::kHalf);
        const at::Tensor* order = a[6] == Py_None ? nullptr : plain(a[6], at::kInt);
        if (!ptr || !col || !val || !rhs || (a[5] != Py_None && !bias) || (a[6] != Py_None && !order) || rhs->dim() != 2) Py_RETURN_NONE;
        const int64_t m_vec = ptr->numel() - 1, K = rhs->size(0), N = rhs->size(1), most = 0x7fffffff;
        if (m_vec < 0 || m_vec > most / V || K > most || N > most) Py_RETURN_NONE;
        if (bias && (bias->numel() != m_vec * V || bias->device() != rhs->device())) Py_RETURN_NONE;
        at::Tensor out = at::empty({m_vec * V, N}, rhs->options().dtype(type).requires_grad(false));
        return result(launch(rhs->get_device(), [&](void* st) {
            return sspmm_counted((int)m_vec, (int)V, (int)N, (int)K, 1, col->numel(), order ? static_cast<const int*>(order->data_ptr()) : nullptr,
                                 static_cast<const int*>(ptr->data_ptr()), static_cast<const int*>(col->data_ptr()), val->data_ptr(), 0,
                                 rhs->data_ptr(), 0, bias ? bias->data_ptr() : nullptr, out.data_ptr(), 0, type == at::kHalf, st);
        }), out);
    });
}

// stacked(row_offsets of each piece, row_indices of each, where the pieces' vectors end, column_indices, values, rhs, vec_length, bias)
PyObject* py_stacked(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        constexpr Py_ssize_t kMost = 4;
        long V;
        if (n != 8 || modes_active() || !small_int(a[6], 1, 1 << 20, &V) || !PyList_CheckExact(a[0]) || !PyList_CheckExact(a[1]) ||
            !PyList_CheckExact(a[2]))
            Py_RETURN_NONE;
        const Py_ssize_t pieces = PyList_GET_SIZE(a[0]);
        if (pieces < 1 || pieces > kMost || PyList_GET_SIZE(a[1]) != pieces || PyList_GET_SIZE(a[2]) != pieces) Py_RETURN_NONE;
        const at::Tensor *col = plain(a[3], at::kInt), *val = plain(a[4], at::kHalf), *rhs = plain(a[5], at::kHalf), *bias = plain(a[7], at::kHalf);
        if (!col || !val || !rhs || !bias || rhs->dim() != 2) Py_RETURN_NONE;
        const int *offsets[kMost], *orders[kMost];
        int64_t nvec[kMost], m_vec = 0;
        long before = 0;
        for (Py_ssize_t i = 0; i < pieces; ++i) {
            const at::Tensor *ptr = plain(PyList_GET_ITEM(a[0], i), at::kInt), *order = plain(PyList_GET_ITEM(a[1], i), at::kInt);
            long end;
            if (!ptr || !order || ptr->device() != rhs->device() || order->device() != rhs->device() ||
                !small_int(PyList_GET_ITEM(a[2], i), before, 0x7fffffff, &end))
                Py_RETURN_NONE;
            if (i == 0) m_vec = ptr->numel() - 1;
            if (ptr->numel() - 1 != m_vec || order->numel() != m_vec) Py_RETURN_NONE;
            offsets[i] = static_cast<const int*>(ptr->data_ptr());
            orders[i] = static_cast<const int*>(order->data_ptr());
            nvec[i] = end - before;
            before = end;
        }
        const int64_t K = rhs->size(0), N = rhs->size(1), most = 0x7fffffff;
        if (m_vec < 1 || m_vec > most / V / pieces || K > most || N > most || col->numel() != before || val->numel() != before * V ||
            bias->numel() != pieces * m_vec * V || bias->device() != rhs->device() || col->device() != rhs->device() || val->device() != rhs->device())
            Py_RETURN_NONE;
        at::Tensor out = at::empty({pieces * m_vec * V, N}, rhs->options().requires_grad(false));
        int taken = 0;
        const int rc = launch(rhs->get_device(), [&](void* st) {
            return sspmm_stacked((int)pieces, (int)m_vec, (int)V, (int)N, (int)K, nvec, orders, offsets, static_cast<const int*>(col->data_ptr()),
                                 val->data_ptr(), rhs->data_ptr(), bias->data_ptr(), out.data_ptr(), 1, st, &taken);
        });
        if (rc == 0 && !taken) Py_RETURN_NONE;
        return result(rc, out);
    });
}

// bspmm(row_indices, row_offsets, column_indices, values, rhs_matrix, vec_length)
PyObject* py_bspmm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long V;
        if (n != 6 || modes_active() || !small_int(a[5], 1, 1 << 20, &V)) Py_RETURN_NONE;
        const at::Tensor *order = plain(a[0], at::kInt), *ptr = plain(a[1], at::kInt), *col = plain(a[2], at::kInt), *val = plain(a[3], at::kHalf),
                         *rhs = plain(a[4], at::kHalf);
        if (!order || !ptr || !col || !val || !rhs || rhs->dim() < 2) Py_RETURN_NONE;
        const int64_t m_vec = ptr->numel() - 1, K = rhs->size(-2), N = rhs->size(-1), most = 0x7fffffff;
        if (m_vec < 0 || m_vec > most / V || K > most || N > most || K * N == 0) Py_RETURN_NONE;
        const int64_t batch = rhs->numel() / (K * N), nnz = col->numel() * V;
        if (batch > most) Py_RETURN_NONE;
        const bool shared = val->numel() == nnz && batch != 1;
        at::Tensor out = at::empty({batch, m_vec * V, N}, rhs->options().requires_grad(false));
        return result(launch(rhs->get_device(), [&](void* st) {
            return sspmm_counted((int)m_vec, (int)V, (int)N, (int)K, (int)batch, col->numel(), static_cast<const int*>(order->data_ptr()),
                                 static_cast<const int*>(ptr->data_ptr()), static_cast<const int*>(col->data_ptr()), val->data_ptr(), shared ? 0 : nnz,
                                 rhs->data_ptr(), K * N, nullptr, out.data_ptr(), m_vec * V * N, 1, st);
        }), out);
    });
}

// planned(handle, rows of the output, K, values, rhs, out_dtype)
PyObject* py_planned(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long rows, K;
        if (n != 6 || modes_active() || !PyLong_CheckExact(a[0]) || !small_int(a[1], 0, 0x7fffffff, &rows) || !small_int(a[2], 0, 0x7fffffff, &K) ||
            !THPDtype_Check(a[5]))
            Py_RETURN_NONE;
        const at::ScalarType type = reinterpret_cast<THPDtype*>(a[5])->scalar_type;
        if (type != at::kHalf && type != at::kFloat) Py_RETURN_NONE;
        const at::Tensor *val = plain(a[3], at::kHalf), *rhs = plain(a[4], at::kHalf);
        if (!val || !rhs || rhs->dim() != 2 || rhs->size(0) != K || rhs->size(1) > 0x7fffffff) Py_RETURN_NONE;
        const sspmm_plan* plan = static_cast<const sspmm_plan*>(PyLong_AsVoidPtr(a[0]));
        if (!plan) Py_RETURN_NONE;
        at::Tensor out = at::empty({rows, rhs->size(1)}, rhs->options().dtype(type).requires_grad(false));
        return result(launch(rhs->get_device(), [&](void* st) {
            return sspmm_planned(plan, val->data_ptr(), rhs->data_ptr(), out.data_ptr(), (int)rhs->size(1), type == at::kHalf, st);
        }), out);
    });
}

// sspmm_sum(row_offsets, column_indices, values, rhs, vec_length, bias, row_indices, add)
PyObject* py_sspmm_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long V;
        if (n != 8 || modes_active() || !small_int(a[4], 1, 1 << 20, &V)) Py_RETURN_NONE;
        const at::Tensor *ptr = plain(a[0], at::kInt), *col = plain(a[1], at::kInt), *val = plain(a[2], at::kHalf), *rhs = plain(a[3], at::kHalf),
                         *bias = plain(a[5], at::kHalf), *order = plain(a[6], at::kInt), *add = plain(a[7], at::kHalf);
        if (!ptr || !col || !val || !rhs || !bias || !order || !add || rhs->dim() != 2) Py_RETURN_NONE;
        const int64_t m_vec = ptr->numel() - 1, K = rhs->size(0), N = rhs->size(1), most = 0x7fffffff;
        if (m_vec < 0 || m_vec > most / V || K > most || N > most || bias->numel() != m_vec * V || add->dim() != 2 || add->size(0) != m_vec * V ||
            add->size(1) != N)
            Py_RETURN_NONE;
        for (const at::Tensor* t : {ptr, col, val, bias, order, add})
            if (t->device() != rhs->device()) Py_RETURN_NONE;
        at::Tensor out = at::empty({m_vec * V, N}, rhs->options().requires_grad(false));
        int taken = 0;
        const int rc = launch(rhs->get_device(), [&](void* st) {
            return sspmm_counted_sum((int)m_vec, (int)V, (int)N, (int)K, col->numel(), static_cast<const int*>(order->data_ptr()),
                                     static_cast<const int*>(ptr->data_ptr()), static_cast<const int*>(col->data_ptr()), val->data_ptr(), rhs->data_ptr(),
                                     bias->data_ptr(), add->data_ptr(), out.data_ptr(), st, &taken);
        });
        if (rc == 0 && !taken) Py_RETURN_NONE;
        return result(rc, out);
    });
}

// dense_copies([(row_offsets of each piece, where the pieces' vectors end, column_indices, values, vec_length, K), ...], N, x, gamma, beta, eps)
//   -> a copy [K, rows] per operand, or None where the product does not work on one, and then LayerNorm of x where there is a copy (x may be
//   None: without it; the caller has compared its operands); None: not operands for it
PyObject* py_dense_copies(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        constexpr Py_ssize_t kMost = 8, kPieces = 4;
        long N;
        if (n != 6 || modes_active() || !PyList_CheckExact(a[0]) || !small_int(a[1], 1, 0x7fffffff, &N) || !PyFloat_Check(a[5])) Py_RETURN_NONE;
        const at::Tensor *x = a[2] == Py_None ? nullptr : plain(a[2], at::kHalf), *gamma = x ? plain(a[3], at::kHalf) : nullptr,
                         *beta = x ? plain(a[4], at::kHalf) : nullptr;
        if (a[2] != Py_None && (!x || !gamma || !beta || x->dim() != 2)) Py_RETURN_NONE;
        const Py_ssize_t count = PyList_GET_SIZE(a[0]);
        if (count < 1 || count > kMost) Py_RETURN_NONE;
        sspmm_dense_operand op[kMost];
        const int* offsets[kMost][kPieces];
        int64_t nvec[kMost][kPieces], at[kMost], bytes = 0;
        const at::Tensor* first = nullptr;
        for (Py_ssize_t k = 0; k < count; ++k) {
            PyObject* const t = PyList_GET_ITEM(a[0], k);
            if (!PyTuple_CheckExact(t) || PyTuple_GET_SIZE(t) != 6) Py_RETURN_NONE;
            PyObject *ptrs = PyTuple_GET_ITEM(t, 0), *ends = PyTuple_GET_ITEM(t, 1);
            const at::Tensor *col = plain(PyTuple_GET_ITEM(t, 2), at::kInt), *val = plain(PyTuple_GET_ITEM(t, 3), at::kHalf);
            long V, K, before = 0;
            if (!PyList_CheckExact(ptrs) || !PyList_CheckExact(ends) || !col || !val || !small_int(PyTuple_GET_ITEM(t, 4), 8, 16, &V) ||
                !small_int(PyTuple_GET_ITEM(t, 5), 1, 0x7fffffff, &K))
                Py_RETURN_NONE;
            const Py_ssize_t pieces = PyList_GET_SIZE(ptrs);
            if (pieces < 1 || pieces > kPieces || PyList_GET_SIZE(ends) != pieces) Py_RETURN_NONE;
            if (!first) first = col;
            if (col->device() != first->device() || val->device() != first->device()) Py_RETURN_NONE;
            int64_t m_vec = 0;
            for (Py_ssize_t i = 0; i < pieces; ++i) {
                const at::Tensor* ptr = plain(PyList_GET_ITEM(ptrs, i), at::kInt);
                long end;
                if (!ptr || ptr->device() != first->device() || !small_int(PyList_GET_ITEM(ends, i), before, 0x7fffffff, &end)) Py_RETURN_NONE;
                if (i == 0) m_vec = ptr->numel() - 1;
                if (ptr->numel() - 1 != m_vec || m_vec < 1 || m_vec > 0x7fffffff / V / pieces) Py_RETURN_NONE;
                offsets[k][i] = static_cast<const int*>(ptr->data_ptr());
                nvec[k][i] = end - before;
                before = end;
            }
            if (col->numel() != before || val->numel() != before * V) Py_RETURN_NONE;
            op[k] = sspmm_dense_operand{(int)pieces, (int)m_vec, (int)V, (int)K, nvec[k], offsets[k], static_cast<const int*>(col->data_ptr()), val->data_ptr()};
        }
        int rc = sspmm_dense_copies((int)count, op, (int)N, nullptr, at, &bytes, nullptr);
        if (rc != 0) return PyLong_FromLong(rc);
        at::Tensor room, norm;
        if (bytes) {
            room = at::empty({bytes / 2}, first->options().dtype(at::kHalf).requires_grad(false));
            if (x) norm = at::empty_like(*x, x->options().requires_grad(false));
            rc = launch(first->get_device(), [&](void* st) {
                return x ? sspmm_layer_norm_copies((int)count, op, (int)N, room.data_ptr(), (int)x->size(0), (int)x->size(1), x->data_ptr(),
                                                   gamma->data_ptr(), beta->data_ptr(), (float)PyFloat_AS_DOUBLE(a[5]), norm.data_ptr(), st)
                         : sspmm_dense_copies((int)count, op, (int)N, room.data_ptr(), at, &bytes, st);
            });
            if (rc != 0) return PyLong_FromLong(rc);
        }
        PyObject* const list = PyList_New(count + (norm.defined() ? 1 : 0));
        if (!list) return nullptr;
        for (Py_ssize_t k = 0; k < count; ++k) {
            PyObject* item = Py_None;
            if (at[k] >= 0) {
                const int64_t rows = (int64_t)op[k].pieces * op[k].m_vec * op[k].vec_length;
                item = THPVariable_Wrap(room.narrow(0, at[k] / 2, op[k].K * rows).view({op[k].K, rows}));
            } else {
                Py_INCREF(item);
            }
            PyList_SET_ITEM(list, k, item);
        }
        if (norm.defined()) PyList_SET_ITEM(list, count, THPVariable_Wrap(norm));
        return list;
    });
}

// of_copy(copy, rhs, vec_length, bias, add or None)
PyObject* py_of_copy(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long V;
        if (n != 5 || modes_active() || !small_int(a[2], 8, 16, &V)) Py_RETURN_NONE;
        const at::Tensor *copy = plain(a[0], at::kHalf), *rhs = plain(a[1], at::kHalf), *bias = plain(a[3], at::kHalf),
                         *add = a[4] == Py_None ? nullptr : plain(a[4], at::kHalf);
        if (!copy || !rhs || !bias || (a[4] != Py_None && !add) || copy->dim() != 2 || rhs->dim() != 2 || rhs->size(0) != copy->size(0)) Py_RETURN_NONE;
        const int64_t K = copy->size(0), rows = copy->size(1), N = rhs->size(1), most = 0x7fffffff;
        if (rows % V != 0 || rows > most || K > most || N > most || N % 8 != 0 || bias->numel() != rows || reinterpret_cast<uintptr_t>(rhs->data_ptr()) % 16 != 0 ||
            copy->device() != rhs->device() || bias->device() != rhs->device())
            Py_RETURN_NONE;
        if (add && (add->dim() != 2 || add->size(0) != rows || add->size(1) != N || add->device() != rhs->device() ||
                    reinterpret_cast<uintptr_t>(add->data_ptr()) % 16 != 0))
            Py_RETURN_NONE;
        at::Tensor out = at::empty({rows, N}, rhs->options().requires_grad(false));
        return result(launch(rhs->get_device(), [&](void* st) {
            return sspmm_of_copy((int)(rows / V), (int)V, (int)N, (int)K, copy->data_ptr(), rhs->data_ptr(), bias->data_ptr(),
                                 add ? add->data_ptr() : nullptr, out.data_ptr(), st);
        }), out);
    });
}

// group_run_sum(handle, rows of the output, bias or None, add) -> the sum, or None
PyObject* py_group_run_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long rows;
        if (n != 4 || modes_active() || !PyLong_CheckExact(a[0]) || !small_int(a[1], 0, 0x7fffffff, &rows)) Py_RETURN_NONE;
        const at::Tensor *add = plain(a[3], at::kHalf), *bias = a[2] == Py_None ? nullptr : plain(a[2], at::kHalf);
        sspmm_group* group = static_cast<sspmm_group*>(PyLong_AsVoidPtr(a[0]));
        if (!group || !add || add->dim() != 2 || add->size(0) != rows || (a[2] != Py_None && (!bias || bias->numel() != rows || bias->device() != add->device())))
            Py_RETURN_NONE;
        at::Tensor out = at::empty({rows, add->size(1)}, add->options().requires_grad(false));
        int taken = 0;
        const int rc = launch(add->get_device(), [&](void* st) { return sspmm_group_run_sum(group, bias ? bias->data_ptr() : nullptr, add->data_ptr(), out.data_ptr(), st, &taken); });
        if (rc == 0 && !taken) Py_RETURN_NONE;
        return result(rc, out);
    });
}

// group_run(handle, device index) -> error code
PyObject* py_group_run(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long device;
        if (n != 2 || !PyLong_CheckExact(a[0]) || !small_int(a[1], 0, 127, &device)) {
            PyErr_SetString(PyExc_TypeError, "group_run(handle, device index)");
            return nullptr;
        }
        sspmm_group* group = static_cast<sspmm_group*>(PyLong_AsVoidPtr(a[0]));
        return PyLong_FromLong(launch((c10::DeviceIndex)device, [&](void* st) { return sspmm_group_run(group, st); }));
    });
}

// same_plain(tensors...): contiguous fp16 tensors on one GPU, 16-byte aligned, outside autograd (see encoder._plain)
PyObject* py_same_plain(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const at::Tensor* first = nullptr;
    for (Py_ssize_t i = 0; i < n; ++i) {
        const at::Tensor* t = plain(a[i], at::kHalf);
        if (!t || (first && t->get_device() != first->get_device()) || reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 != 0 ||
            (t->requires_grad() && c10::GradMode::is_enabled()))
            Py_RETURN_FALSE;
        if (!first) first = t;
    }
    if (!first) Py_RETURN_FALSE;
    Py_RETURN_TRUE;
}

void* address(PyObject* o) { return o == Py_None ? nullptr : THPVariable_Unpack(o).data_ptr(); }
bool on_gpu(PyObject* o) { return THPVariable_Check(o) && THPVariable_Unpack(o).is_cuda(); }
bool tensors_or_none(PyObject* const* a, Py_ssize_t n) {
    for (Py_ssize_t i = 0; i < n; ++i)
        if (a[i] != Py_None && !THPVariable_Check(a[i])) return false;
    return true;
}

// layer_norm_fm(x, gamma, beta, eps, out, add, sum_out, bias), attention_fm(q, k, v, heads, batch, seq, out, bias_q, bias_v) and
// add_bias_fm(x, bias, add, out): for a caller that has compared the operands; -> error code
PyObject* py_layer_norm_fm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 8 || !PyFloat_Check(a[3]) || !on_gpu(a[0]) || !tensors_or_none(a + 1, 2) || !tensors_or_none(a + 4, 4)) Py_RETURN_NONE;
        const at::Tensor& x = THPVariable_Unpack(a[0]);
        return PyLong_FromLong(launch(x.get_device(), [&](void* st) {
            return sspmm_layer_norm_fm((int)x.size(0), (int)x.size(1), x.data_ptr(), address(a[7]), address(a[5]), address(a[6]), address(a[1]),
                                       address(a[2]), (float)PyFloat_AS_DOUBLE(a[3]), address(a[4]), st);
        }));
    });
}
PyObject* py_attention_fm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long heads, batch, seq;
        if (n != 9 || !on_gpu(a[0]) || !tensors_or_none(a + 1, 2) || !tensors_or_none(a + 6, 3) || !small_int(a[3], 0, 0x7fffffff, &heads) ||
            !small_int(a[4], 0, 0x7fffffff, &batch) || !small_int(a[5], 0, 0x7fffffff, &seq))
            Py_RETURN_NONE;
        const at::Tensor& q = THPVariable_Unpack(a[0]);
        return PyLong_FromLong(launch(q.get_device(), [&](void* st) {
            return sspmm_attention_fm((int)heads, 64, (int)batch, (int)seq, q.data_ptr(), address(a[1]), address(a[2]), address(a[7]), address(a[8]),
                                      address(a[6]), st);
        }));
    });
}
PyObject* py_add_bias_fm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 4 || !on_gpu(a[0]) || !tensors_or_none(a + 1, 3)) Py_RETURN_NONE;
        const at::Tensor& x = THPVariable_Unpack(a[0]);
        return PyLong_FromLong(launch(x.get_device(), [&](void* st) {
            return sspmm_add_bias_fm((int)x.size(0), (int)x.size(1), x.data_ptr(), address(a[1]), address(a[2]), address(a[3]), st);
        }));
    });
}

// svc(row_ptr, col_idx, values or None, M, K, vec_length) -> (vec_ptr, vec_col, vec_values or None, replayed rows)
PyObject* py_svc(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long M, K, V;
        if (n != 6 || modes_active() || !small_int(a[3], 0, 0x7ffffff0, &M) || !small_int(a[4], 0, 0x7fffffff, &K) || !small_int(a[5], 1, 1 << 20, &V))
            Py_RETURN_NONE;
        const at::Tensor *ptr = plain(a[0], at::kInt), *col = plain(a[1], at::kInt), *val = a[2] == Py_None ? nullptr : plain(a[2], at::kHalf);
        if (!ptr || !col || (a[2] != Py_None && !val)) Py_RETURN_NONE;
        const c10::cuda::CUDAGuard guard(ptr->device());
        struct Job {
            svc_job* job = nullptr;
            ~Job() { svc_free(job); }
        } j;
        int64_t nvec = 0, replayed = 0;
        int rc = launch(ptr->get_device(), [&](void* st) {
            return svc_begin((int)M, (int)K, (int)V, static_cast<const int*>(ptr->data_ptr()), static_cast<const int*>(col->data_ptr()),
                             val ? val->data_ptr() : nullptr, st, &j.job, &nvec);
        });
        if (rc != 0) return PyLong_FromLong(rc);
        const auto ints = ptr->options().requires_grad(false);
        at::Tensor out_ptr = at::empty({(M + V - 1) / V + 1}, ints), out_col = at::empty({nvec}, ints), out_val;
        if (val) out_val = at::empty({nvec * V}, ints.dtype(at::kHalf));
        rc = launch(ptr->get_device(), [&](void* st) {
            const int e = svc_replayed_rows(j.job, &replayed);
            return e != 0 ? e : svc_finish(j.job, static_cast<int*>(out_ptr.data_ptr()), static_cast<int*>(out_col.data_ptr()),
                                           val ? out_val.data_ptr() : nullptr, st);
        });
        if (rc != 0) return PyLong_FromLong(rc);
        PyObject* values = Py_None;
        if (val) values = THPVariable_Wrap(out_val); else Py_INCREF(Py_None);
        return Py_BuildValue("(NNNL)", THPVariable_Wrap(out_ptr), THPVariable_Wrap(out_col), values, (long long)replayed);
    });
}

// svc_batch(list of (row_ptr, col_idx, values or None, M, K), vec_length, list of entries per matrix or None)
//   -> (list of (vec_ptr, vec_col, vec_values or None), replayed rows)
PyObject* py_svc_batch(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        long V;
        if (n != 3 || modes_active() || !PyList_CheckExact(a[0]) || !small_int(a[1], 1, 1 << 20, &V) || (a[2] != Py_None && !PyList_CheckExact(a[2])))
            Py_RETURN_NONE;
        const Py_ssize_t count = PyList_GET_SIZE(a[0]);
        if (count < 1 || count > 0x7fffffff || (a[2] != Py_None && PyList_GET_SIZE(a[2]) != count)) Py_RETURN_NONE;
        std::vector<int> M((size_t)count), K((size_t)count), nnz((size_t)count);
        std::vector<const int*> ptrs((size_t)count), cols((size_t)count);
        std::vector<const void*> vals((size_t)count);
        bool with_values = true;
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject* const m = PyList_GET_ITEM(a[0], i);
            if (!PyTuple_CheckExact(m) || PyTuple_GET_SIZE(m) != 5) Py_RETURN_NONE;
            with_values = with_values && PyTuple_GET_ITEM(m, 2) != Py_None;
        }
        const at::Tensor* first = nullptr;
        for (Py_ssize_t i = 0; i < count; ++i) {
            PyObject* const m = PyList_GET_ITEM(a[0], i);
            long rows, width, entries;
            const at::Tensor *ptr = plain(PyTuple_GET_ITEM(m, 0), at::kInt), *col = plain(PyTuple_GET_ITEM(m, 1), at::kInt);
            const at::Tensor* val = with_values ? plain(PyTuple_GET_ITEM(m, 2), at::kHalf) : nullptr;
            if (!ptr || !col || (with_values && !val) || !small_int(PyTuple_GET_ITEM(m, 3), 0, 0x7ffffff0, &rows) ||
                !small_int(PyTuple_GET_ITEM(m, 4), 0, 0x7fffffff, &width))
                Py_RETURN_NONE;
            if (a[2] == Py_None) entries = col->numel() <= 0x7fffffff ? (long)col->numel() : -1;
            else if (!small_int(PyList_GET_ITEM(a[2], i), 0, 0x7fffffff, &entries)) Py_RETURN_NONE;
            if (!first) first = ptr;
            if (entries < 0 || ptr->device() != first->device() || col->device() != first->device() || (val && val->device() != first->device()))
                Py_RETURN_NONE;
            M[i] = (int)rows; K[i] = (int)width; nnz[i] = (int)entries;
            ptrs[i] = static_cast<const int*>(ptr->data_ptr());
            cols[i] = static_cast<const int*>(col->data_ptr());
            vals[i] = val ? val->data_ptr() : nullptr;
        }
        const c10::cuda::CUDAGuard guard(first->device());
        struct Job {
            svc_batch_job* job = nullptr;
            ~Job() { svc_batch_free(job); }
        } j;
        std::vector<int64_t> nvec((size_t)count);
        int64_t replayed = 0, total = 0, vec_rows = 0;
        const auto ints = first->options().requires_grad(false);
        int rc = launch(first->get_device(), [&](void* st) {
            return svc_batch_begin((int)count, (int)V, M.data(), K.data(), nnz.data(), ptrs.data(), cols.data(), with_values ? vals.data() : nullptr, st,
                                   &j.job, nvec.data());
        });
        if (rc != 0) return PyLong_FromLong(rc);
        for (Py_ssize_t i = 0; i < count; ++i) { total += nvec[i]; vec_rows += (M[i] + V - 1) / V; }
        at::Tensor out_ptr = at::empty({vec_rows + (int64_t)count}, ints), out_col = at::empty({total}, ints), out_val;
        if (with_values) out_val = at::empty({total * V}, ints.dtype(at::kHalf));
        rc = launch(first->get_device(), [&](void* st) {
            const int e = svc_batch_replayed_rows(j.job, &replayed);
            return e != 0 ? e : svc_batch_finish(j.job, static_cast<int*>(out_ptr.data_ptr()), static_cast<int*>(out_col.data_ptr()),
                                                 with_values ? out_val.data_ptr() : nullptr, st);
        });
        if (rc != 0) return PyLong_FromLong(rc);
        PyObject* const list = PyList_New(count);
        if (!list) return nullptr;
        int64_t po = 0, vo = 0;
        for (Py_ssize_t i = 0; i < count; ++i) {
            const int64_t rows = (M[i] + V - 1) / V + 1;
            PyObject* values = Py_None;
            if (with_values) values = THPVariable_Wrap(out_val.narrow(0, vo * V, nvec[i] * V)); else Py_INCREF(Py_None);
            PyObject* const item = Py_BuildValue("(NNN)", THPVariable_Wrap(out_ptr.narrow(0, po, rows)), THPVariable_Wrap(out_col.narrow(0, vo, nvec[i])), values);
            if (!item) { Py_DECREF(list); return nullptr; }
            PyList_SET_ITEM(list, i, item);
            po += rows;
            vo += nvec[i];
        }
        return Py_BuildValue("(NL)", list, (long long)replayed);
    });
}

// sorted_row_swizzle(row_offsets)
PyObject* py_sorted_row_swizzle(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const at::Tensor* ptr = n == 1 && !modes_active() ? plain(a[0], at::kInt) : nullptr;
        if (!ptr || ptr->numel() < 1 || ptr->numel() > 0x7fffffff) Py_RETURN_NONE;
        const int m_vec = (int)(ptr->numel() - 1);
        at::Tensor out = at::empty({m_vec}, ptr->options().requires_grad(false));
        return result(launch(ptr->get_device(), [&](void* st) {
            return sspmm_sorted_row_swizzle(m_vec, static_cast<const int*>(ptr->data_ptr()), static_cast<int*>(out.data_ptr()), st);
        }), out);
    });
}

PyMethodDef methods[] = {
    {"svc", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_svc)), METH_FASTCALL, nullptr},
    {"svc_batch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_svc_batch)), METH_FASTCALL, nullptr},
    {"sorted_row_swizzle", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_sorted_row_swizzle)), METH_FASTCALL, nullptr},
    {"sspmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_sspmm)), METH_FASTCALL, nullptr},
    {"stacked", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_stacked)), METH_FASTCALL, nullptr},
    {"bspmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_bspmm)), METH_FASTCALL, nullptr},
    {"planned", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_planned)), METH_FASTCALL, nullptr},
    {"dense_copies", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_dense_copies)), METH_FASTCALL, nullptr},
    {"of_copy", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_of_copy)), METH_FASTCALL, nullptr},
    {"sspmm_sum", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_sspmm_sum)), METH_FASTCALL, nullptr},
    {"group_run_sum", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_group_run_sum)), METH_FASTCALL, nullptr},
    {"group_run", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_group_run)), METH_FASTCALL, nullptr},
    {"same_plain", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_same_plain)), METH_FASTCALL, nullptr},
    {"layer_norm_fm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_layer_norm_fm)), METH_FASTCALL, nullptr},
    {"attention_fm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention_fm)), METH_FASTCALL, nullptr},
    {"add_bias_fm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_add_bias_fm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_sspmm_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__sspmm_native(void) { return PyModule_Create(&module); }
