// Native half of the host mirror (zllm_b200/backend.py): the operators a decode step calls per projection, from Python objects
// straight to the C ABI.
//
// A decode projection of a small model runs for about 4 us on the GPU; building its ctypes arguments, reading the weight's
// shape through the ABI and allocating the output from Python took 6 us on top of the launch itself (10.1 us per call of a
// 1536 -> 512 projection, 3.8 us of them inside zq_linear).  Here a call costs one argument walk and one allocation from
// torch's caching allocator.  Checks, errors and results are those of the Python methods that call in.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/detail/CUDAHooksInterface.h>
#include <ATen/record_function.h>
#include <c10/core/DeviceGuard.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "../../include/zq_b200.h"

namespace {

PyObject *g_failure = nullptr;  // zllm_b200.ffi.ZqFailure
PyObject *s_handle, *s_rows, *s_cols;

struct PyError {};  // a Python exception is set

[[noreturn]] void fail(int code, const std::string &message) {
    PyObject *e = PyObject_CallFunction(g_failure, "is", code, message.c_str());
    if (e) {
        PyErr_SetObject(g_failure, e);
        Py_DECREF(e);
    }
    throw PyError();
}
void check(int rc, const zq_error &err) {
    if (rc) fail(rc, err.message);
}
[[noreturn]] void type_error(const std::string &message) {
    PyErr_SetString(PyExc_TypeError, message.c_str());
    throw PyError();
}

size_t attr_size(PyObject *o, PyObject *name) {
    PyObject *v = PyObject_GetAttr(o, name);
    if (!v) throw PyError();
    const size_t r = PyLong_AsSize_t(v);
    Py_DECREF(v);
    if (r == (size_t)-1 && PyErr_Occurred()) throw PyError();
    return r;
}
struct WeightRef {
    zq_weight *h;
    size_t rows, cols;
};
WeightRef weight_of(PyObject *o) { return {reinterpret_cast<zq_weight *>(attr_size(o, s_handle)), attr_size(o, s_rows), attr_size(o, s_cols)}; }

zq_ctx *ctx_of(PyObject *o) {
    void *p = PyLong_AsVoidPtr(o);
    if (!p && PyErr_Occurred()) throw PyError();
    return reinterpret_cast<zq_ctx *>(p);
}
at::Tensor tensor_of(PyObject *o) {
    if (!THPVariable_Check(o)) type_error("a tensor is expected, got " + std::string(Py_TYPE(o)->tp_name));
    return THPVariable_Unpack(o);
}
bool is_none(PyObject *o) { return o == Py_None; }
int zq_dtype(at::ScalarType t) { return t == at::kFloat ? ZQ_F32 : t == at::kHalf ? ZQ_F16 : t == at::kBFloat16 ? ZQ_BF16 : -1; }
std::string dtype_name(at::ScalarType t) {
    std::string n = at::toString(t);
    const char *known = t == at::kDouble ? "torch.float64" : t == at::kLong ? "torch.int64" : t == at::kInt ? "torch.int32" : t == at::kByte ? "torch.uint8" : t == at::kChar ? "torch.int8" : t == at::kBool ? "torch.bool" : nullptr;
    return known ? known : "torch." + n;
}
int in_dtype(const at::Tensor &x) {
    const int d = zq_dtype(x.scalar_type());
    if (d < 0) type_error("unsupported activation dtype " + dtype_name(x.scalar_type()));
    return d;
}
at::ScalarType dtype_of(PyObject *o) {
    if (!THPDtype_Check(o)) type_error("a torch dtype is expected");
    return reinterpret_cast<THPDtype *>(o)->scalar_type;
}
// out_dtype, or the input's dtype when it is None; KeyError for a dtype the library does not write
at::ScalarType out_dtype_of(PyObject *o, at::ScalarType fallback) {
    const at::ScalarType t = is_none(o) ? fallback : dtype_of(o);
    if (zq_dtype(t) < 0) {
        if (is_none(o)) type_error("unsupported activation dtype " + dtype_name(t));
        PyErr_SetObject(PyExc_KeyError, o);
        throw PyError();
    }
    return t;
}
size_t rows_of(const at::Tensor &x, size_t cols) {
    const int64_t last = x.dim() ? x.size(-1) : 1;
    if (cols == 0 || (size_t)last != cols) fail(1, "linear input cols=" + std::to_string(last) + ", weight cols=" + std::to_string(cols));
    return (size_t)x.numel() / cols;
}
// Other threads run while torch allocates (which may wait for the device) and inside the ABI (workspace growth, host-buffer calls).
struct NoGil {
    PyThreadState *s = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(s); }
};
// without the GIL.  On the GPU from torch's allocator directly (0.4 us instead of the 0.8 of at::empty), by way of its hooks, so that this library
// needs no CUDA build of torch to load, unless something is on that would see the call (dispatch modes, tracing, function transforms, autocast, the callbacks of
// profilers) or fill the tensor.
at::Tensor new_rows(const at::Tensor &like, size_t m, size_t n, at::ScalarType t) {
    const int64_t size[2] = {(int64_t)m, (int64_t)n};
    const bool watched = !(c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set).empty() || at::getStepCallbacksUnlessEmpty(at::RecordScope::FUNCTION).has_value();
    if (like.is_cuda() && !watched && !at::globalContext().deterministicAlgorithms()) {
        const c10::DeviceGuard on(like.device());
        return at::Tensor(at::detail::empty_generic(size, at::detail::getCUDAHooks().getCUDADeviceAllocator(), c10::DispatchKeySet(c10::DispatchKey::CUDA), t, std::nullopt));
    }
    return at::empty(size, like.options().dtype(t));
}
at::Tensor contiguous(const at::Tensor &t) {
    if (t.is_contiguous()) return t;
    NoGil g;
    return t.contiguous();
}
at::Tensor as_f32(const at::Tensor &t) {
    if (t.scalar_type() == at::kFloat) return t;
    NoGil g;
    return t.to(at::kFloat);
}

template <class Fn> PyObject *guarded(Fn fn) {
    try {
        return fn();
    } catch (const PyError &) {
        return nullptr;
    } catch (...) {  // torch's own errors become the exceptions torch raises from Python (an allocation that fails: torch.OutOfMemoryError)
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}
template <class Tensors> PyObject *wrap_list(Tensors &ys) {
    PyObject *out = PyList_New((Py_ssize_t)ys.size());
    if (!out) throw PyError();
    for (size_t i = 0; i < ys.size(); ++i) PyList_SET_ITEM(out, (Py_ssize_t)i, THPVariable_Wrap(std::move(ys[i])));
    return out;
}
// The items of a sequence for the time of a call.
struct Items {
    PyObject *fast;
    Items(PyObject *seq) : fast(PySequence_Fast(seq, "a sequence is expected")) {
        if (!fast) throw PyError();
    }
    ~Items() { Py_DECREF(fast); }
    size_t size() const { return (size_t)PySequence_Fast_GET_SIZE(fast); }
    PyObject *operator[](size_t i) const { return PySequence_Fast_GET_ITEM(fast, (Py_ssize_t)i); }
};

// KeyError(x.dtype): what a batch raises for inputs the library does not read
[[noreturn]] void dtype_key_error(PyObject *x) {
    PyObject *dtype = PyObject_GetAttrString(x, "dtype");
    if (dtype) {
        PyErr_SetObject(PyExc_KeyError, dtype);
        Py_DECREF(dtype);
    }
    throw PyError();
}

// linear(ctx, x, weight, out_dtype, residual)
PyObject *py_linear(PyObject *, PyObject *const *a, Py_ssize_t) {
    return guarded([&]() -> PyObject * {
        zq_ctx *ctx = ctx_of(a[0]);
        const at::Tensor x = contiguous(tensor_of(a[1]));
        const WeightRef w = weight_of(a[2]);
        const size_t m = rows_of(x, w.cols);
        const at::ScalarType od = out_dtype_of(a[3], x.scalar_type());
        at::Tensor y, r;
        if (!is_none(a[4])) {
            r = contiguous(tensor_of(a[4]));
            if ((size_t)r.numel() != m * w.rows || r.scalar_type() != od) fail(1, "residual shape/dtype mismatch: " + std::to_string(r.numel()) + " values of " + dtype_name(r.scalar_type()) + " vs " + std::to_string(m * w.rows) + " of " + dtype_name(od));
        }
        const int xd = in_dtype(x);
        zq_error err;
        int rc;
        {
            NoGil g;
            y = new_rows(x, m, w.rows, od);
            rc = zq_linear(ctx, w.h, x.data_ptr(), xd, m, y.data_ptr(), zq_dtype(od), r.defined() ? r.data_ptr() : nullptr, &err);
        }
        check(rc, err);
        return THPVariable_Wrap(std::move(y));
    });
}

// linear_batch(ctx, jobs, out_dtype)
PyObject *py_linear_batch(PyObject *, PyObject *const *a, Py_ssize_t) {
    return guarded([&]() -> PyObject * {
        zq_ctx *ctx = ctx_of(a[0]);
        Items jobs(a[1]);
        const size_t n = jobs.size();
        std::vector<zq_linear_job> arr(n);
        std::vector<at::Tensor> ys(n), inputs(n), keep;
        std::vector<size_t> rows(n);
        at::ScalarType xt = at::kFloat, od = at::kFloat;
        for (size_t i = 0; i < n; ++i) {
            Items job(jobs[i]);
            if (job.size() < 2) type_error("linear_batch: a job is (x, weight[, residual]) or (x, gate, up, \"gated\") or (x, weight, residual, \"row\")");
            bool gated = false, row = false;
            if (job.size() == 4 && PyUnicode_Check(job[3])) {
                gated = PyUnicode_CompareWithASCIIString(job[3], "gated") == 0;
                row = PyUnicode_CompareWithASCIIString(job[3], "row") == 0;
            }
            const at::Tensor x = contiguous(tensor_of(job[0]));
            const WeightRef w = weight_of(job[1]);
            const size_t m = rows_of(x, w.cols);
            if (i == 0) {
                xt = x.scalar_type();
                if (zq_dtype(xt) < 0) dtype_key_error(job[0]);
                od = out_dtype_of(a[2], xt);
            }
            if (x.scalar_type() != xt) type_error("linear_batch: all inputs must share one dtype");
            zq_linear_job &j = arr[i];
            j = {};
            j.w = w.h;
            j.w_up = gated ? weight_of(job[2]).h : nullptr;
            j.dev_x = x.data_ptr();
            j.m = m;
            rows[i] = w.rows;
            inputs[i] = x;
            if ((job.size() == 3 || row) && !is_none(job[2])) {
                const at::Tensor r = contiguous(tensor_of(job[2]));
                j.dev_residual = r.data_ptr();
                keep.push_back(r);
            }
            j.flags = row ? ZQ_JOB_ROW_PARALLEL : 0;
        }
        if (n) {
            zq_error err;
            int rc;
            {
                NoGil g;
                for (size_t i = 0; i < n; ++i) {
                    ys[i] = new_rows(inputs[i], arr[i].m, rows[i], od);
                    arr[i].dev_y = ys[i].data_ptr();
                }
                rc = zq_linear_batch(ctx, arr.data(), n, zq_dtype(xt), zq_dtype(od), &err);
            }
            check(rc, err);
        }
        return wrap_list(ys);
    });
}

// linear_multi(ctx, x, weights, out_dtype, norm_weight | None, eps, weight_offset)
PyObject *py_linear_multi(PyObject *, PyObject *const *a, Py_ssize_t) {
    return guarded([&]() -> PyObject * {
        zq_ctx *ctx = ctx_of(a[0]);
        const at::Tensor x = contiguous(tensor_of(a[1]));
        Items ws(a[2]);
        const size_t n = ws.size();
        if (!n) {
            PyErr_SetString(PyExc_IndexError, "no weights given");
            throw PyError();
        }
        c10::SmallVector<const zq_weight *, 4> wh(n);
        c10::SmallVector<at::Tensor, 4> ys(n);
        c10::SmallVector<void *, 4> yp(n);
        c10::SmallVector<size_t, 4> rows(n);
        const size_t cols = weight_of(ws[0]).cols, m = rows_of(x, cols);
        at::Tensor norm;
        if (!is_none(a[4])) {
            norm = as_f32(contiguous(tensor_of(a[4])));
            if ((size_t)norm.numel() != cols) fail(1, "norm weight has " + std::to_string(norm.numel()) + " elements, input width is " + std::to_string(cols));
        }
        const at::ScalarType od = out_dtype_of(a[3], x.scalar_type());
        for (size_t i = 0; i < n; ++i) {
            const WeightRef w = weight_of(ws[i]);
            wh[i] = w.h;
            rows[i] = w.rows;
        }
        const int xd = in_dtype(x);
        const double eps = PyFloat_AsDouble(a[5]), offset = PyFloat_AsDouble(a[6]);
        if (PyErr_Occurred()) throw PyError();
        zq_error err;
        int rc;
        {
            NoGil g;
            for (size_t i = 0; i < n; ++i) {
                ys[i] = new_rows(x, m, rows[i], od);
                yp[i] = ys[i].data_ptr();
            }
            rc = norm.defined() ? zq_rmsnorm_linear(ctx, wh.data(), n, x.data_ptr(), xd, m, norm.data_ptr<float>(), (float)eps, (float)offset, yp.data(), zq_dtype(od), &err)
                                : zq_linear_multi(ctx, wh.data(), n, x.data_ptr(), xd, m, yp.data(), zq_dtype(od), &err);
        }
        check(rc, err);
        return wrap_list(ys);
    });
}

// gated(ctx, x, gate, up, down | None, out_dtype, residual)
PyObject *py_gated(PyObject *, PyObject *const *a, Py_ssize_t) {
    return guarded([&]() -> PyObject * {
        zq_ctx *ctx = ctx_of(a[0]);
        const at::Tensor x = contiguous(tensor_of(a[1]));
        const WeightRef gate = weight_of(a[2]), up = weight_of(a[3]);
        const bool mlp = !is_none(a[4]);
        const WeightRef down = mlp ? weight_of(a[4]) : WeightRef{nullptr, gate.rows, 0};
        const size_t m = rows_of(x, gate.cols);
        const at::ScalarType od = out_dtype_of(a[5], x.scalar_type());
        at::Tensor y, r;
        if (!is_none(a[6])) r = contiguous(tensor_of(a[6]));
        const int xd = in_dtype(x);
        zq_error err;
        int rc;
        {
            NoGil g;
            y = new_rows(x, m, down.rows, od);
            rc = mlp ? zq_gated_mlp(ctx, gate.h, up.h, down.h, x.data_ptr(), xd, m, y.data_ptr(), zq_dtype(od), r.defined() ? r.data_ptr() : nullptr, &err)
                     : zq_gated_silu(ctx, gate.h, up.h, x.data_ptr(), xd, m, y.data_ptr(), zq_dtype(od), &err);
        }
        check(rc, err);
        return THPVariable_Wrap(std::move(y));
    });
}

// rope(ctx, query, key | None, num_heads, num_kv_heads, rotary_dim, position, cos, sin, interleaved, suffix)
PyObject *py_rope(PyObject *, PyObject *const *a, Py_ssize_t) {
    return guarded([&]() -> PyObject * {
        zq_ctx *ctx = ctx_of(a[0]);
        const at::Tensor q = tensor_of(a[1]);
        at::Tensor k;
        if (!is_none(a[2])) k = tensor_of(a[2]);
        long v[6];
        const int at_[6] = {3, 4, 5, 6, 9, 10};
        for (int i = 0; i < 6; ++i) {
            v[i] = i < 4 ? PyLong_AsLong(a[at_[i]]) : PyObject_IsTrue(a[at_[i]]);
            if (v[i] == -1 && PyErr_Occurred()) throw PyError();
        }
        const int64_t rows = q.dim() > 1 ? q.size(0) : 1;
        if (rows == 0 || v[0] == 0) {
            PyErr_SetString(PyExc_ZeroDivisionError, "rope: no rows or no heads");
            throw PyError();
        }
        const int64_t head_dim = q.numel() / rows / v[0];
        if (k.defined() && (k.scalar_type() != q.scalar_type() || k.numel() != rows * v[1] * head_dim)) fail(1, "rope: key shape or dtype does not match the query's");
        const at::Tensor c = as_f32(contiguous(tensor_of(a[7]))), s = as_f32(contiguous(tensor_of(a[8])));
        if (c.numel() != s.numel()) fail(1, "rope: cos and sin tables differ in length (" + std::to_string(c.numel()) + " / " + std::to_string(s.numel()) + ")");
        const int d = in_dtype(q);
        zq_error err;
        int rc;
        {
            NoGil g;
            rc = zq_rope_qk(ctx, q.data_ptr(), (size_t)v[0], k.defined() ? k.data_ptr() : nullptr, k.defined() ? (size_t)v[1] : 0, d, (size_t)rows, (size_t)head_dim, (size_t)v[2], (int)v[4], (int)v[5], (size_t)v[3],
                            c.data_ptr<float>(), s.data_ptr<float>(), (size_t)c.numel(), &err);
        }
        check(rc, err);
        Py_RETURN_NONE;
    });
}

// gather_rows(ctx, weight, row_ids, dtype): row_ids on the weight's device, int32, contiguous
PyObject *py_gather_rows(PyObject *, PyObject *const *a, Py_ssize_t) {
    return guarded([&]() -> PyObject * {
        zq_ctx *ctx = ctx_of(a[0]);
        const WeightRef w = weight_of(a[1]);
        const at::Tensor ids = tensor_of(a[2]);
        const at::ScalarType t = dtype_of(a[3]);
        zq_error err;
        int rc;
        at::Tensor y;
        {
            NoGil g;
            y = new_rows(ids, (size_t)ids.numel(), w.cols, t);
            rc = zq_gather_rows(ctx, w.h, reinterpret_cast<const uint32_t *>(ids.data_ptr<int>()), (size_t)ids.numel(), y.data_ptr(), zq_dtype(t), &err);
        }
        check(rc, err);
        return THPVariable_Wrap(std::move(y));
    });
}

// linear_host_batch(ctx, jobs): (x, weight, y) with x and y buffers of f32 or f16
PyObject *py_linear_host_batch(PyObject *, PyObject *const *a, Py_ssize_t) {
    return guarded([&]() -> PyObject * {
        zq_ctx *ctx = ctx_of(a[0]);
        Items jobs(a[1]);
        const size_t n = jobs.size();
        std::vector<zq_linear_host_job> arr(n);
        struct View {
            Py_buffer b;
            bool held = false;
            ~View() {
                if (held) PyBuffer_Release(&b);
            }
        };
        std::vector<View> views(2 * n);
        int dt[2] = {ZQ_F32, ZQ_F32};
        for (size_t i = 0; i < n; ++i) {
            Items job(jobs[i]);
            if (job.size() != 3) type_error("linear_host_batch: a job is (x, weight, y)");
            const WeightRef w = weight_of(job[1]);
            for (int k = 0; k < 2; ++k) {
                View &v = views[2 * i + k];
                if (PyObject_GetBuffer(job[2 * k], &v.b, PyBUF_FORMAT | PyBUF_STRIDES)) throw PyError();
                v.held = true;
                if (i == 0) {
                    const char *f = v.b.format ? v.b.format : "";
                    dt[k] = !strcmp(f, "f") ? ZQ_F32 : !strcmp(f, "e") ? ZQ_F16 : -1;
                    if (dt[k] < 0) {
                        PyErr_SetString(PyExc_KeyError, f);
                        throw PyError();
                    }
                }
            }
            if (w.cols == 0) fail(4, "linear_host_batch: the weight was released");
            arr[i] = {w.h, views[2 * i].b.buf, (size_t)(views[2 * i].b.len / views[2 * i].b.itemsize) / w.cols, views[2 * i + 1].b.buf};
        }
        if (!n) {
            PyErr_SetString(PyExc_IndexError, "list index out of range");
            throw PyError();
        }
        zq_error err;
        int rc;
        {
            NoGil g;
            rc = zq_linear_host_batch(ctx, arr.data(), n, dt[0], dt[1], &err);
        }
        check(rc, err);
        Py_RETURN_NONE;
    });
}

PyObject *py_setup(PyObject *, PyObject *failure) {
    Py_INCREF(failure);
    Py_XSETREF(g_failure, failure);
    Py_RETURN_NONE;
}

template <Py_ssize_t N, PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)> PyObject *counted(PyObject *self, PyObject *const *a, Py_ssize_t n) {
    if (n != N) {
        PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", N, n);
        return nullptr;
    }
    return F(self, a, n);
}
#define ZQ_FAST(name, n, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&counted<n, fn>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    ZQ_FAST("linear", 5, py_linear), ZQ_FAST("linear_batch", 3, py_linear_batch), ZQ_FAST("linear_multi", 7, py_linear_multi), ZQ_FAST("gated", 7, py_gated),
    ZQ_FAST("rope", 11, py_rope), ZQ_FAST("gather_rows", 4, py_gather_rows), ZQ_FAST("linear_host_batch", 2, py_linear_host_batch), {"setup", py_setup, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_zq_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__zq_torch() {
    s_handle = PyUnicode_InternFromString("_h");
    s_rows = PyUnicode_InternFromString("_rows");
    s_cols = PyUnicode_InternFromString("_cols");
    return PyModule_Create(&module);
}
