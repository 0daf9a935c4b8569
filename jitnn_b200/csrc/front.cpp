// The Python front of calls on torch CUDA tensors, in native code.
//
// A decode linear is done on the GPU in 2 to 5 us, and its launch takes the host 2.5; the checks, the new output tensor and the ctypes call take Python 5 more
// (256 x 1024, one row of x: 7.4 us a call, of them new_empty 1.8 and ctypes 0.7; with this module 4.0). Here the whole call is one method of this module.
//
// A method takes the plain case only: an ordinary strided, contiguous CUDA tensor (or parameter) with the weight's type, row length and device, while nothing
// intercepts torch calls (function and dispatch modes, functorch transforms, tracing). For everything else, wrong arguments among it, it returns None
// before it has done anything, and the caller goes on with the general code in ops.py, which knows the errors. Python.h's and torch's headers are all
// this needs; the kernels are reached through the addresses of the C ABI's functions that bind() is given.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty_cuda_dispatch.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>

namespace {

using Linear = int (*)(const void* w, const void* x, int64_t m, const float* bias, float* y, int mem, void* stream);
using Backward = int (*)(const void* w, const float* g, int64_t m, float* gx, int mem, void* stream);
using Dequantize = int (*)(const void* w, float* dst, int mem, void* stream);
using Quantize = int (*)(int device, const float* x, int64_t count, void* out, int mem, void* stream);
constexpr int MEM_DEVICE = 1;

Linear g_linear = nullptr, g_linear_bf16 = nullptr;
Backward g_backward = nullptr;
Dequantize g_dequantize = nullptr;
Quantize g_quantize = nullptr;
PyObject* g_check = nullptr;   // raises what a status code stands for
PyObject* g_weight = nullptr;  // the class of weights
PyObject *s_addr = nullptr, *s_dims = nullptr, *s_device = nullptr;

PyObject* not_plain() { Py_RETURN_NONE; }

// Nothing stands between a torch call and its kernel.
bool undisturbed() {
    using c10::DispatchKey;
    constexpr c10::DispatchKeySet taken({DispatchKey::Python, DispatchKey::PythonTLSSnapshot, DispatchKey::PythonDispatcher, DispatchKey::PreDispatch, DispatchKey::Tracer,
                                         DispatchKey::Functionalize, DispatchKey::FuncTorchDynamicLayerFrontMode, DispatchKey::FuncTorchDynamicLayerBackMode,
                                         DispatchKey::FuncTorchVmapMode, DispatchKey::FuncTorchBatched, DispatchKey::VmapMode, DispatchKey::Batched});
    return !c10::impl::tls_local_dispatch_key_set().included_.has_any(taken) && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
           at::impl::PythonTorchFunctionTLS::stack_len() == 0;
}

// The tensor behind a plain CUDA tensor or parameter, or null.
const at::Tensor* plain(PyObject* obj, at::ScalarType type) {
    using c10::DispatchKey;
    if (!THPVariable_CheckExact(obj)) {
        return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(obj);
    constexpr c10::DispatchKeySet special({DispatchKey::Python, DispatchKey::FuncTorchBatched, DispatchKey::FuncTorchGradWrapper, DispatchKey::Functionalize, DispatchKey::Batched,
                                           DispatchKey::Conjugate, DispatchKey::Negative, DispatchKey::ZeroTensor});
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.scalar_type() != type || t.dim() < 1 || t.key_set().has_any(special) || !t.is_contiguous()) {
        return nullptr;
    }
    return &t;
}

struct Weight {
    void* handle;
    int64_t n, k;
    int device;
};

bool attribute(PyObject* obj, PyObject* name, int64_t& out) {
    PyObject* v = PyObject_GetAttr(obj, name);
    if (v == nullptr) {
        PyErr_Clear();
        return false;
    }
    const bool is_int = PyLong_Check(v);
    out = is_int ? PyLong_AsLongLong(v) : 0;
    Py_DECREF(v);
    if (PyErr_Occurred() != nullptr) {
        PyErr_Clear();
        return false;
    }
    return is_int;
}

bool weight_of(PyObject* obj, Weight& w) {
    if ((PyObject*)Py_TYPE(obj) != g_weight) {
        return false;
    }
    int64_t addr = 0, device = 0;
    if (!attribute(obj, s_addr, addr) || addr == 0 || !attribute(obj, s_device, device)) {
        return false;
    }
    PyObject* dims = PyObject_GetAttr(obj, s_dims);
    if (dims == nullptr) {
        PyErr_Clear();
        return false;
    }
    bool ok = PyTuple_Check(dims) && PyTuple_GET_SIZE(dims) == 2 && PyLong_Check(PyTuple_GET_ITEM(dims, 0)) && PyLong_Check(PyTuple_GET_ITEM(dims, 1));
    if (ok) {
        w = Weight{(void*)addr, PyLong_AsLongLong(PyTuple_GET_ITEM(dims, 0)), PyLong_AsLongLong(PyTuple_GET_ITEM(dims, 1)), (int)device};
        ok = w.n > 0 && w.k > 0;
    }
    Py_DECREF(dims);
    return ok;
}

void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

at::Tensor empty_like_rows(const at::Tensor& x, int64_t last, at::ScalarType type) {
    at::DimVector sizes(x.sizes());
    sizes.back() = last;
    return at::cuda::empty(sizes, x.options().dtype(type));
}

// y, or the exception of a status code.
PyObject* finish(int rc, PyObject* y) {
    if (rc == 0) {
        return y;
    }
    Py_XDECREF(y);
    PyObject* code = PyLong_FromLong(rc);
    PyObject* none = code != nullptr ? PyObject_CallOneArg(g_check, code) : nullptr;
    Py_XDECREF(code);
    if (none != nullptr) {
        Py_DECREF(none);
        PyErr_SetString(PyExc_RuntimeError, "a call of the library failed");
    }
    return nullptr;
}

template <typename F>
PyObject* guarded(F body) {
    try {
        return body();
    } catch (const c10::OutOfMemoryError& e) {  // the general code raises torch's own
        (void)e;
        return not_plain();
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyObject* product(PyObject* const* args, Py_ssize_t count, at::ScalarType type, Linear fn) {
    return guarded([&]() -> PyObject* {
        Weight w;
        if (count != 3 || !weight_of(args[1], w) || !undisturbed()) {
            return not_plain();
        }
        const at::Tensor* const x = plain(args[0], type);
        if (x == nullptr || x->sizes().back() != w.k || x->get_device() != w.device) {
            return not_plain();
        }
        const float* bias = nullptr;
        if (args[2] != Py_None) {
            const at::Tensor* const b = plain(args[2], at::kFloat);
            if (b == nullptr || b->numel() != w.n || b->get_device() != w.device) {
                return not_plain();
            }
            bias = (const float*)b->const_data_ptr();
        }
        at::Tensor y = empty_like_rows(*x, w.n, at::kFloat);
        const void* const xp = x->const_data_ptr();
        float* const yp = (float*)y.mutable_data_ptr();
        const int64_t m = x->numel() / w.k;
        void* const stream = stream_of(w.device);
        int rc;
        Py_BEGIN_ALLOW_THREADS;
        rc = fn(w.handle, xp, m, bias, yp, MEM_DEVICE, stream);
        Py_END_ALLOW_THREADS;
        return finish(rc, rc == 0 ? THPVariable_Wrap(std::move(y)) : nullptr);
    });
}

PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t count) { return product(args, count, at::kFloat, g_linear); }
PyObject* linear_bf16(PyObject*, PyObject* const* args, Py_ssize_t count) { return product(args, count, at::kBFloat16, g_linear_bf16); }

PyObject* backward(PyObject*, PyObject* const* args, Py_ssize_t count) {
    return guarded([&]() -> PyObject* {
        Weight w;
        if (count != 2 || !weight_of(args[1], w) || !undisturbed()) {
            return not_plain();
        }
        const at::Tensor* const g = plain(args[0], at::kFloat);
        if (g == nullptr || g->sizes().back() != w.n || g->get_device() != w.device) {
            return not_plain();
        }
        at::Tensor gx = empty_like_rows(*g, w.k, at::kFloat);
        const float* const gp = (const float*)g->const_data_ptr();
        float* const xp = (float*)gx.mutable_data_ptr();
        const int64_t m = g->numel() / w.n;
        void* const stream = stream_of(w.device);
        int rc;
        Py_BEGIN_ALLOW_THREADS;
        rc = g_backward(w.handle, gp, m, xp, MEM_DEVICE, stream);
        Py_END_ALLOW_THREADS;
        return finish(rc, rc == 0 ? THPVariable_Wrap(std::move(gx)) : nullptr);
    });
}

PyObject* dequantize(PyObject*, PyObject* const* args, Py_ssize_t count) {  // weight, out
    return guarded([&]() -> PyObject* {
        Weight w;
        if (count != 2 || !weight_of(args[0], w) || !undisturbed()) {
            return not_plain();
        }
        const at::Tensor* const out = plain(args[1], at::kFloat);
        if (out == nullptr || out->numel() < w.n * w.k || out->get_device() != w.device) {
            return not_plain();
        }
        float* const to = (float*)out->mutable_data_ptr();
        void* const stream = stream_of(w.device);
        int rc;
        Py_BEGIN_ALLOW_THREADS;
        rc = g_dequantize(w.handle, to, MEM_DEVICE, stream);
        Py_END_ALLOW_THREADS;
        return finish(rc, rc == 0 ? Py_NewRef(args[1]) : nullptr);
    });
}

PyObject* quantize(PyObject*, PyObject* const* args, Py_ssize_t count) {
    return guarded([&]() -> PyObject* {
        if (count != 1 || !undisturbed()) {
            return not_plain();
        }
        const at::Tensor* const x = plain(args[0], at::kFloat);
        if (x == nullptr || x->numel() == 0 || x->sizes().back() % 32 != 0) {
            return not_plain();
        }
        const int device = (int)x->get_device();
        at::Tensor out = at::cuda::empty({x->numel() / 32 * 34}, x->options().dtype(at::kByte));
        const float* const xp = (const float*)x->const_data_ptr();
        void* const to = out.mutable_data_ptr();
        const int64_t n = x->numel();
        void* const stream = stream_of(device);
        int rc;
        Py_BEGIN_ALLOW_THREADS;
        rc = g_quantize(device, xp, n, to, MEM_DEVICE, stream);
        Py_END_ALLOW_THREADS;
        return finish(rc, rc == 0 ? THPVariable_Wrap(std::move(out)) : nullptr);
    });
}

// bind(weight class, check, addresses of jq_linear_f32, jq_linear_bf16, jq_linear_backward_f32, jq_dequantize, jq_quantize_q8_0)
PyObject* bind(PyObject*, PyObject* args) {
    PyObject *weight, *check;
    unsigned long long f[5];
    if (!PyArg_ParseTuple(args, "OOKKKKK", &weight, &check, &f[0], &f[1], &f[2], &f[3], &f[4])) {
        return nullptr;
    }
    Py_XSETREF(g_weight, Py_NewRef(weight));
    Py_XSETREF(g_check, Py_NewRef(check));
    g_linear = (Linear)f[0];
    g_linear_bf16 = (Linear)f[1];
    g_backward = (Backward)f[2];
    g_dequantize = (Dequantize)f[3];
    g_quantize = (Quantize)f[4];
    Py_RETURN_NONE;
}

PyMethodDef METHODS[] = {
    {"bind", bind, METH_VARARGS, nullptr},
    {"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, nullptr},
    {"linear_bf16", (PyCFunction)(void (*)(void))linear_bf16, METH_FASTCALL, nullptr},
    {"backward", (PyCFunction)(void (*)(void))backward, METH_FASTCALL, nullptr},
    {"dequantize", (PyCFunction)(void (*)(void))dequantize, METH_FASTCALL, nullptr},
    {"quantize", (PyCFunction)(void (*)(void))quantize, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef MODULE = {PyModuleDef_HEAD_INIT, "_front", nullptr, -1, METHODS, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__front(void) {
    s_addr = PyUnicode_InternFromString("_addr");
    s_dims = PyUnicode_InternFromString("_dims");
    s_device = PyUnicode_InternFromString("_device");
    return s_addr != nullptr && s_dims != nullptr && s_device != nullptr ? PyModule_Create(&MODULE) : nullptr;
}
