// The host path of a call, natively: what stands between a Python caller and the C ABI when everything is as it
// usually is.  A launch costs the driver 2.2 us; around it, through ctypes and torch's Python operators, a call of a bound operator
// took 3.3 us, of a linear layer 19 (two launches, two allocations, a view), of a convolution module 23 (three launches).
//
//   bind               the addresses of the library's functions; False where the states of the two builds differ, or torch is not
//                      the one whose headers this module was compiled with (they lay out at::Tensor)
//   spmm / spconv      one call of a bound operator, by the address of its state
//   linear / conv2d    one forward of a module, for plain operands; None for everything else (subclasses, operands under a
//                      transform, a mode or a trace, values not in memory, gradients to record, another device, layouts that
//                      need a copy, and calls that the library refuses): the module's Python code is then the one that runs
//
// The library's functions come as addresses (bind), so that this module links nothing of it.  The GIL is released while
// a call is enqueued, as ctypes does: a launch may wait for room in the queue.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <climits>
#include <cstring>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/grad_mode.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "shflbw.h"

namespace {

decltype(&shflbw_spmm_exec) spmm_exec = nullptr;
decltype(&shflbw_spconv_exec) spconv_exec = nullptr;
decltype(&shflbw_spconv_exec_bias) spconv_exec_bias = nullptr;
decltype(&shflbw_spconv_init) spconv_init = nullptr;
decltype(&shflbw_linear_exec) linear_exec = nullptr;
decltype(&shflbw_linear_direct) linear_direct = nullptr;
PyObject* name_cuda_stream = nullptr;

PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 8) { PyErr_SetString(PyExc_TypeError, "bind(spmm_exec, spconv_exec, spconv_exec_bias, spconv_init, linear_exec, linear_direct, size of a state, torch.__version__)"); return nullptr; }
    const long long size = PyLong_AsLongLong(args[6]);
    const char* const torch_version = PyUnicode_AsUTF8(args[7]);
    if (PyErr_Occurred()) return nullptr;
    if (size != (long long)sizeof(shflbw_spconv_state_t) || strcmp(torch_version, SHFLBW_TORCH_VERSION)) Py_RETURN_FALSE;
    void* a[6];
    for (int i = 0; i < 6; ++i)
        if (!(a[i] = PyLong_AsVoidPtr(args[i]))) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null address"); return nullptr; }
    spmm_exec = (decltype(spmm_exec))a[0];
    spconv_exec = (decltype(spconv_exec))a[1];
    spconv_exec_bias = (decltype(spconv_exec_bias))a[2];
    spconv_init = (decltype(spconv_init))a[3];
    linear_exec = (decltype(linear_exec))a[4];
    linear_direct = (decltype(linear_direct))a[5];
    Py_RETURN_TRUE;
}

// None, an object with a `cuda_stream`, or an integer.
bool stream_of(PyObject* o, void** s) {
    *s = nullptr;
    if (o == Py_None) return true;
    PyObject* v = PyLong_CheckExact(o) ? Py_NewRef(o) : PyObject_GetAttr(o, name_cuda_stream);
    if (!v) {
        if (!PyErr_ExceptionMatches(PyExc_AttributeError)) return false;
        PyErr_Clear();
        v = Py_NewRef(o);
    }
    PyObject* number = PyNumber_Long(v);
    Py_DECREF(v);
    if (!number) return false;
    *s = (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(number);
    Py_DECREF(number);
    return !PyErr_Occurred();
}

template <class Exec>
PyObject* exec_state(Exec exec, PyObject* const* args, Py_ssize_t n) {
    void* stream;
    if (n != 2) { PyErr_SetString(PyExc_TypeError, "(address of a state, stream)"); return nullptr; }
    const auto* state = (decltype(exec(nullptr, nullptr), (const void*)nullptr))PyLong_AsVoidPtr(args[0]);
    if (!state && PyErr_Occurred()) return nullptr;
    if (!stream_of(args[1], &stream)) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = exec(state, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}
PyObject* spmm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return exec_state([](const void* st, void* s) { return spmm_exec((const shflbw_spmm_state_t*)st, s); }, args, n);
}
PyObject* spconv(PyObject*, PyObject* const* args, Py_ssize_t n) {
    return exec_state([](const void* st, void* s) { return spconv_exec((const shflbw_spconv_state_t*)st, s); }, args, n);
}

// (DispatchKeySet's own difference keeps the backend bits.)
bool within(c10::DispatchKeySet a, c10::DispatchKeySet b) { return (a.raw_repr() & ~b.raw_repr()) == 0; }
// A tensor that is nothing but its values in this device's memory.
bool plain(const at::Tensor& t) {
    constexpr c10::DispatchKeySet usual({c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutogradCUDA,
                                         c10::DispatchKey::AutocastCUDA});
    return t.defined() && within(t.key_set(), usual) && t.scalar_type() == at::kHalf && t.const_data_ptr() != nullptr;
}
// Nothing watches or replaces the operators that run: no mode, transform, dispatcher or trace.
bool unobserved() {
    const c10::DispatchKeySet on = c10::impl::tls_local_dispatch_key_set().included_;
    const c10::DispatchKeySet usual = c10::default_included_set | c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView);
    return within(on, usual) && at::impl::PythonTorchFunctionTLS::stack_len() == 0 && !torch::jit::tracer::isTracing();
}
// The bias as nn.py's _fused_bias asks for it: -1 not so, 0 none, 1 to be added by the kernels.
int bias_of(PyObject* o, const at::Tensor& x, int64_t n, uintptr_t align, at::Tensor* bias) {
    if (o == Py_None) return 0;
    if (!THPVariable_CheckExact(o)) return -1;
    *bias = THPVariable_Unpack(o);
    if (!plain(*bias) || bias->device() != x.device() || bias->dim() != 1 || bias->size(0) != n || !bias->is_contiguous()) return -1;
    if ((uintptr_t)bias->const_data_ptr() % align != 0) return -1;
    if (bias->requires_grad() && at::GradMode::is_enabled()) return -1;
    if (bias->_fw_grad(0).defined()) return -1;
    return 1;
}

// linear(x, bias, matrix, in_features, out_features)
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 5) { PyErr_SetString(PyExc_TypeError, "linear(x, bias, matrix, in_features, out_features)"); return nullptr; }
    const long long K = PyLong_AsLongLong(args[3]), M = PyLong_AsLongLong(args[4]);
    const auto* m = (const shflbw_matrix_t*)PyLong_AsVoidPtr(args[2]);
    if (PyErr_Occurred()) return nullptr;
    if (!THPVariable_CheckExact(args[0])) Py_RETURN_NONE;
    try {
        const at::Tensor x = THPVariable_Unpack(args[0]);
        at::Tensor bias, y;
        if (!unobserved() || !plain(x) || x.dim() != 2 || x.size(1) != K || x.size(0) <= 0 || x.size(0) > (1 << 30) || !x.is_contiguous()) Py_RETURN_NONE;
        if (x.device().index() != c10::cuda::current_device()) Py_RETURN_NONE;
        const int with_bias = bias_of(args[1], x, M, 2, &bias);
        if (with_bias < 0) Py_RETURN_NONE;
        int rc;
        Py_BEGIN_ALLOW_THREADS
        try {
            const int64_t tokens = x.size(0), padded = (tokens + 7) / 8 * 8;
            const at::Tensor out = at::empty({M, padded}, x.options());
            const void* const b = with_bias ? bias.const_data_ptr() : nullptr;
            void* const stream = c10::cuda::getCurrentCUDAStream().stream();
            rc = linear_direct(m, (int)tokens, x.const_data_ptr(), b, (int)padded, out.data_ptr(), stream);
            if (rc == SHFLBW_ERR_UNSUPPORTED) {
                const at::Tensor xt = at::empty({K, padded}, x.options());
                rc = linear_exec(m, (int)tokens, x.const_data_ptr(), b, xt.data_ptr(), (int)padded, out.data_ptr(), stream);
            }
            if (rc == SHFLBW_OK) y = out.as_strided({tokens, M}, {1, padded});
        } catch (...) {
            Py_BLOCK_THREADS
            throw;
        }
        Py_END_ALLOW_THREADS
        if (rc != SHFLBW_OK) Py_RETURN_NONE;
        return THPVariable_Wrap(std::move(y));
    } catch (...) { Py_RETURN_NONE; }                        // (the Python code meets the same error and raises it as torch does)
}

// conv2d(x, bias, filter, stride, in_channels, out_channels)
PyObject* conv2d(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 6) { PyErr_SetString(PyExc_TypeError, "conv2d(x, bias, filter, stride, in_channels, out_channels)"); return nullptr; }
    const long long stride = PyLong_AsLongLong(args[3]), C = PyLong_AsLongLong(args[4]), F = PyLong_AsLongLong(args[5]);
    auto* f = (shflbw_matrix_t*)PyLong_AsVoidPtr(args[2]);
    if (PyErr_Occurred()) return nullptr;
    if (!THPVariable_CheckExact(args[0]) || stride < 1 || stride > INT_MAX) Py_RETURN_NONE;
    try {
        const at::Tensor x = THPVariable_Unpack(args[0]);
        at::Tensor bias, y;
        if (!unobserved() || !plain(x) || x.dim() != 4 || x.size(1) != C || x.numel() == 0 || x.numel() > (1ll << 31)) Py_RETURN_NONE;
        const int64_t B = x.size(0), H = x.size(2), W = x.size(3);
        if (x.stride(1) != 1 || x.stride(3) != C || x.stride(2) != W * C || x.stride(0) != H * W * C) Py_RETURN_NONE;   // NHWC in memory
        if (x.device().index() != c10::cuda::current_device()) Py_RETURN_NONE;
        const int with_bias = bias_of(args[1], x, F, 16, &bias);
        if (with_bias < 0) Py_RETURN_NONE;
        int rc;
        Py_BEGIN_ALLOW_THREADS
        try {
            const at::Tensor out = at::empty({B, (H + stride - 1) / stride, (W + stride - 1) / stride, F}, x.options().memory_format(c10::nullopt));
            shflbw_spconv_state_t st;
            rc = spconv_init(f, (int)B, (int)H, (int)W, (int)stride, x.const_data_ptr(), out.data_ptr(), 1.f, SHFLBW_KERNEL_AUTO, &st);
            if (rc == SHFLBW_OK) rc = spconv_exec_bias(&st, with_bias ? bias.const_data_ptr() : nullptr, c10::cuda::getCurrentCUDAStream().stream());
            if (rc == SHFLBW_OK) y = out.permute({0, 3, 1, 2});
        } catch (...) {
            Py_BLOCK_THREADS
            throw;
        }
        Py_END_ALLOW_THREADS
        if (rc != SHFLBW_OK) Py_RETURN_NONE;
        return THPVariable_Wrap(std::move(y));
    } catch (...) { Py_RETURN_NONE; }                        // (the Python code meets the same error and raises it as torch does)
}

PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void (*)())bind, METH_FASTCALL, "addresses of the library's functions"},
    {"spmm", (PyCFunction)(void (*)())spmm, METH_FASTCALL, "status of shflbw_spmm_exec"},
    {"spconv", (PyCFunction)(void (*)())spconv, METH_FASTCALL, "status of shflbw_spconv_exec"},
    {"linear", (PyCFunction)(void (*)())linear, METH_FASTCALL, "forward of a linear layer, or None"},
    {"conv2d", (PyCFunction)(void (*)())conv2d, METH_FASTCALL, "forward of a convolution module, or None"},
    {nullptr, nullptr, 0, nullptr}};
// (build.py looks for the end of this text in the built file)
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "host path of a call, compiled for torch " SHFLBW_TORCH_VERSION, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    name_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    return name_cuda_stream ? PyModule_Create(&module) : nullptr;
}
