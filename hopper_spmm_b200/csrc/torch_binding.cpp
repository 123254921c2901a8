// The device-tensor product for Python: argument checks, output allocation, stream lookup and the call into the C
// ABI in one native function.  Through torch's Python attributes and ctypes the same steps take 8 us a call, more
// than the GPU needs for a 4096 x 4096 matrix at 1 % density.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#if __has_include(<ATen/cuda/EmptyTensor.h>)
#include <ATen/cuda/EmptyTensor.h>
#define HAS_EMPTY_CUDA 1
#endif
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b200_spmm.h"

namespace {

PyObject *refuse(const char *what) {
    PyErr_SetString(PyExc_ValueError, what);
    return nullptr;
}

// Other Python threads run while this exists.
struct ThreadsAllowed {
    PyThreadState *state = PyEval_SaveThread();
    ~ThreadsAllowed() { PyEval_RestoreThread(state); }
};

#ifdef HAS_EMPTY_CUDA
// torch's own, and not part of its interface: taken where it has the signature known here.
template <typename Type>
auto empty_direct(int, at::IntArrayRef sizes, Type type, at::Device device)
    -> decltype(at::Tensor(at::detail::empty_cuda(sizes, type, device, std::nullopt))) {
    return at::Tensor(at::detail::empty_cuda(sizes, type, device, std::nullopt));
}
#endif
template <typename Type>
at::Tensor empty_direct(long, at::IntArrayRef, Type, at::Device) {
    return at::Tensor();
}

// A new CUDA tensor.  Through the dispatcher it is 1.2 of the 4.1 us that a small product takes the host, directly 0.9.  The
// dispatcher is left out only where nothing would happen in it but the allocation: no mode, tracer, transform or inference mode
// (the thread's keys are the default ones), no profiler or other observer of calls, and no fill that deterministic runs ask for.
at::Tensor new_cuda(int64_t rows, int64_t n, at::ScalarType type, const at::Tensor &like) {
    const c10::impl::LocalDispatchKeySet keys = c10::impl::tls_local_dispatch_key_set();
    if (keys.included_ == c10::default_included_set && keys.excluded_ == c10::default_excluded_set && !at::hasCallbacks() &&
        !at::globalContext().deterministicAlgorithms()) {
        at::Tensor out = empty_direct(0, {rows, n}, type, like.device());
        if (out.defined()) return out;
    }
    return at::empty({rows, n}, like.options().dtype(type).requires_grad(false));
}

// spmm(plan, is_f16, rows, cols, B, C or None, c_half, stream or None) -> C, or a status code that is not 0
// Any tensor accessor may throw: a sparse tensor has no strides, a tensor subclass may answer for sizes and strides in
// Python.  The macros turn whatever comes (a Python error among it) into the exception the caller sees.
PyObject *spmm(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (n_args != 8) {
        PyErr_SetString(PyExc_TypeError, "spmm takes 8 arguments");
        return nullptr;
    }
    auto *plan = static_cast<b200spmm_plan_t *>(PyLong_AsVoidPtr(args[0]));
    const bool f16 = args[1] == Py_True, c_half = PyObject_IsTrue(args[6]) == 1;
    const int64_t rows = PyLong_AsLongLong(args[2]), cols = PyLong_AsLongLong(args[3]);
    if (PyErr_Occurred()) return nullptr;
    const char *bad_b = f16 ? "B must be a CUDA float16 tensor of shape [cols, n] with unit column stride"
                            : "B must be a CUDA float32 tensor of shape [cols, n] with unit column stride";
    if (!THPVariable_Check(args[4])) return refuse(bad_b);
    const at::Tensor &B = THPVariable_Unpack(args[4]);
    if (!B.is_cuda() || B.scalar_type() != (f16 ? at::kHalf : at::kFloat) || B.dim() != 2 || B.stride(1) != 1 || B.size(0) != cols)
        return refuse(bad_b);
    const int64_t n = B.size(1);
    const at::ScalarType c_type = c_half ? at::kHalf : at::kFloat;
    at::Tensor C;
    if (args[5] != Py_None) {
        if (!THPVariable_Check(args[5])) return refuse("C has the wrong shape, dtype or layout");
        C = THPVariable_Unpack(args[5]);
        if (!C.is_cuda() || C.scalar_type() != c_type || C.dim() != 2 || C.size(0) != rows || C.size(1) != n || C.stride(1) != 1)
            return refuse("C has the wrong shape, dtype or layout");
    }
    void *stream = nullptr;
    if (args[7] != Py_None) {
        stream = PyLong_AsVoidPtr(args[7]);
        if (PyErr_Occurred()) return nullptr;
    }
    if (args[5] == Py_None) C = new_cuda(rows, n, c_type, B);
    if (args[7] == Py_None) stream = c10::cuda::getCurrentCUDAStream(B.get_device()).stream();
    const void *b = B.data_ptr();
    void *c = C.data_ptr();
    const int64_t ldb = B.stride(0), ldc = C.stride(0);
    int st;
    {  // the call waits for the device when a buffer of the plan grows, and for room when the stream's queue is full
        const ThreadsAllowed threads;
        st = b200spmm_spmm(plan, b, ldb, n, c, ldc, c_half ? B200SPMM_C_F16 : B200SPMM_C_F32, stream);
    }
    if (st != B200SPMM_OK) return PyLong_FromLong(st);
    if (args[5] != Py_None) {
        Py_INCREF(args[5]);
        return args[5];
    }
    return THPVariable_Wrap(std::move(C));
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"spmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(spmm)), METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_binding(void) { return PyModule_Create(&module); }
