// Host path of the calls whose launches take a few microseconds: argument checks, output allocation and launch in native code.
// Every function serves the plain case (CUDA tensors with storage, contiguous, of the expected types and sizes) and returns None for
// anything else and for a call that the library refuses, without having launched anything: the caller's Python, which repeats the call,
// then raises or handles it as it does without this module.  Errors behind a launch are raised here: the call is not made twice.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include "latentq.h"

namespace {

using at::Tensor;

bool plain(PyObject* o, at::ScalarType dtype) {
    if (!THPVariable_Check(o)) return false;
    const Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.scalar_type() != dtype || !t.has_storage()) return false;
    const c10::DispatchKeySet keys = t.key_set();                    // tensors that stand for others (functorch, __torch_dispatch__)
    return !keys.has(c10::DispatchKey::Python) && !keys.has(c10::DispatchKey::FuncTorchBatched) && !keys.has(c10::DispatchKey::FuncTorchGradWrapper) &&
           !keys.has(c10::DispatchKey::Functionalize) && t.is_contiguous();
}
bool plain_or_none(PyObject* o, at::ScalarType dtype) { return o == Py_None || plain(o, dtype); }
const Tensor& tensor(PyObject* o) { return THPVariable_Unpack(o); }
void* ptr(PyObject* o) { return o == Py_None ? nullptr : tensor(o).data_ptr(); }
// Allocation and launch with the GIL released, as torch.empty and a ctypes call do it: both may wait (cudaMalloc, a full launch queue), and
// what they wait for may need another Python thread.  `f` uses nothing of the arguments' Python objects.
template <typename F> int without_gil(F f) {
    pybind11::gil_scoped_release nogil;
    return f();
}
lq_stream_t stream() { return (lq_stream_t)c10::cuda::getCurrentCUDAStream().stream(); }
// A status other than LQ_OK.  These three are decided before anything is launched; any other is raised as `_lib.check` raises it.
PyObject* refused(const char* name, int rc) {
    if (rc == LQ_EINVAL || rc == LQ_EUNSUPPORTED || rc == LQ_EWORKSPACE) Py_RETURN_NONE;
    PyObject* lib = PyImport_ImportModule("latentq_llm_b200._lib");
    PyObject* r = lib ? PyObject_CallMethod(lib, "check", "si", name, rc) : nullptr;
    if (r) PyErr_Format(PyExc_RuntimeError, "%s failed with status %d", name, rc);
    Py_XDECREF(r); Py_XDECREF(lib);
    return nullptr;
}
bool count(Py_ssize_t n, Py_ssize_t want) {
    if (n == want) return true;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
    return false;
}
PyObject* pair(Tensor a, Tensor b) {
    PyObject* pa = THPVariable_Wrap(std::move(a));
    PyObject* pb = pa ? THPVariable_Wrap(std::move(b)) : nullptr;
    PyObject* r = pb ? PyTuple_Pack(2, pa, pb) : nullptr;
    Py_XDECREF(pa); Py_XDECREF(pb);
    return r;
}

// (grad_input, x, qweight, scales, zeros, bias, N, K, group, workspace, workspace_bytes)
PyObject* w4_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!count(n, 11)) return nullptr;
    const bool dgrad = a[0] == Py_True;
    if (!plain(a[1], at::kBFloat16) || !plain(a[2], at::kChar) || !plain(a[3], at::kBFloat16) || !plain(a[4], at::kBFloat16) || !plain_or_none(a[5], at::kBFloat16) ||
        !plain_or_none(a[9], at::kByte))
        Py_RETURN_NONE;
    const int64_t N = PyLong_AsLongLong(a[6]), K = PyLong_AsLongLong(a[7]), group = PyLong_AsLongLong(a[8]), nb = PyLong_AsLongLong(a[10]);
    if (PyErr_Occurred()) return nullptr;
    const Tensor& x = tensor(a[1]);
    if (x.dim() != 2 || x.size(1) != (dgrad ? N : K) || tensor(a[2]).numel() * 2 != N * K) Py_RETURN_NONE;
    const int64_t M = x.size(0);
    const at::TensorOptions opt = x.options();
    const int8_t* w = (const int8_t*)ptr(a[2]);
    const void *px = ptr(a[1]), *s = ptr(a[3]), *z = ptr(a[4]), *bias = ptr(a[5]);
    void* ws = ptr(a[9]);
    Tensor y;
    const int rc = without_gil([&] {
        y = at::empty({M, dgrad ? K : N}, opt);
        return dgrad ? lq_gemm_a16w4_dgrad(px, w, s, z, y.data_ptr(), M, N, K, (int)group, ws, (size_t)nb, stream())
                     : lq_gemm_a16w4_fwd(px, w, s, z, bias, y.data_ptr(), M, N, K, (int)group, ws, (size_t)nb, stream());
    });
    if (rc != LQ_OK) return refused(dgrad ? "lq_gemm_a16w4_dgrad" : "lq_gemm_a16w4_fwd", rc);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// (x8, w8, row_scale, col_scale, alpha, bias, workspace, workspace_bytes)
PyObject* a8w8_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!count(n, 8)) return nullptr;
    if (!plain(a[0], at::kChar) || !plain(a[1], at::kChar) || !plain_or_none(a[2], at::kFloat) || !plain_or_none(a[3], at::kFloat) || !plain_or_none(a[5], at::kBFloat16) ||
        !plain_or_none(a[6], at::kByte))
        Py_RETURN_NONE;
    const double alpha = PyFloat_AsDouble(a[4]);
    const int64_t nb = PyLong_AsLongLong(a[7]);
    if (PyErr_Occurred()) return nullptr;
    const Tensor &x = tensor(a[0]), &w = tensor(a[1]);
    if (x.dim() != 2 || w.dim() != 2 || x.size(1) != w.size(1)) Py_RETURN_NONE;
    const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
    const at::TensorOptions opt = x.options().dtype(at::kBFloat16);
    const int8_t *px = (const int8_t*)ptr(a[0]), *pw = (const int8_t*)ptr(a[1]);
    const float *row_scale = (const float*)ptr(a[2]), *col_scale = (const float*)ptr(a[3]);
    const void* bias = ptr(a[5]);
    void* ws = ptr(a[6]);
    Tensor y;
    const int rc = without_gil([&] {
        y = at::empty({M, N}, opt);
        return lq_gemm_a8w8(px, pw, row_scale, col_scale, (float)alpha, bias, y.data_ptr(), nullptr, M, N, K, ws, (size_t)nb, stream());
    });
    if (rc != LQ_OK) return refused("lq_gemm_a8w8", rc);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// (x8, w8, clampv, alpha, bias, qscales, workspace, workspace_bytes)
PyObject* a8w8_module(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!count(n, 8)) return nullptr;
    if (!plain(a[0], at::kChar) || !plain(a[1], at::kChar) || !plain_or_none(a[2], at::kFloat) || !plain_or_none(a[4], at::kBFloat16) || !plain(a[5], at::kBFloat16) ||
        !plain_or_none(a[6], at::kByte))
        Py_RETURN_NONE;
    const double alpha = PyFloat_AsDouble(a[3]);
    const int64_t nb = PyLong_AsLongLong(a[7]);
    if (PyErr_Occurred()) return nullptr;
    const Tensor &x = tensor(a[0]), &w = tensor(a[1]);
    if (x.dim() != 2 || w.dim() != 2 || x.size(1) != w.size(1) || tensor(a[5]).numel() != w.size(0) || (a[2] != Py_None && tensor(a[2]).numel() != 1) ||
        (a[4] != Py_None && tensor(a[4]).numel() != w.size(0)))
        Py_RETURN_NONE;
    const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
    const at::TensorOptions opt = x.options().dtype(at::kBFloat16);
    const int8_t *px = (const int8_t*)ptr(a[0]), *pw = (const int8_t*)ptr(a[1]);
    const float* clampv = (const float*)ptr(a[2]);
    const void *bias = ptr(a[4]), *qscales = ptr(a[5]);
    void* ws = ptr(a[6]);
    Tensor y;
    const int rc = without_gil([&] {
        y = at::empty({M, N}, opt);
        return lq_gemm_a8w8_module(px, pw, clampv, (float)alpha, bias, qscales, y.data_ptr(), M, N, K, ws, (size_t)nb, stream());
    });
    if (rc != LQ_OK) return refused("lq_gemm_a8w8_module", rc);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// (x) -> (x8, scale per token)
PyObject* act_quant_per_token(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!count(n, 1)) return nullptr;
    if (!plain(a[0], at::kBFloat16) || tensor(a[0]).dim() != 2) Py_RETURN_NONE;
    const Tensor& x = tensor(a[0]);
    const int64_t M = x.size(0), K = x.size(1);
    const at::TensorOptions opt = x.options();
    const void* px = ptr(a[0]);
    Tensor x8, s;
    const int rc = without_gil([&] {
        x8 = at::empty({M, K}, opt.dtype(at::kChar));
        s = at::empty({M}, opt.dtype(at::kFloat));
        return lq_act_quant_per_token(px, M, K, (int8_t*)x8.data_ptr(), (float*)s.data_ptr(), stream());
    });
    if (rc != LQ_OK) return refused("lq_act_quant_per_token", rc);
    return pair(std::move(x8), std::move(s));
    END_HANDLE_TH_ERRORS
}

// (x) -> (x8, maximum)
PyObject* act_quant_per_tensor(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!count(n, 1)) return nullptr;
    if (!plain(a[0], at::kBFloat16)) Py_RETURN_NONE;
    const Tensor& x = tensor(a[0]);
    const std::vector<int64_t> shape = x.sizes().vec();
    const int64_t numel = x.numel();
    const at::TensorOptions opt = x.options();
    const void* px = ptr(a[0]);
    Tensor x8, c;
    const int rc = without_gil([&] {
        x8 = at::empty(shape, opt.dtype(at::kChar));
        c = at::empty({1}, opt.dtype(at::kFloat));
        return lq_act_quant_per_tensor(px, numel, (float*)c.data_ptr(), (int8_t*)x8.data_ptr(), stream());
    });
    if (rc != LQ_OK) return refused("lq_act_quant_per_tensor", rc);
    return pair(std::move(x8), std::move(c));
    END_HANDLE_TH_ERRORS
}

// (codes, row_scales, clampv): one of the two scales
PyObject* i8_dequant(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (!count(n, 3)) return nullptr;
    const bool rows = a[1] != Py_None;
    if (!plain(a[0], at::kChar) || tensor(a[0]).dim() != 2 || !(rows ? plain(a[1], at::kBFloat16) : plain(a[2], at::kFloat))) Py_RETURN_NONE;
    const Tensor& c = tensor(a[0]);
    if (rows ? tensor(a[1]).numel() != c.size(0) : tensor(a[2]).numel() != 1) Py_RETURN_NONE;
    const int64_t M = c.size(0), N = c.size(1);
    const at::TensorOptions opt = c.options().dtype(at::kBFloat16);
    const int8_t* codes = (const int8_t*)ptr(a[0]);
    const void* row_scales = rows ? ptr(a[1]) : nullptr;
    const float* clampv = rows ? nullptr : (const float*)ptr(a[2]);
    Tensor y;
    const int rc = without_gil([&] {
        y = at::empty({M, N}, opt);
        return lq_i8_dequant(codes, row_scales, clampv, M, N, y.data_ptr(), stream());
    });
    if (rc != LQ_OK) return refused("lq_i8_dequant", rc);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

#define LQ_METHOD(f) {#f, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {LQ_METHOD(w4_gemm), LQ_METHOD(a8w8_gemm), LQ_METHOD(a8w8_module), LQ_METHOD(act_quant_per_token), LQ_METHOD(act_quant_per_tensor),
                         LQ_METHOD(i8_dequant), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_lqhost", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__lqhost() {
    PyObject* m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch_build", LQ_TORCH_BUILD) != 0) { Py_DECREF(m); return nullptr; }   // what it was compiled against
    return m;
}
