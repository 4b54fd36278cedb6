// The host side of a product call on device tensors, in native code: torch_ops.product without bias, activation or `out`.
//
// The checks, allocations and argument conversions of a one-row product take 15.5 us of host time a call in Python and ctypes and
// 6.5 here, on the tensors themselves, with output and workspace from torch's allocator and the C ABI called directly. A loop of
// int8 [768, 768] rows went from 15.3 to 6.4 us a call. One of [11008, 4096] rows takes 16.4 either way, also when it is queued
// behind other work: a 14.5 us kernel (graph replay) and what the device leaves between two plain launches.
//
// It takes the plain case only: exact torch tensors (no subclass, no functorch or python-dispatch wrapper) of the storage
// types, contiguous, on the current device, extents that agree, no torch mode active. For anything else it returns None and the
// caller's Python path decides, so refusals keep their exceptions and messages.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <cstdint>
#include <map>

namespace {

constexpr int64_t OP_NN = 0, OP_NT = 1, OP_TN = 2, W_F32 = 0, W_BF16 = 1, W_INT8_EXP = 2, W_INT8_SCALE = 3, PLAN_AUTO = -1;
constexpr int64_t ERR_CAP = 512;

using GemmFn = int64_t (*)(int64_t, void *, float *, const float *, const void *, const void *, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                           void *, int64_t, char *, int64_t);
using NeedFn = int64_t (*)(int64_t, int64_t, int64_t, int64_t, int64_t);
GemmFn g_gemm = nullptr;      // b200i_gemm_w_plan
NeedFn g_auto_need = nullptr; // b200i_product_workspace_bytes
NeedFn g_plan_need = nullptr; // b200i_plan_workspace_bytes
PyObject *g_error = nullptr;  // the package's exception for a refusal

// Workspace sizes by the call's form: a pure function of it and of the device's SM count. Reached with the GIL held; bounded.
std::map<std::array<int64_t, 8>, int64_t> g_need;
constexpr size_t MAX_NEEDS = 4096;

bool plain(PyObject *o, at::Tensor &t) {
    if (!THPVariable_CheckExact(o)) return false;
    t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided) return false;
    const c10::DispatchKeySet keys = t.key_set();
    if (keys.has(c10::DispatchKey::FuncTorchBatched) || keys.has(c10::DispatchKey::FuncTorchGradWrapper) || keys.has(c10::DispatchKey::Batched) ||
        keys.has(c10::DispatchKey::Python) || keys.has(c10::DispatchKey::Negative) || keys.has(c10::DispatchKey::Functionalize) || keys.has(c10::DispatchKey::ZeroTensor))
        return false;
    return t.has_storage() && t.is_contiguous();
}

PyObject *bind(PyObject *, PyObject *args) {
    unsigned long long gemm, auto_need, plan_need;
    PyObject *error;
    if (!PyArg_ParseTuple(args, "KKKO", &gemm, &auto_need, &plan_need, &error)) return nullptr;
    g_gemm = reinterpret_cast<GemmFn>(static_cast<uintptr_t>(gemm));
    g_auto_need = reinterpret_cast<NeedFn>(static_cast<uintptr_t>(auto_need));
    g_plan_need = reinterpret_cast<NeedFn>(static_cast<uintptr_t>(plan_need));
    Py_XINCREF(error);
    Py_XDECREF(g_error);
    g_error = error;
    g_need.clear();
    Py_RETURN_NONE;
}

// product(a, b, bscale or None, wkind, op, plan, group_leaves) -> the output tensor, or None where this is not the plain case
PyObject *product(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    // (a torch mode wants to see the allocations)
    if (nargs != 7 || !g_gemm || c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::PythonTorchFunctionTLS::stack_len() > 0) Py_RETURN_NONE;
    int64_t v[4];
    for (int i = 0; i < 4; i++) {
        if (!PyLong_Check(args[3 + i])) Py_RETURN_NONE;
        v[i] = PyLong_AsLongLong(args[3 + i]);
        if (v[i] == -1 && PyErr_Occurred()) {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
    }
    const int64_t wkind = v[0], op = v[1], plan = v[2], group_leaves = v[3];
    at::Tensor a, b, scale;
    if (!plain(args[0], a) || !plain(args[1], b) || a.dim() != 2 || b.dim() != 2 || a.scalar_type() != at::kFloat) Py_RETURN_NONE;
    const at::ScalarType stored = b.scalar_type();
    const bool int8 = wkind == W_INT8_EXP || wkind == W_INT8_SCALE;
    if (wkind == W_F32 ? stored != at::kFloat
                       : (wkind == W_BF16 ? stored != at::kUInt16 && stored != at::kShort && stored != at::kBFloat16 : !int8 || stored != at::kChar))
        Py_RETURN_NONE;
    const int64_t k = op == OP_TN ? a.size(0) : a.size(1), m = op == OP_TN ? a.size(1) : a.size(0);
    const int64_t n = op == OP_NT ? b.size(0) : b.size(1), k2 = op == OP_NT ? b.size(1) : b.size(0);
    if ((op != OP_NN && op != OP_NT && op != OP_TN) || k != k2 || m <= 0 || n <= 0 || k <= 0) Py_RETURN_NONE;
    if (int8 != (args[2] != Py_None)) Py_RETURN_NONE;
    if (int8 && (!plain(args[2], scale) || scale.scalar_type() != (wkind == W_INT8_EXP ? at::kInt : at::kFloat) || scale.dim() != 1 || scale.size(0) != n ||
                 scale.device() != a.device()))
        Py_RETURN_NONE;
    const c10::Device dev = a.device();
    if (b.device() != dev || c10::cuda::current_device() != dev.index()) Py_RETURN_NONE;

    const std::array<int64_t, 8> form{dev.index(), m, n, k, op, wkind, plan, group_leaves};
    auto found = g_need.find(form);
    if (found == g_need.end()) {
        if (g_need.size() >= MAX_NEEDS) g_need.clear();
        found = g_need.emplace(form, plan == PLAN_AUTO ? g_auto_need(m, n, k, op, wkind) : g_plan_need(m, n, k, plan, group_leaves)).first;
    }
    const int64_t need = found->second;
    at::Tensor out = at::empty({m, n}, a.options().requires_grad(false)), ws;
    if (need > 0) ws = at::empty({need < 16 ? 16 : need}, a.options().requires_grad(false).dtype(at::kByte));
    char message[ERR_CAP] = "";
    int64_t status;
    Py_BEGIN_ALLOW_THREADS;
    status = g_gemm(dev.index(), c10::cuda::getCurrentCUDAStream(dev.index()).stream(), static_cast<float *>(out.data_ptr()),
                    static_cast<const float *>(a.const_data_ptr()), b.const_data_ptr(), int8 ? scale.const_data_ptr() : nullptr, wkind, m, n, k, op, plan, group_leaves,
                    need > 0 ? ws.data_ptr() : nullptr, need, message, ERR_CAP);
    Py_END_ALLOW_THREADS;
    if (status != 0) {
        PyErr_SetString(g_error, message[0] ? message : "b200i_gemm_w_plan failed");
        return nullptr;
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

PyMethodDef METHODS[] = {{"bind", bind, METH_VARARGS, "addresses of the C entry points, and the exception of a refusal"},
                         {"product", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(product)), METH_FASTCALL, "a product of plain device tensors, or None"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef MODULE = {PyModuleDef_HEAD_INIT, "_host_call", "native host side of a product call", -1, METHODS, nullptr, nullptr, nullptr, nullptr};

} // namespace

// BUILT_FOR, of the compiler's command line: the versions of torch and Python whose headers this was compiled with. The package
// does not use a module of others.
PyMODINIT_FUNC PyInit__host_call() {
    PyObject *m = PyModule_Create(&MODULE);
    if (m && PyModule_AddStringConstant(m, "BUILT_FOR", BUILT_FOR) < 0) Py_CLEAR(m);
    return m;
}
