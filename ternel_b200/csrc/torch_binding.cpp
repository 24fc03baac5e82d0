// Eager-mode call path of the packed ops: one C function per call, from the Python wrapper straight to
// the C ABI of libternel_b200.so.
//
// A decoded token is hundreds of calls of a few microseconds each, so what the host spends per call is
// what a small product costs. Through torch.library's Python custom op, ctypes and a dozen attribute checks
// in Python a call took 33-48 us of host time, against 6 us on the GPU for a 1024x5120 product; through
// these functions it is an output allocation, the stream lookup and the launch.
//
// A function here serves only the plain case (CUDA tensors without subclass, mode or gradient, right
// dtypes and shapes, contiguous, workspace large enough), in which the dispatcher would do nothing but
// call the CUDA kernel, and returns None for anything else; the caller then takes its ordinary path, which raises
// the proper error or goes through the dispatcher (fake tensors, torch.compile, torch.jit.trace, vmap).
// Arguments of the C ABI are never invented here: a call either matches what that path would have done
// or is left to it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/core/Tensor.h>
#include <ATen/record_function.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/PyInterpreter.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <vector>

#include <cuda_runtime_api.h>

#include "../../include/ternel_b200.h"

namespace {

// Entry points of the library the Python side has loaded (which may be an alternative build).
decltype(&tq1_linear_workspace_bytes) g_workspace_bytes = nullptr;
decltype(&tq1_linear_f16) g_linear = nullptr;
decltype(&tq1_linear_swiglu_f16) g_swiglu = nullptr;
decltype(&tq1_embedding_f16) g_embedding = nullptr;

// The workspaces that the Python side makes and grows, per device one for each stream that has called lately. The table is only
// touched under the GIL; a call takes a reference, because it lets the GIL go while it launches and another thread may
// replace the buffer meanwhile. Never destroyed: at exit the allocator may be gone before it.
constexpr int kMaxDevices = 64;
struct Workspace {
    cudaStream_t stream;
    at::Tensor buffer;
};
std::array<std::vector<Workspace>, kMaxDevices> &g_workspaces = *new std::array<std::vector<Workspace>, kMaxDevices>();

// The buffer for calls on `stream`, undefined where there is none yet (the Python side makes it). Captured calls hold the
// default stream's, which is never given back; the default stream itself cannot be captured.
at::Tensor workspace_of(int device, cudaStream_t stream) {
    if (stream) {
        cudaStreamCaptureStatus status;
        if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) return {};
        if (status != cudaStreamCaptureStatusNone) stream = nullptr;
    }
    for (const Workspace &w : g_workspaces[device])
        if (w.stream == stream) return w.buffer;
    return {};
}

bool plain_cuda(const at::Tensor &t) {
    return t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() && !at::isTensorSubclassLike(t);
}

// Whether packed blocks of the canonical shape; rows and 128-weight groups per row out.
bool canonical_blocks(const at::Tensor &b, int64_t &rows, int64_t &groups) {
    if (b.scalar_type() != at::kByte || b.dim() != 3 || !plain_cuda(b)) return false;
    rows = b.size(0);
    groups = b.size(1);
    return b.size(2) == TQ1_BLOCK_BYTES && rows > 0 && groups > 0 && rows <= INT32_MAX && groups * TQ1_GROUP <= INT32_MAX;
}

// None or torch.float16 / torch.float32; -1 for anything else
int wants_f32(PyObject *dtype) {
    if (dtype == Py_None) return 0;
    if (!THPDtype_Check(dtype)) return -1;
    const at::ScalarType s = reinterpret_cast<THPDtype *>(dtype)->scalar_type;
    return s == at::kHalf ? 0 : s == at::kFloat ? 1 : -1;
}

// Whether the dispatcher has something to do for these arguments before the CUDA kernel: tensors that are not what their
// memory holds (negative views, ...), modes, and what a thread has switched on (tracing, functionalization, transforms, a profiler).
// The outputs here are made without the dispatcher, so a tracer would take them for constants.
bool dispatcher_needed(const at::Tensor &a, const at::Tensor &b) {
    using c10::DispatchKey;
    constexpr c10::DispatchKeySet special(
        {DispatchKey::Python, DispatchKey::Fake, DispatchKey::FuncTorchDynamicLayerBackMode, DispatchKey::Functionalize,
         DispatchKey::Named, DispatchKey::Conjugate, DispatchKey::Negative, DispatchKey::ZeroTensor, DispatchKey::Tracer,
         DispatchKey::FuncTorchBatched, DispatchKey::FuncTorchVmapMode, DispatchKey::Batched, DispatchKey::VmapMode,
         DispatchKey::FuncTorchGradWrapper, DispatchKey::FuncTorchDynamicLayerFrontMode, DispatchKey::PreDispatch,
         DispatchKey::PythonDispatcher});
    const c10::impl::LocalDispatchKeySet local = c10::impl::tls_local_dispatch_key_set();
    return c10::impl::TorchDispatchModeTLS::any_modes_set() ||
           at::getStepCallbacksUnlessEmpty(at::RecordScope::FUNCTION).has_value() ||
           ((a.key_set() | b.key_set() | local.included_) - local.excluded_).has_any(special);
}

PyTypeObject *g_device_context = nullptr;       // torch.utils._device.DeviceContext

// Whether Python wants to see the operation: a TorchFunctionMode other than that of a default device (which looks at
// factory functions alone), or an argument of a subclass, whose __torch_function__ decides what comes back.
bool python_watches(PyObject *a, PyObject *b) {
    if (!THPVariable_CheckExact(a) || !THPVariable_CheckExact(b)) return true;
    if (!at::impl::torch_function_mode_enabled()) return false;
    for (int64_t i = 0; i < at::impl::PythonTorchFunctionTLS::stack_len(); ++i)
        if (Py_TYPE(at::impl::PythonTorchFunctionTLS::get_stack_at(i)->ptr(getPyInterpreter())) != g_device_context) return true;
    return false;
}

// linear(blocks, x, out_dtype, swiglu, flat): x of any leading dimensions (exactly two with `flat`)
PyObject *fast_linear(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 5 || !g_linear || python_watches(args[0], args[1])) Py_RETURN_NONE;
    const at::Tensor &blocks = THPVariable_Unpack(args[0]);
    const at::Tensor &x = THPVariable_Unpack(args[1]);
    const bool swiglu = args[3] == Py_True, flat = args[4] == Py_True;
    const int f32 = wants_f32(args[2]);
    int64_t rows, groups;
    if (f32 < 0 || dispatcher_needed(blocks, x) || !canonical_blocks(blocks, rows, groups)) Py_RETURN_NONE;
    const int64_t columns = groups * TQ1_GROUP, dims = x.dim();
    if (x.scalar_type() != at::kHalf || !plain_cuda(x) || x.device() != blocks.device() || dims < 1 ||
        (flat && dims != 2) || x.size(dims - 1) != columns || x.requires_grad() || (swiglu && rows % 2))
        Py_RETURN_NONE;
    const int64_t batch = x.numel() / columns;
    const int device = x.device().index();
    if (batch <= 0 || batch > INT32_MAX || device < 0 || device >= kMaxDevices) Py_RETURN_NONE;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
    const at::Tensor ws = workspace_of(device, stream);
    const size_t need = g_workspace_bytes((int)batch, (int)rows, (int)columns), have = ws.defined() ? ws.nbytes() : 0;
    if (need > have) Py_RETURN_NONE;
    void *scratch = have ? ws.mutable_data_ptr() : nullptr;
    c10::SmallVector<int64_t, 6> shape(x.sizes().begin(), x.sizes().end());
    shape[dims - 1] = swiglu ? rows / 2 : rows;
    const auto *w = static_cast<const uint8_t *>(blocks.const_data_ptr());
    at::Tensor out;
    int rc;
    {
        // a launch waits while the stream's queue is full, perhaps for work of another thread that needs the GIL
        const pybind11::gil_scoped_release no_gil;
        const c10::cuda::CUDAGuard guard(x.device());
        out = at::detail::empty_cuda(shape, f32 ? at::kFloat : at::kHalf, x.device(), std::nullopt);
        rc = swiglu ? g_swiglu(w, x.const_data_ptr(), out.mutable_data_ptr(), f32, (int)batch, (int)(rows / 2),
                               (int)columns, scratch, have, stream)
                    : g_linear(w, x.const_data_ptr(), out.mutable_data_ptr(), f32, (int)batch, (int)rows,
                               (int)columns, scratch, have, stream);
    }
    if (rc != TQ1_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
}

// embedding(blocks, ids, dtype, flat): ids int64 of any shape (one-dimensional with `flat`)
PyObject *fast_embedding(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 4 || !g_embedding || python_watches(args[0], args[1])) Py_RETURN_NONE;
    const at::Tensor &blocks = THPVariable_Unpack(args[0]);
    const at::Tensor &ids = THPVariable_Unpack(args[1]);
    const bool flat = args[3] == Py_True;
    const int f32 = wants_f32(args[2]);
    int64_t rows, groups;
    if (f32 < 0 || args[2] == Py_None || dispatcher_needed(blocks, ids) || !canonical_blocks(blocks, rows, groups)) Py_RETURN_NONE;
    if (ids.scalar_type() != at::kLong || !plain_cuda(ids) || ids.device() != blocks.device() ||
        (flat && ids.dim() != 1) || ids.numel() <= 0)
        Py_RETURN_NONE;
    c10::SmallVector<int64_t, 6> shape(ids.sizes().begin(), ids.sizes().end());
    shape.push_back(groups * TQ1_GROUP);
    at::Tensor out;
    int rc;
    {
        const pybind11::gil_scoped_release no_gil;
        const c10::cuda::CUDAGuard guard(blocks.device());
        out = at::detail::empty_cuda(shape, f32 ? at::kFloat : at::kHalf, blocks.device(), std::nullopt);
        void *stream = c10::cuda::getCurrentCUDAStream(blocks.device().index()).stream();
        rc = g_embedding(static_cast<const uint8_t *>(blocks.const_data_ptr()), ids.const_data_ptr<int64_t>(),
                         out.mutable_data_ptr(), f32, ids.numel(), rows, (int)(groups * TQ1_GROUP), stream);
    }
    if (rc != TQ1_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(out));
}

// C++ exceptions (an allocation that fails, say) become the Python exceptions torch raises for them.
template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
PyObject *guarded(PyObject *self, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    return F(self, args, nargs);
    END_HANDLE_TH_ERRORS
}

// bind(workspace_bytes, linear, swiglu, embedding, device_context): addresses of the C ABI functions, and the type of the
// mode that a default device puts up
PyObject *bind(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    void *p[4];
    if (nargs != 5 || !PyType_Check(args[4])) {
        PyErr_SetString(PyExc_TypeError, "bind takes four addresses and a type");
        return nullptr;
    }
    Py_INCREF(args[4]);
    g_device_context = reinterpret_cast<PyTypeObject *>(args[4]);
    for (int i = 0; i < 4; ++i) {
        p[i] = PyLong_AsVoidPtr(args[i]);
        if (!p[i] && PyErr_Occurred()) return nullptr;
    }
    g_workspace_bytes = reinterpret_cast<decltype(g_workspace_bytes)>(p[0]);
    g_linear = reinterpret_cast<decltype(g_linear)>(p[1]);
    g_swiglu = reinterpret_cast<decltype(g_swiglu)>(p[2]);
    g_embedding = reinterpret_cast<decltype(g_embedding)>(p[3]);
    Py_RETURN_NONE;
}

// set_workspace(device, stream, tensor): None takes the stream's buffer out of the table
PyObject *set_workspace(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 3 || (args[2] != Py_None && !THPVariable_Check(args[2]))) {
        PyErr_SetString(PyExc_TypeError, "set_workspace takes a device index, a stream and a tensor or None");
        return nullptr;
    }
    const long device = PyLong_AsLong(args[0]);
    const auto stream = static_cast<cudaStream_t>(PyLong_AsVoidPtr(args[1]));
    if (PyErr_Occurred()) return nullptr;
    if (device < 0 || device >= kMaxDevices) Py_RETURN_NONE;
    std::vector<Workspace> &table = g_workspaces[device];
    for (size_t i = 0; i < table.size(); ++i)
        if (table[i].stream == stream) {
            table.erase(table.begin() + i);
            break;
        }
    if (args[2] != Py_None) table.push_back({stream, THPVariable_Unpack(args[2])});
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<fast_linear>)), METH_FASTCALL, nullptr},
    {"embedding", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<fast_embedding>)), METH_FASTCALL, nullptr},
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {"set_workspace", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<set_workspace>)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ternel_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ternel_torch() { return PyModule_Create(&module); }
