// The calls a decode step makes most — quantise the activations, multiply them with packed weights — without the Python around
// them: argument checks, output allocation and the launch through the C ABI in one native function each.  What bounds the
// smallest calls is the host: one token through a quantiser and a 4096 -> 12288 linear is 14 us of GPU work; through the Python of
// flh_b200/_CUDA.py (checks, views, torch.empty, ctypes) it takes 35 us, so 17 (16 tokens through 11008 -> 4096: 42 and 21).
//
// Every function takes the plain case only and returns None for anything else — another type, layout or device than the
// current one, a tensor subclass, a transform, mode or trace that has to see the operations — and the caller then goes the
// way in Python, which has the error messages and the general shapes.  Nothing is kept between calls.
//
// Allocations and launches run without the interpreter's lock: an allocation may free blocks and synchronise, and a launch waits
// while the stream's queue is full, for as long as the GPU takes; other Python threads run meanwhile, among them the one that
// what is queued may be waiting for.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <cmath>

#include "../../include/flh_b200.h"

namespace {

// operations that something other than this process's kernels has to see
bool observed() {
    return at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() || torch::jit::tracer::isTracing();
}
// a contiguous CUDA tensor on `device` (the current one, which is asked for only once a tensor is known to be a CUDA tensor: there may
// be no driver) with memory of its own kind and nothing wrapped around it
bool plain(const at::Tensor &t, c10::DeviceIndex device) {
    if (!t.is_cuda() || t.device().index() != device || t.layout() != at::kStrided || !t.is_contiguous() || t.is_neg() || t.is_conj()) return false;
    const c10::DispatchKeySet ks = t.key_set();
    return !ks.has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::FuncTorchBatched,
                                            c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched, c10::DispatchKey::ZeroTensor}));
}
const at::Tensor *tensor(PyObject *o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

// the interpreter's lock given up for a scope, taken back also where an exception leaves it
struct Unlocked {
    PyThreadState *state = PyEval_SaveThread();
    Unlocked() = default;
    Unlocked(const Unlocked &) = delete;
    ~Unlocked() { PyEval_RestoreThread(state); }
};

PyObject *failed(const char *what, int rc) {
    PyErr_Format(PyExc_RuntimeError, "%s failed (status %d): %s", what, rc, flh_b200_last_error());
    return nullptr;
}
at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Tensor &like) {
    return at::empty(sizes, at::TensorOptions().dtype(type).device(like.device()));
}
// the sizes of x with the last one replaced
c10::SmallVector<int64_t, 6> with_last(const at::Tensor &x, int64_t last) {
    c10::SmallVector<int64_t, 6> s(x.sizes().begin(), x.sizes().end());
    s.back() = last;
    return s;
}

// act_quant_group(x, group_size, hadamard) -> (q, scale)
PyObject *act_quant_group(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const at::Tensor *x = n == 3 ? tensor(args[0]) : nullptr;
    const long gs = x ? PyLong_AsLong(args[1]) : 0;
    const int had = x ? PyObject_IsTrue(args[2]) : 0;
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (!x || !x->is_cuda() || observed() || (gs != 32 && gs != 64 && gs != 128) || x->dim() < 1 || x->scalar_type() != at::kHalf) Py_RETURN_NONE;
    const c10::DeviceIndex dev = c10::cuda::current_device();
    const int64_t K = x->size(-1);
    if (!plain(*x, dev) || x->numel() == 0 || K % gs) Py_RETURN_NONE;
    const at::Tensor in = *x;
    const void *in_p = in.data_ptr();
    at::Tensor q, s;
    int rc;
    // torch divides a CUDA tensor by a number by multiplying with the number's reciprocal, rounded to binary32
    const float factor = had ? 1.0f / (float)std::sqrt((double)gs) : 1.0f;
    {
        const Unlocked unlocked;
        q = empty(with_last(in, K / 2), at::kByte, in);
        s = empty(with_last(in, K / gs), at::kHalf, in);
        rc = flh_b200_quant_group_sym_scaled_i4(in_p, in.numel() / gs, (int)gs, had, factor, static_cast<uint8_t *>(q.data_ptr()), s.data_ptr(),
                                                c10::cuda::getCurrentCUDAStream(dev).stream());
    }
    if (rc) return failed("quant_group_sym_i4", rc);
    return Py_BuildValue("(NN)", THPVariable_Wrap(std::move(q)), THPVariable_Wrap(std::move(s)));
    END_HANDLE_TH_ERRORS
}

// act_quant_token(x, hadamard, clip, kfac, sign table or None) -> (q, scale, zero)
PyObject *act_quant_token(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    const at::Tensor *x = n == 5 ? tensor(args[0]) : nullptr;
    const at::Tensor *bits = x ? tensor(args[4]) : nullptr;
    const int had = x ? PyObject_IsTrue(args[1]) : 0;
    const double clip = x ? PyFloat_AsDouble(args[2]) : 0;
    const long kfac = x ? PyLong_AsLong(args[3]) : 0;
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (!x || !x->is_cuda() || (!bits && args[4] != Py_None) || observed() || x->dim() < 1) Py_RETURN_NONE;
    if (x->scalar_type() != at::kHalf && x->scalar_type() != at::kBFloat16) Py_RETURN_NONE;
    const c10::DeviceIndex dev = c10::cuda::current_device();
    if (!plain(*x, dev) || x->numel() == 0) Py_RETURN_NONE;
    const at::Tensor in = *x, table = bits ? *bits : at::Tensor();
    const void *in_p = in.data_ptr();
    const uint32_t *table_p = bits ? static_cast<const uint32_t *>(table.data_ptr()) : nullptr;
    const int64_t K = in.size(-1);
    at::Tensor q, s, z;
    int rc;
    {
        const Unlocked unlocked;
        const auto one = with_last(in, 1);
        q = empty(with_last(in, K / 2), at::kByte, in);
        s = empty(one, at::kHalf, in);
        z = empty(one, at::kHalf, in);
        rc = flh_b200_quant_token_asym_i4(in_p, in.scalar_type() == at::kBFloat16 ? FLH_B200_BF16 : FLH_B200_F16, in.numel() / K, K, K, had ? 1 : 0,
                                          (int)kfac, table_p, (float)clip, static_cast<uint8_t *>(q.data_ptr()), s.data_ptr(), z.data_ptr(),
                                          c10::cuda::getCurrentCUDAStream(dev).stream());
    }
    if (rc) return failed("quant_token_asym_i4", rc);
    return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(q)), THPVariable_Wrap(std::move(s)), THPVariable_Wrap(std::move(z)));
    END_HANDLE_TH_ERRORS
}

// gemm(x, w, a_scale, a_zero, w_scale, rowsum, bias, bfloat16, algo, workspace) -> y: algo and workspace as the plan of
// flh_b200/_CUDA.py names them, the workspace a tensor, the bytes of scratch that this call alone uses, or None.
// x [.., K / 2], w flat or [N, K / 2].
PyObject *gemm(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 10) Py_RETURN_NONE;
    const at::Tensor *t[7];
    for (int i = 0; i < 7; ++i) {
        t[i] = tensor(args[i]);
        if (!t[i] && (args[i] != Py_None || i < 3 || i == 4)) Py_RETURN_NONE;
    }
    const at::Tensor *ws = tensor(args[9]);
    const long scratch = PyLong_Check(args[9]) ? PyLong_AsLong(args[9]) : 0;
    const int bf16 = PyObject_IsTrue(args[7]);
    const long algo = PyLong_AsLong(args[8]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if ((!ws && !PyLong_Check(args[9]) && args[9] != Py_None) || observed()) Py_RETURN_NONE;
    const at::Tensor &x = *t[0], &w = *t[1], &sa = *t[2], &sb = *t[4];
    if (!x.is_cuda()) Py_RETURN_NONE;
    const c10::DeviceIndex dev = c10::cuda::current_device();
    for (int i = 0; i < 7; ++i)
        if (t[i] && !plain(*t[i], dev)) Py_RETURN_NONE;
    if (x.dim() < 1 || sb.dim() != 2 || x.numel() == 0 || sb.numel() == 0) Py_RETURN_NONE;
    const int64_t K = 2 * x.size(-1), M = x.numel() / x.size(-1), N = sb.size(0);
    if (sa.numel() == 0 || sa.numel() % M || w.numel() != N * (K / 2)) Py_RETURN_NONE;
    const int64_t ga = sa.numel() / M, gb = sb.size(1);
    if (K % ga || K % gb || x.scalar_type() != at::kByte || w.scalar_type() != at::kByte || sa.scalar_type() != at::kHalf ||
        sb.scalar_type() != at::kHalf || (t[3] && (t[3]->scalar_type() != at::kHalf || t[3]->numel() != sa.numel())) ||
        (t[5] && t[5]->scalar_type() != at::kInt) || (t[6] && (t[6]->scalar_type() != at::kHalf || t[6]->numel() != N)))
        Py_RETURN_NONE;
    at::Tensor held[8], y, own;                                  // the operands and the workspace stay alive while the lock is given up
    void *ptr[8] = {};
    for (int i = 0; i < 7; ++i)
        if (t[i]) { held[i] = *t[i]; ptr[i] = t[i]->data_ptr(); }
    size_t ws_bytes = 0;
    if (ws) { held[7] = *ws; ptr[7] = ws->data_ptr(); ws_bytes = (size_t)ws->numel(); }
    int rc;
    bool fits = true;
    {
        const Unlocked unlocked;
        y = empty(with_last(held[0], N), bf16 ? at::kBFloat16 : at::kHalf, held[0]);
        if (scratch > 0) {
            try {
                own = empty({(int64_t)scratch}, at::kByte, held[0]);     // freed in stream order when the call returns
                ptr[7] = own.data_ptr();
                ws_bytes = (size_t)scratch;
            } catch (const c10::OutOfMemoryError &) {
                fits = false;                                    // AUTO has a kernel that needs none
            }
        }
        rc = !fits ? 0 : flh_b200_gemm_i4_dequant(
            static_cast<const uint8_t *>(ptr[0]), static_cast<const uint8_t *>(ptr[1]), ptr[2], ptr[3], ptr[4], static_cast<const int32_t *>(ptr[5]),
            ptr[6], y.data_ptr(), M, N, K, K / ga, K / gb, bf16 ? FLH_B200_BF16 : FLH_B200_F16, (int)algo, ptr[7], ws_bytes,
            c10::cuda::getCurrentCUDAStream(dev).stream());
    }
    if (!fits) Py_RETURN_NONE;
    if (rc) return failed("gemm_i4_dequant", rc);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// square(x) -> x * x in binary32, for values that no derivative is taken of
PyObject *square(PyObject *, PyObject *x_) {
    HANDLE_TH_ERRORS
    const at::Tensor *x = tensor(x_);
    if (!x || !x->is_cuda() || observed() || (x->scalar_type() != at::kHalf && x->scalar_type() != at::kBFloat16)) Py_RETURN_NONE;
    const c10::DeviceIndex dev = c10::cuda::current_device();
    if (!plain(*x, dev) || x->numel() % 8 || reinterpret_cast<uintptr_t>(x->data_ptr()) % 16) Py_RETURN_NONE;
    if ((c10::GradMode::is_enabled() && x->requires_grad()) || x->_fw_grad(0).defined()) Py_RETURN_NONE;
    const at::Tensor in = *x;
    const void *in_p = in.data_ptr();
    at::Tensor y;
    int rc;
    {
        const Unlocked unlocked;
        y = empty(in.sizes(), at::kFloat, in);
        rc = flh_b200_square_f32(in_p, in.scalar_type() == at::kBFloat16 ? FLH_B200_BF16 : FLH_B200_F16, in.numel(), y.data_ptr(),
                                 c10::cuda::getCurrentCUDAStream(dev).stream());
    }
    if (rc) return failed("square_f32", rc);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"square", square, METH_O, nullptr},
    {"act_quant_group", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(act_quant_group)), METH_FASTCALL, nullptr},
    {"act_quant_token", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(act_quant_token)), METH_FASTCALL, nullptr},
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(gemm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// torch_version: what the tensors' layout was compiled against; flh_b200/_CUDA.py uses the module under that version only
PyMODINIT_FUNC PyInit__host(void) {
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch_version", FLH_TORCH) < 0) { Py_DECREF(m); return nullptr; }
    return m;
}
