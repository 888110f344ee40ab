// Host side of one linear layer: what stands between a Python call and the kernel launches of the C interface, in one
// native call (Python: fp6_llm_b200._native.host()).
//
// Checking the tensors, taking the stream, allocating output and workspace and passing 14 arguments through ctypes took
// 20 - 33 us a layer in Python, more than the layer's kernels up to ~100 tokens of a 7B model: its decode block at one token
// took 135 us a pass for 37 us of kernels.  Here a layer costs about its launches.
//
// A function of this module either does the whole call or returns NotImplemented and has done nothing: anything out of the
// ordinary (tensor subclasses, functorch wrappers, tensors that are not laid out as the kernels read them, every invalid
// argument) is left to the Python form of the same operator, which converts or raises.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TracerMode.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/DispatchKeySet.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>
#include <vector>

#include "../../include/fp6_llm_b200.h"

namespace {

constexpr int kSiluMul = FP6B200_ACT_SILU_MUL;

// The wrappers a tensor of the exact type may still stand for: they have no memory of their own.
const c10::DispatchKeySet kWrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                    c10::DispatchKey::Batched, c10::DispatchKey::Functionalize, c10::DispatchKey::Negative,
                                    c10::DispatchKey::Conjugate, c10::DispatchKey::ZeroTensor});

// a contiguous CUDA tensor of this type, on `device` unless that is -1
const at::Tensor* plain(PyObject* o, at::ScalarType type, int device) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || t.scalar_type() != type || !t.is_cuda() || t.layout() != at::kStrided || t.key_set().has_any(kWrapped) ||
        !t.is_contiguous() || (device >= 0 && t.get_device() != device))
        return nullptr;
    return &t;
}

bool whole(PyObject* o, long* v) {
    if (!PyLong_Check(o)) return false;
    *v = PyLong_AsLong(o);
    if (*v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

struct Call {
    int e = 0, m = 0, activation = 0;
    const at::Tensor *x = nullptr, *weight = nullptr, *native = nullptr, *scales = nullptr, *bias = nullptr;
};

// The workspace of one call, allocated when it is asked for.  Called from C: an exception waits in `failed`.
struct Workspace {
    at::TensorOptions options;
    at::Tensor memory;
    std::exception_ptr failed;
    bool full = false;   // it was: no memory left
    static void* get(void* self, size_t bytes) noexcept {
        Workspace* w = static_cast<Workspace*>(self);
        try {
            w->memory = at::empty({(int64_t)bytes}, w->options);
            return w->memory.data_ptr();
        } catch (const c10::OutOfMemoryError&) {
            w->failed = std::current_exception();
            w->full = true;
            return nullptr;
        } catch (...) {
            w->failed = std::current_exception();
            return nullptr;
        }
    }
};

PyObject* fail(const char* what, int rc) {
    const char* msg = fp6b200_error_string(rc);
    PyErr_Format(PyExc_RuntimeError, "%s failed: CUDA error %d (%s)", what, rc, msg ? msg : "?");
    return nullptr;
}

PyObject* not_mine() { Py_RETURN_NOTIMPLEMENTED; }

// Runs a call whose tensors are plain.  last_dim_only: x is [..., IC] and the result [..., OC]; otherwise x is [B, IC].
PyObject* run(const Call& c, bool last_dim_only) {
    const at::Tensor& x = *c.x;
    const int64_t dim = x.dim();
    if (dim < 1 || (!last_dim_only && dim != 2)) return not_mine();
    const int64_t ic = x.size(dim - 1), oc = c.scales->numel();
    if (ic < 64 || ic % 64 || oc < 256 || oc % 256) return not_mine();
    const int64_t batch = x.numel() / ic;
    if (batch < 1) return not_mine();
    if (c.activation != 0 && c.activation != kSiluMul) return not_mine();
    if (c.bias && c.bias->numel() != oc) return not_mine();
    if (c.native) {
        if (!fp6b200_native_supported(c.e, c.m, oc, batch, ic) || (size_t)c.native->numel() != fp6b200_native_weight_bytes(oc, ic))
            return not_mine();
    } else {
        const at::Tensor& w = *c.weight;
        if (w.dim() != 2 || w.size(0) != oc || w.size(1) * 32 != ic * (1 + c.e + c.m)) return not_mine();
    }
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    c10::DimVector sizes(x.sizes());
    sizes[dim - 1] = c.activation == kSiluMul ? oc / 2 : oc;
    at::Tensor out = at::empty(sizes, at::TensorOptions().device(x.device()).dtype(at::kHalf));
    // The workspace goes back to the allocator when this returns; the stream orders whoever gets it next behind these kernels.
    Workspace ws{at::TensorOptions().device(x.device()).dtype(at::kByte), {}, nullptr, false};
    void* stream = c10::cuda::getCurrentCUDAStream(x.get_device()).stream();
    const void* bias = c.bias ? c.bias->data_ptr() : nullptr;
    void *xp = x.data_ptr(), *op = out.data_ptr(), *sp = c.scales->data_ptr();
    void* wp = c.native ? c.native->data_ptr() : c.weight->data_ptr();
    void* planes = c.native ? Workspace::get(&ws, fp6b200_native_workspace_bytes(batch, ic)) : nullptr;
    int rc = 0;
    Py_BEGIN_ALLOW_THREADS   // a full launch queue blocks
    if (!c.native) {
        rc = fp6b200_linear_scratch(c.e, c.m, stream, wp, sp, xp, op, oc, batch, ic, &Workspace::get, &ws, bias, c.activation);
        if (ws.full) {   // nothing was launched: the call runs as one that offers no workspace
            ws.failed = nullptr;
            rc = fp6b200_linear_ex(c.e, c.m, stream, wp, sp, xp, op, oc, batch, ic, nullptr, 1, bias, c.activation);
        }
    } else if (planes) {
        rc = fp6b200_linear_native(c.e, c.m, stream, wp, sp, xp, op, oc, batch, ic, planes, bias, c.activation);
    }
    Py_END_ALLOW_THREADS
    if (ws.failed) std::rethrow_exception(ws.failed);
    if (rc != 0) return fail(c.native ? "fp6b200_linear_native" : "fp6b200_linear", rc);
    return THPVariable_Wrap(std::move(out));
}

// format, activations, scales, bias and activation, which every form has; false: not for this module
bool common(Call* c, PyObject* e, PyObject* m, PyObject* x, PyObject* scales, PyObject* bias, PyObject* activation) {
    long ev, mv, av;
    if (!whole(e, &ev) || !whole(m, &mv) || !whole(activation, &av)) return false;
    if (ev < 0 || ev > 7 || mv < 0 || mv > 7 || av < 0 || av > 7 || !fp6b200_native_supported((int)ev, (int)mv, 256, 1, 64)) return false;
    c->e = (int)ev;
    c->m = (int)mv;
    c->activation = (int)av;
    if (!(c->x = plain(x, at::kHalf, -1))) return false;
    const int device = c->x->get_device();
    if (!(c->scales = plain(scales, at::kHalf, device))) return false;
    return bias == Py_None || (c->bias = plain(bias, at::kHalf, device));
}

// linear(e, m, x, packed, scales, split_k, bias, activation); split_k is checked, how K is split is the library's choice
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Call c;
    long split;
    if (n != 8 || !whole(a[5], &split) || split < 0 || split > 65535 || !common(&c, a[0], a[1], a[2], a[4], a[6], a[7])) return not_mine();
    if (!(c.weight = plain(a[3], at::kInt, c.x->get_device()))) return not_mine();
    return run(c, false);
    END_HANDLE_TH_ERRORS
}

// native(e, m, x, tiles, scales, bias, activation)
PyObject* native(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Call c;
    if (n != 7 || !common(&c, a[0], a[1], a[2], a[4], a[5], a[6])) return not_mine();
    if (!(c.native = plain(a[3], at::kByte, c.x->get_device()))) return not_mine();
    return run(c, false);
    END_HANDLE_TH_ERRORS
}

// layer(e, m, x, packed, tiles or None, scales, split_k, bias, activation): the modules' forward, x of any rank; the tile
// layout is taken when the library prefers it for this batch and split_k is 0, which is all that split_k says
PyObject* layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Call c;
    long split;
    if (n != 9 || !whole(a[6], &split) || split < 0 || split > 65535 || !common(&c, a[0], a[1], a[2], a[5], a[7], a[8])) return not_mine();
    const int device = c.x->get_device();
    if (!(c.weight = plain(a[3], at::kInt, device))) return not_mine();
    const int64_t dim = c.x->dim(), oc = c.scales->numel();
    const int64_t ic = dim ? c.x->size(dim - 1) : 0;
    if (ic < 64 || c.weight->dim() != 2 || c.weight->size(0) != oc || c.weight->size(1) * 32 != ic * (1 + c.e + c.m)) return not_mine();
    if (a[4] != Py_None && split == 0 && fp6b200_native_preferred(c.e, c.m, oc, c.x->numel() / ic, ic)) {
        if (!(c.native = plain(a[4], at::kByte, device))) return not_mine();
    }
    return run(c, true);
    END_HANDLE_TH_ERRORS
}

// a contiguous fp16 CPU tensor
const at::Tensor* plain_host(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || t.scalar_type() != at::kHalf || !t.is_cpu() || t.layout() != at::kStrided || t.key_set().has_any(kWrapped) ||
        !t.is_contiguous())
        return nullptr;
    return &t;
}

// host_batch([(e, m, act_host, packed, scales, out_host, split_k[, tiles or None]), ...]) -> True.  The first copy of a batch can
// start only when all its calls are laid out: in Python that took longer than the copy.
PyObject* host_batch(PyObject*, PyObject* calls) {
    HANDLE_TH_ERRORS
    if (!PyList_CheckExact(calls) || PyList_GET_SIZE(calls) < 1 || PyList_GET_SIZE(calls) > 4096) return not_mine();
    std::vector<fp6b200_host_call> batch((size_t)PyList_GET_SIZE(calls));
    int device = -1;
    for (size_t i = 0; i < batch.size(); i++) {
        PyObject* c = PyList_GET_ITEM(calls, (Py_ssize_t)i);
        if (!PyTuple_CheckExact(c) || PyTuple_GET_SIZE(c) < 7 || PyTuple_GET_SIZE(c) > 8) return not_mine();
        long e, m, split;
        if (!whole(PyTuple_GET_ITEM(c, 0), &e) || !whole(PyTuple_GET_ITEM(c, 1), &m) || !whole(PyTuple_GET_ITEM(c, 6), &split)) return not_mine();
        if (e < 0 || e > 7 || m < 0 || m > 7 || split < 0 || split > 65535 || !fp6b200_native_supported((int)e, (int)m, 256, 1, 64)) return not_mine();
        const at::Tensor* packed = plain(PyTuple_GET_ITEM(c, 3), at::kInt, device);
        if (!packed || packed->dim() != 2) return not_mine();
        device = packed->get_device();
        const at::Tensor* scales = plain(PyTuple_GET_ITEM(c, 4), at::kHalf, device);
        const at::Tensor *act = plain_host(PyTuple_GET_ITEM(c, 2)), *out = plain_host(PyTuple_GET_ITEM(c, 5)), *tiles = nullptr;
        if (!scales || !act || !out || act->dim() != 2 || out->dim() != 2) return not_mine();
        if (PyTuple_GET_SIZE(c) == 8 && PyTuple_GET_ITEM(c, 7) != Py_None && !(tiles = plain(PyTuple_GET_ITEM(c, 7), at::kByte, device)))
            return not_mine();
        const int64_t tokens = act->size(0), ic = act->size(1), oc = packed->size(0);
        if (packed->size(1) * 32 != ic * (1 + e + m) || scales->numel() != oc || out->size(0) != tokens || out->size(1) != oc) return not_mine();
        // tiles that this call would read past the end of
        if (tiles && split == 0 && fp6b200_native_preferred((int)e, (int)m, oc, tokens, ic) &&
            (size_t)tiles->numel() < fp6b200_native_weight_bytes(oc, ic))
            return not_mine();
        batch[i] = {(int)e, (int)m, packed->data_ptr(), scales->data_ptr(), act->data_ptr(), out->data_ptr(), (size_t)oc, (size_t)tokens,
                    (size_t)ic, (int)split, tiles ? tiles->data_ptr() : nullptr};
    }
    const c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, (c10::DeviceIndex)device));
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fp6b200_linear_host_io_batch(batch.data(), (int)batch.size());
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail("fp6b200_linear_host_io_batch", rc);
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// unwatched(t): ops.is_plain_memory without its calls into Python, which took 3 us of the 80 of a small layer's loading
PyObject* unwatched(PyObject*, PyObject* o) {
    HANDLE_TH_ERRORS
    if (at::impl::PythonTorchFunctionTLS::stack_len() != 0) return not_mine();   // which modes these are is known in Python
    if (!THPVariable_CheckExact(o)) Py_RETURN_FALSE;
    const at::Tensor& t = THPVariable_Unpack(o);
    const bool watched = t.key_set().has_any(kWrapped) || (t.requires_grad() && c10::GradMode::is_enabled()) || t._fw_grad(0).defined() ||
                         c10::impl::TorchDispatchModeTLS::any_modes_set() || at::tracer::impl::is_dispatch_enabled();
    return PyBool_FromLong(!watched);
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"unwatched", unwatched, METH_O, nullptr},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(linear)), METH_FASTCALL, nullptr},
    {"native", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(native)), METH_FASTCALL, nullptr},
    {"layer", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(layer)), METH_FASTCALL, nullptr},
    {"host_batch", host_batch, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "fp6_b200_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_fp6_b200_host(void) { return PyModule_Create(&module); }
