// Python binding of the operators whose kernels take microseconds: argument checks, output, stream and launch in native code.
//
// Written in Python, the checks, a deep-copied configuration and a ctypes call of sixteen arguments cost 25 to 60 us per call, several times
// the kernel.  A function here takes the tensors of an ordinary call, and returns None for everything else (a wrong shape, another dtype,
// a capture without a workspace, ...): the caller then goes its Python way, which raises the error or serves the call.
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TracerMode.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContextLight.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <map>
#include <tuple>
#include <vector>

#include "../../include/lemoq_b200.h"

namespace {

PyObject* none() { Py_RETURN_NONE; }

PyObject* raise(int status) {
    PyObject* type = status == LEMOQ_ERR_INVALID ? PyExc_ValueError : status == LEMOQ_ERR_UNSUPPORTED ? PyExc_NotImplementedError : PyExc_RuntimeError;
    PyErr_SetString(type, lemoq_last_error());
    return nullptr;
}

// The kernels of these calls leave their flags in the device's status word (the calls pass no error word).  A wait that ran out in an earlier
// call has voided its results: that is said here, at the next call, as the CUDA runtime does with errors of its own.
bool healthy() {
    volatile int* word = lemoq_status_word();
    if (!word || !(*word & LEMOQ_FLAG_WAIT_TIMEOUT)) return true;
    *word = *word & ~LEMOQ_FLAG_WAIT_TIMEOUT;
    PyErr_SetString(PyExc_RuntimeError, "a wait ran out in the kernel of an earlier attention, linear or experts call: its results are void");
    return false;
}

// Is the first argument a CUDA tensor?  (Asked before anything that needs a CUDA device.)
bool on_cuda(PyObject* o) { return THPVariable_Check(o) && THPVariable_Unpack(o).is_cuda(); }

// The tensor behind an argument when it is a CUDA tensor of the current device, else null.
const at::Tensor* cuda_tensor(PyObject* o, int device) {
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && t.get_device() == device ? &t : nullptr;
}

// Nothing but the numbers of this call is wanted: no tensor class or mode that has to see the operation, no tangent, no trace, no autocast, no
// gradient.  (The Python ways that remain are made of torch's operators where those matter.)
bool ordinary(PyObject* o, const at::Tensor& x, const at::Tensor& scale) {
    static const c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                              c10::DispatchKey::Functionalize, c10::DispatchKey::ZeroTensor, c10::DispatchKey::Negative});
    return THPVariable_CheckExact(o) && !x.unsafeGetTensorImpl()->key_set().has_any(wrapped) && !x._fw_grad(0).defined() && !scale._fw_grad(0).defined() &&
           !(at::GradMode::is_enabled() && (x.requires_grad() || scale.requires_grad())) && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
           !at::impl::torch_function_mode_enabled() && !at::tracer::impl::is_dispatch_enabled() && !at::autocast::is_autocast_enabled(at::kCUDA);
}
bool aligned(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

bool is(const at::Tensor* t, at::ScalarType type, int dim) { return t && t->scalar_type() == type && t->dim() == dim; }
bool rows(const at::Tensor* t, at::ScalarType type, int dim) { return is(t, type, dim) && t->is_contiguous(); }

at::Tensor fp16(at::IntArrayRef shape, int device) {
    return at::empty(shape, at::TensorOptions().dtype(at::kHalf).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
}

// ---- attention ------------------------------------------------------------------------------------------------------------
// Partials and arrival counters by (device, stream, heads, head_dim, splits).  Launches on one stream are ordered, so they may share; a capture
// gets none from here (its graph would outlive the entry), and the cache is emptied when it has grown to kMostScratch entries.
using ScratchKey = std::tuple<int, void*, int64_t, int64_t, int>;
std::map<ScratchKey, at::Tensor>& scratch() {
    static auto* all = new std::map<ScratchKey, at::Tensor>;
    return *all;
}
constexpr size_t kMostScratch = 64;

void* attn_scratch(int device, const c10::cuda::CUDAStream& stream, int64_t heads, int64_t dim, int splits) {
    const ScratchKey key{device, stream.stream(), heads, dim, splits};
    auto at = scratch().find(key);
    if (at == scratch().end()) {
        if (scratch().size() >= kMostScratch) scratch().clear();
        const auto bytes = static_cast<int64_t>(lemoq_attn_workspace_bytes(static_cast<int>(heads), static_cast<int>(dim), splits));
        at::Tensor t = at::zeros({bytes}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
        at = scratch().emplace(key, std::move(t)).first;
    }
    return at->second.data_ptr();
}

// attention(q, k, ks | None, v, vs | None, filled, scale | None): the default split count, as resolve_num_splits gives it
PyObject* attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 7 || !on_cuda(args[0])) return none();
    if (!healthy()) return nullptr;
    const int device = c10::cuda::current_device();
    const bool int8 = args[2] != Py_None;
    const at::Tensor *q = cuda_tensor(args[0], device), *k = cuda_tensor(args[1], device), *v = cuda_tensor(args[3], device), *filled = cuda_tensor(args[5], device);
    const auto type = int8 ? at::kChar : at::kHalf;
    if (!rows(q, at::kHalf, 4) || !is(k, type, 4) || !is(v, type, 4) || !filled || filled->scalar_type() != at::kInt || filled->numel() != 1) return none();
    const int64_t heads = k->size(1), capacity = k->size(2), dim = k->size(3);
    if (q->size(0) != 1 || q->size(1) != heads || q->size(2) != 1 || q->size(3) != dim || k->size(0) != 1 || k->sizes() != v->sizes()) return none();
    if ((dim != 64 && dim != 128) || heads < 1 || capacity < 1 || k->numel() >= (int64_t(1) << 31)) return none();
    if (k->stride(3) != 1 || v->stride(3) != 1 || k->stride(2) != dim || v->stride(2) != dim || k->stride(1) != v->stride(1) || k->stride(1) < capacity * dim) return none();
    const at::Tensor *ks = nullptr, *vs = nullptr;
    if (int8) {
        ks = cuda_tensor(args[2], device);
        vs = cuda_tensor(args[4], device);
        if (!rows(ks, at::kHalf, 3) || !rows(vs, at::kHalf, 3) || ks->sizes() != k->sizes().slice(0, 3) || vs->sizes() != ks->sizes()) return none();
    }
    double scale = 1.0 / std::sqrt(static_cast<double>(dim));
    if (args[6] != Py_None) {
        scale = PyFloat_AsDouble(args[6]);
        if (scale == -1.0 && PyErr_Occurred()) {
            PyErr_Clear();
            return none();
        }
    }
    const auto stream = c10::cuda::getCurrentCUDAStream();
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return none();
    const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    const int splits = static_cast<int>(std::min<int64_t>(64, std::max<int64_t>(1, (2 * sms + heads - 1) / heads)));
    at::Tensor out = fp16({1, heads, 1, dim}, device);
    void* ws = attn_scratch(device, stream, heads, dim, splits);
    const int S = static_cast<int>(capacity), H = static_cast<int>(heads), D = static_cast<int>(dim);
    const auto* len = static_cast<const int32_t*>(filled->data_ptr());
    const int rc = int8 ? lemoq_attn_decode_int8(q->data_ptr(), static_cast<const int8_t*>(k->data_ptr()), ks->data_ptr(), static_cast<const int8_t*>(v->data_ptr()),
                                                 vs->data_ptr(), k->stride(1), len, out.data_ptr(), H, S, D, splits, static_cast<float>(scale), ws, nullptr, stream.stream())
                        : lemoq_attn_decode_fp16(q->data_ptr(), k->data_ptr(), v->data_ptr(), k->stride(1), len, out.data_ptr(), H, S, D, splits,
                                                 static_cast<float>(scale), ws, nullptr, stream.stream());
    return rc ? raise(rc) : THPVariable_Wrap(out);
}

// ---- W8 linear ------------------------------------------------------------------------------------------------------------
// linear(x (..., K), codes (N, K), scale (N, K / group), group, exact): one token through the GEMV, several through the tensor-core GEMM
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 5 || !on_cuda(args[0])) return none();
    if (!healthy()) return nullptr;
    const int device = c10::cuda::current_device();
    const at::Tensor *x = cuda_tensor(args[0], device), *codes = cuda_tensor(args[1], device), *scale = cuda_tensor(args[2], device);
    if (!x || x->scalar_type() != at::kHalf || x->dim() < 1 || !x->is_contiguous() || !rows(codes, at::kChar, 2) || !rows(scale, at::kHalf, 2)) return none();
    if (!ordinary(args[0], *x, *scale) || !aligned(*x) || !aligned(*codes)) return none();
    const int64_t N = codes->size(0), K = codes->size(1), group = PyLong_AsLongLong(args[3]);
    if (group <= 0 || K % group || scale->size(0) != N || scale->size(1) != K / group || x->size(-1) != K || K == 0 || N == 0) {
        PyErr_Clear();
        return none();
    }
    const int64_t tokens = x->numel() / K;
    if (tokens < 1 || (tokens == 1 ? group % 16 || K > 8192 : K % 128 || group % 128) || tokens > (1 << 22) || N > (1 << 30)) return none();
    c10::DimVector shape(x->sizes().begin(), x->sizes().end());
    shape.back() = N;
    at::Tensor y = fp16(shape, device);
    const auto stream = c10::cuda::getCurrentCUDAStream().stream();
    const auto* w = static_cast<const int8_t*>(codes->data_ptr());
    const int T = static_cast<int>(tokens), n32 = static_cast<int>(N), k32 = static_cast<int>(K), g32 = static_cast<int>(group);
    const int rc = tokens == 1 ? lemoq_dequant_gemv_w8(x->data_ptr(), 1, w, scale->data_ptr(), n32, k32, g32, y.data_ptr(), LEMOQ_DTYPE_F16, stream)
                               : lemoq_w8_gemm(x->data_ptr(), T, w, scale->data_ptr(), n32, k32, g32, nullptr, 1, 0, args[4] == Py_True, nullptr, y.data_ptr(), nullptr, stream);
    return rc ? raise(rc) : THPVariable_Wrap(y);
}

// ---- routed W8 experts ----------------------------------------------------------------------------------------------------
// experts(x (T, H) | (H), gate_up, gate_up_scale, down, down_scale, ids (T, K) | (K), weights, group)
PyObject* experts(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 8 || !on_cuda(args[0])) return none();
    if (!healthy()) return nullptr;
    const int device = c10::cuda::current_device();
    const at::Tensor* a[7];
    for (int i = 0; i < 7; ++i)
        if (!(a[i] = cuda_tensor(args[i], device)) || !a[i]->is_contiguous()) return none();
    const at::Tensor &x = *a[0], &gu = *a[1], &gs = *a[2], &dn = *a[3], &ds = *a[4], &ids = *a[5], &w = *a[6];
    const int64_t group = PyLong_AsLongLong(args[7]);
    if (group <= 0) {
        PyErr_Clear();
        return none();
    }
    if (!is(&gu, at::kChar, 3) || !is(&dn, at::kChar, 3) || !is(&gs, at::kHalf, 3) || !is(&ds, at::kHalf, 3) || x.scalar_type() != at::kHalf ||
        ids.scalar_type() != at::kLong || w.scalar_type() != at::kHalf || (x.dim() != 1 && x.dim() != 2))
        return none();
    const int64_t E = gu.size(0), H = gu.size(2), F = dn.size(2), T = x.dim() == 2 ? x.size(0) : 1;
    if (T < 1 || T > 65535 || x.size(-1) != H || gu.size(1) != 2 * F || dn.size(0) != E || dn.size(1) != H || H % group || F % group ||
        (x.dim() == 2 && (ids.dim() != 2 || ids.size(0) != T || w.sizes() != ids.sizes())) || w.numel() != ids.numel() || gu.numel() >= (int64_t(1) << 31) || gs.numel() * group != gu.numel() || ds.numel() * group != dn.numel())
        return none();
    const int64_t K = ids.numel() / T;
    if (K < 1 || K > 64 || group % 16 || (T > 1 && (H % 128 || F % 128 || group % 128))) return none();
    at::Tensor out = fp16(x.sizes(), device);
    const auto stream = c10::cuda::getCurrentCUDAStream().stream();
    const int t = static_cast<int>(T), k = static_cast<int>(K), e = static_cast<int>(E), h = static_cast<int>(H), f = static_cast<int>(F), g = static_cast<int>(group);
    const auto *gc = static_cast<const int8_t*>(gu.data_ptr()), *dc = static_cast<const int8_t*>(dn.data_ptr());
    const auto* id = static_cast<const int64_t*>(ids.data_ptr());
    int rc;
    if (T == 1) {
        at::Tensor act = fp16({K, F}, device);
        rc = lemoq_moe_grouped_w8(x.data_ptr(), gc, gs.data_ptr(), dc, ds.data_ptr(), id, w.data_ptr(), 1, k, e, h, f, g, act.data_ptr(), out.data_ptr(), nullptr, stream);
    } else {
        const size_t bytes = lemoq_moe_tokens_workspace_bytes(t, k, e, h, f);
        at::Tensor ws = at::empty({static_cast<int64_t>(bytes)}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
        rc = lemoq_moe_tokens_w8(x.data_ptr(), gc, gs.data_ptr(), dc, ds.data_ptr(), id, w.data_ptr(), t, k, e, h, f, g, out.data_ptr(), ws.data_ptr(), bytes, nullptr, stream);
    }
    return rc ? raise(rc) : THPVariable_Wrap(out);
}

// ---- a model's tensors ----------------------------------------------------------------------------------------------------
// pointers(tensors, forms, device): the addresses of the tensors as bytes, 64 bits each (None: 0).  Tensor i has the form forms[i % n], a tuple
// (0 for fp16 or 1 for int8, *sizes).  None when one is not contiguous, 16-byte aligned, of its form and on the device (-1: the CPU).  A prompt
// asks this of some 250 tensors: 2 us here, 200 us as Python expressions.
PyObject* pointers(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 3 || !PyList_Check(args[0]) || !PyTuple_Check(args[1])) return none();
    const Py_ssize_t count = PyList_GET_SIZE(args[0]), period = PyTuple_GET_SIZE(args[1]);
    const long device = PyLong_AsLong(args[2]);
    if (period == 0 || (device == -1 && PyErr_Occurred())) {
        PyErr_Clear();
        return none();
    }
    struct Form {
        at::ScalarType type;
        c10::DimVector sizes;
    };
    std::vector<Form> forms;
    for (Py_ssize_t i = 0; i < period; ++i) {
        PyObject* f = PyTuple_GET_ITEM(args[1], i);
        if (!PyTuple_Check(f) || PyTuple_GET_SIZE(f) < 1) return none();
        Form form;
        for (Py_ssize_t d = 0; d < PyTuple_GET_SIZE(f); ++d) {
            const int64_t v = PyLong_AsLongLong(PyTuple_GET_ITEM(f, d));
            if (v == -1 && PyErr_Occurred()) {
                PyErr_Clear();
                return none();
            }
            if (d == 0) form.type = v ? at::kChar : at::kHalf;
            else form.sizes.push_back(v);
        }
        forms.push_back(std::move(form));
    }
    std::vector<uint64_t> words(static_cast<size_t>(count), 0);
    for (Py_ssize_t i = 0; i < count; ++i) {
        PyObject* o = PyList_GET_ITEM(args[0], i);
        if (o == Py_None) continue;
        if (!THPVariable_Check(o)) return none();
        const at::Tensor& t = THPVariable_Unpack(o);
        const Form& form = forms[static_cast<size_t>(i % period)];
        if (t.scalar_type() != form.type || t.sizes() != at::IntArrayRef(form.sizes) || !t.is_contiguous()) return none();
        if (device < 0 ? !t.device().is_cpu() : !t.is_cuda() || t.get_device() != device) return none();
        words[static_cast<size_t>(i)] = reinterpret_cast<uint64_t>(t.data_ptr());
        if (words[static_cast<size_t>(i)] & 15) return none();
    }
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(words.data()), static_cast<Py_ssize_t>(8 * words.size()));
}

// plain(modules, forwards): True when no module of the list has a forward (pre-)hook, nor a forward of its own other than a bound method of one
// of the functions `forwards`; else None.  (200 modules: 6 us here, 30 us as Python expressions.)
PyObject* plain(PyObject*, PyObject* const* args, Py_ssize_t n) {
    static PyObject *const hooks = PyUnicode_InternFromString("_forward_hooks"), *const pre_hooks = PyUnicode_InternFromString("_forward_pre_hooks"),
                            *const forward = PyUnicode_InternFromString("forward");
    if (n != 2 || !PyList_Check(args[0]) || !PyTuple_Check(args[1]) || !hooks || !pre_hooks || !forward) return none();
    auto is_plain = [&](PyObject* dict) {
        for (PyObject* name : {hooks, pre_hooks}) {
            PyObject* registered = PyDict_GetItemWithError(dict, name);
            if (!registered || !PyDict_Check(registered) || PyDict_Size(registered) != 0) return false;
        }
        PyObject* own = PyDict_GetItemWithError(dict, forward);
        if (!own) return !PyErr_Occurred();
        for (Py_ssize_t j = 0; PyMethod_Check(own) && j < PyTuple_GET_SIZE(args[1]); ++j)
            if (PyMethod_GET_FUNCTION(own) == PyTuple_GET_ITEM(args[1], j)) return true;
        return false;
    };
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(args[0]); ++i) {
        PyObject* dict = PyObject_GenericGetDict(PyList_GET_ITEM(args[0], i), nullptr);
        const bool yes = dict && PyDict_Check(dict) && is_plain(dict);
        Py_XDECREF(dict);
        if (!yes) {
            PyErr_Clear();
            return none();
        }
    }
    Py_RETURN_TRUE;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    try {
        return F(self, args, n);
    } catch (const std::exception& e) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

PyMethodDef kMethods[] = {
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<attention>)), METH_FASTCALL, "decode attention, or None"},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<linear>)), METH_FASTCALL, "W8 linear, or None"},
    {"experts", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<experts>)), METH_FASTCALL, "routed W8 experts, or None"},
    {"pointers", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<pointers>)), METH_FASTCALL, "addresses of tensors of given forms, or None"},
    {"plain", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<plain>)), METH_FASTCALL, "True for modules without hooks, or None"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_bind", "native call path of the lemoq operators", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__bind(void) { return PyModule_Create(&kModule); }
