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
#include <initializer_list>
#include <map>
#include <set>
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

// The first call of a shape goes the Python way, which makes the workspace that captures of the shape take (they take none from here).
bool first_of_shape(int device, int64_t heads, int64_t dim, int splits) {
    static auto* seen = new std::set<std::tuple<int, int64_t, int64_t, int>>;
    return seen->emplace(device, heads, dim, splits).second;
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
    if (first_of_shape(device, heads, dim, splits)) return none();
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

// ---- a whole model ---------------------------------------------------------------------------------------------------------
// A prompt asks about some 250 tensors and 200 modules before it launches anything: 20 us here, 110 us as Python expressions.  Each function
// answers the ordinary case and returns None for anything else; the Python expressions it stands for then decide, and name the reason.
struct Form {
    at::ScalarType type;
    c10::DimVector sizes;
};
// forms: a tuple of tuples (0 for fp16 or 1 for int8, *sizes)
bool read_forms(PyObject* o, std::vector<Form>& forms) {
    if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) == 0) return false;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(o); ++i) {
        PyObject* f = PyTuple_GET_ITEM(o, i);
        if (!PyTuple_Check(f) || PyTuple_GET_SIZE(f) < 1) return false;
        Form form{};
        for (Py_ssize_t d = 0; d < PyTuple_GET_SIZE(f); ++d) {
            const int64_t v = PyLong_AsLongLong(PyTuple_GET_ITEM(f, d));
            if (v == -1 && PyErr_Occurred()) return false;
            if (d == 0) form.type = v ? at::kChar : at::kHalf;
            else form.sizes.push_back(v);
        }
        forms.push_back(std::move(form));
    }
    return true;
}
// The address of a tensor that is contiguous, 16-byte aligned, of the form and on the device (-1: the CPU); 0 for any other.
uint64_t address(PyObject* o, const Form& form, long device) {
    if (!THPVariable_Check(o)) return 0;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (t.scalar_type() != form.type || t.sizes() != at::IntArrayRef(form.sizes) || !t.is_contiguous()) return 0;
    if (device < 0 ? !t.device().is_cpu() : !t.is_cuda() || t.get_device() != device) return 0;
    const auto at = reinterpret_cast<uint64_t>(t.data_ptr());
    return at & 15 ? 0 : at;
}

// pointers(weights, forms, device[, caches, cache_forms]): the addresses as bytes, 64 bits each.  Weight i has the form forms[i % n]; behind every n
// weights come the next m caches (None: 0).  None when a tensor misfits.
PyObject* pointers(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if ((n != 3 && n != 5) || !PyList_Check(args[0]) || (n == 5 && !PyList_Check(args[3]))) return none();
    std::vector<Form> forms, more;
    const long device = PyLong_AsLong(args[2]);
    if ((device == -1 && PyErr_Occurred()) || !read_forms(args[1], forms) || (n == 5 && !read_forms(args[4], more))) {
        PyErr_Clear();
        return none();
    }
    const size_t w = forms.size(), c = more.size(), rounds = static_cast<size_t>(PyList_GET_SIZE(args[0])) / w;
    if (rounds * w != static_cast<size_t>(PyList_GET_SIZE(args[0])) || (c && rounds * c != static_cast<size_t>(PyList_GET_SIZE(args[3])))) return none();
    std::vector<uint64_t> words;
    words.reserve(rounds * (w + c));
    for (size_t r = 0; r < rounds; ++r) {
        for (size_t i = 0; i < w; ++i) {
            words.push_back(address(PyList_GET_ITEM(args[0], static_cast<Py_ssize_t>(r * w + i)), forms[i], device));
            if (!words.back()) return none();
        }
        for (size_t i = 0; i < c; ++i) {
            PyObject* o = PyList_GET_ITEM(args[3], static_cast<Py_ssize_t>(r * c + i));
            words.push_back(o == Py_None ? 0 : address(o, more[i], device));
            if (o != Py_None && !words.back()) return none();
        }
    }
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(words.data()), static_cast<Py_ssize_t>(8 * words.size()));
}

struct Name {
    PyObject* o;
    explicit Name(const char* text) : o(PyUnicode_InternFromString(text)) {}
};
PyObject* item(PyObject* dict, const Name& name) {  // borrowed; null when absent
    PyObject* v = dict && PyDict_Check(dict) ? PyDict_GetItemWithError(dict, name.o) : nullptr;
    if (!v) PyErr_Clear();
    return v;
}
// The attribute dictionaries of objects, held until the end of a call.
struct Dicts {
    std::vector<PyObject*> held;
    PyObject* of(PyObject* o) {
        PyObject* d = o ? PyObject_GenericGetDict(o, nullptr) : nullptr;
        if (d) held.push_back(d);
        else PyErr_Clear();
        return d;
    }
    ~Dicts() {
        for (PyObject* d : held) Py_DECREF(d);
    }
};
bool equal(PyObject* a, PyObject* b) {
    if (!a || !b) return false;
    const int eq = PyObject_RichCompareBool(a, b, Py_EQ);
    if (eq < 0) PyErr_Clear();
    return eq == 1;
}
PyObject* function_of(PyObject* method) { return method && PyMethod_Check(method) ? PyMethod_GET_FUNCTION(method) : nullptr; }

// No forward (pre-)hook on a module, and no forward of its own other than a bound method of one of the functions given.
bool unwatched(PyObject* dict, std::initializer_list<PyObject*> forwards) {
    static const Name hooks("_forward_hooks"), pre_hooks("_forward_pre_hooks"), forward("forward");
    for (const Name* name : {&hooks, &pre_hooks}) {
        PyObject* registered = item(dict, *name);
        if (!registered || !PyDict_Check(registered) || PyDict_Size(registered) != 0) return false;
    }
    PyObject* own = item(dict, forward);
    if (!own) return true;
    for (PyObject* f : forwards)
        if (function_of(own) == f) return true;
    return false;
}

// layers(decoder layers, known, wanted) -> (tensors, linears, unwatched): of every layer the thirteen weights in the order of LayerDesc, the W8 linears
// that a forward of the module tree calls, and whether no module would notice that the tree's forward is left out.  known: (OlmoeDecoderLayer,
// QuantLinear, QuantFusedExperts, OlmoeRMSNorm, decode forward, plain attention forward, silu, fused norm forward, plain norm forward); wanted:
// (group size, eps, top_k, renormalised).  None for a layer that is not of that kind.
PyObject* layers(PyObject*, PyObject* const* args, Py_ssize_t n) {
    static const Name modules("_modules"), buffers("_buffers"), parameters("_parameters"), self_attn("self_attn"), mlp_name("mlp"), o_proj_name("o_proj"),
        packed_qkv("_lemoq_packed_qkv"), original("_lemoq_original_forward"), forward("forward"), groups("num_key_value_groups"), bias("bias"), packed_name("packed"),
        scale("scale"), group_size("group_size"), bits("bits"), experts_name("_static_experts"), act("_static_act"), top_k("_static_top_k"), norm_name("_static_norm"),
        router_name("_static_router"), eps_name("variance_epsilon"), weight("weight"), of_block("of_block");
    static const Name norm_names[4] = {Name("input_layernorm"), Name("post_attention_layernorm"), Name("q_norm"), Name("k_norm")};
    static const Name expert_tensors[4] = {Name("packed_gate_up"), Name("scale_gate_up"), Name("packed_down"), Name("scale_down")};
    static const Name projections[3] = {Name("q_proj"), Name("k_proj"), Name("v_proj")};
    static PyObject *const one = PyLong_FromLong(1), *const eight = PyLong_FromLong(8);
    if (n != 3 || !PyList_Check(args[0]) || !PyTuple_Check(args[1]) || PyTuple_GET_SIZE(args[1]) != 9 || !PyTuple_Check(args[2]) || PyTuple_GET_SIZE(args[2]) != 4) return none();
    auto known = [&](int i) { return PyTuple_GET_ITEM(args[1], i); };
    auto wanted = [&](int i) { return PyTuple_GET_ITEM(args[2], i); };
    auto is_a = [&](PyObject* o, int i) { return o && reinterpret_cast<PyObject*>(Py_TYPE(o)) == known(i); };
    Dicts dicts;
    std::vector<PyObject*> tensors, linears;  // borrowed from the dictionaries
    bool quiet = true;
    for (Py_ssize_t l = 0; l < PyList_GET_SIZE(args[0]); ++l) {
        PyObject* layer = PyList_GET_ITEM(args[0], l);
        if (!is_a(layer, 0)) return none();
        PyObject *own = dicts.of(layer), *parts = item(own, modules), *attn = item(parts, self_attn), *mlp = item(parts, mlp_name);
        PyObject *attn_own = dicts.of(attn), *inner = item(attn_own, modules), *mlp_own = dicts.of(mlp);
        PyObject *packed = dicts.of(item(attn_own, packed_qkv)), *o_proj = item(inner, o_proj_name), *o_own = dicts.of(o_proj), *o_buffers = item(o_own, buffers);
        PyObject *stacks = item(mlp_own, experts_name), *stacks_own = dicts.of(stacks);
        if (!is_a(o_proj, 1) || item(o_buffers, bias) != Py_None || !is_a(stacks, 2) || !equal(item(stacks_own, bits), eight)) return none();
        PyObject* activation = item(mlp_own, act);
        if (activation != Py_None && activation != known(6)) return none();
        PyObject* attn_forward = function_of(item(attn_own, forward));
        if (attn_forward != known(4) || function_of(item(attn_own, original)) != known(5) || !equal(item(attn_own, groups), one)) return none();
        for (PyObject* of : {packed, o_own, stacks_own})
            if (!equal(item(of, group_size), wanted(0))) return none();
        if (!equal(item(mlp_own, top_k), wanted(2)) || !equal(item(mlp_own, norm_name), wanted(3))) return none();
        PyObject* mlp_forward = item(mlp_own, forward);
        PyObject* block = mlp_forward ? PyObject_GetAttr(mlp_forward, of_block.o) : nullptr;
        if (!block) PyErr_Clear();
        quiet = quiet && block == mlp && unwatched(own, {}) && unwatched(attn_own, {known(4)}) && unwatched(o_own, {});
        Py_XDECREF(block);
        if (quiet) {  // (its forward is the block's: looked at above)
            static const Name hooks("_forward_hooks"), pre_hooks("_forward_pre_hooks");
            for (const Name* name : {&hooks, &pre_hooks}) {
                PyObject* registered = item(mlp_own, *name);
                quiet = quiet && registered && PyDict_Check(registered) && PyDict_Size(registered) == 0;
            }
        }
        for (int i = 0; i < 4; ++i) {
            PyObject *norm = item(i < 2 ? parts : inner, norm_names[i]), *norm_own = dicts.of(norm);
            if (!is_a(norm, 3) || !equal(item(norm_own, eps_name), wanted(1))) return none();
            tensors.push_back(item(item(norm_own, parameters), weight));
            quiet = quiet && unwatched(norm_own, {known(7), known(8)});
        }
        tensors.push_back(item(packed, packed_name));
        tensors.push_back(item(packed, scale));
        tensors.push_back(item(o_buffers, packed_name));
        tensors.push_back(item(o_buffers, scale));
        PyObject* router = item(mlp_own, router_name);
        if (!router || !THPVariable_Check(router) || !THPVariable_Unpack(router).is_contiguous()) return none();  // Python lays it out
        tensors.push_back(router);
        for (const Name& name : expert_tensors) tensors.push_back(item(stacks_own, name));
        linears.push_back(o_proj);
        for (const Name& name : projections) {
            PyObject* linear = item(inner, name);
            if (!linear) continue;  // absent where only the stacked rows were kept
            quiet = quiet && is_a(linear, 1) && unwatched(dicts.of(linear), {});
            linears.push_back(linear);
        }
    }
    for (PyObject* t : tensors)
        if (!t || !THPVariable_Check(t)) return none();
    auto list = [](const std::vector<PyObject*>& from) {
        PyObject* to = PyList_New(static_cast<Py_ssize_t>(from.size()));
        for (size_t i = 0; to && i < from.size(); ++i) {
            Py_INCREF(from[i]);
            PyList_SET_ITEM(to, static_cast<Py_ssize_t>(i), from[i]);
        }
        return to;
    };
    PyObject *a = list(tensors), *b = list(linears);
    PyObject* answer = a && b ? PyTuple_Pack(3, a, b, quiet ? Py_True : Py_False) : nullptr;
    Py_XDECREF(a);
    Py_XDECREF(b);
    return answer;
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
    {"layers", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<layers>)), METH_FASTCALL, "weights and linears of decoder layers, or None"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_bind", "native call path of the lemoq operators", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__bind(void) { return PyModule_Create(&kModule); }
