// The torch.ops.xg_sm100.* operators: schemas, and their CUDA kernels as native code.
//
// Each kernel checks its tensors, allocates the outputs, and hands pointers, extents and the current stream to the C ABI of
// libxg_sm100.so; no arithmetic happens here. What bounds a small call is the host: the same marshalling as Python code
// behind torch.library.custom_op took 31 us (RMSNorm) to 46 us (split-K dense layer) a call on the B200 box, several times
// the kernel's own duration, so every operator that a compiled graph calls in its hot path lives here. Fake implementations
// (shape propagation) stay in ops.py; there is no CPU implementation on purpose.
//
// Observers (lib.call_hook) see the calls made from here as well: while a hook is set, every C-ABI call is reported to it
// with its arguments in the header's order.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include <atomic>
#include <cmath>
#include <cstdlib>
#include <initializer_list>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "../../include/xg_sm100.h"

// ---- routing rules, also asked by ops.py for the graph rewrites -------------------------------------
// fp32 dense layers above this many FLOPs run on the bf16 tensor cores from three bf16 planes per operand (fp32-grade results at
// several times the FMA rate); smaller ones stay on the FMA kernel, whose launch is cheaper. ops.F32_TENSOR_MIN_FLOPS sets it.
extern "C" {
int64_t xg_torch_f32_min_flops = []() {
    const char* set = std::getenv("XG_F32_TENSOR_MIN_FLOPS");
    return set ? (int64_t)std::atoll(set) : (int64_t)1 << 30;
}();
int64_t xg_torch_f32_max_k = 8192;  // measured error vs fp64 grows from 2e-6 (K = 1728) to 6e-6 (K = 4096) of the output scale
}

extern "C" int xg_torch_f32_on_tensor_cores(int64_t M, int64_t N, int64_t K) {
    if (2 * M * N * K < xg_torch_f32_min_flops || K > xg_torch_f32_max_k) return 0;
    const char* e = std::getenv("XG_F32_TENSOR");
    return !(e && e[0] == '0' && e[1] == 0);
}

// The one-launch FMA tower (dims: layers + 1 widths) is the faster form where a launch per layer is mostly launch and latency: few
// rows, or very narrow layers (figures: ops.mlp_small_worth_it).
extern "C" int xg_torch_small_tower_worth_it(int64_t M, const int64_t* dims, int layers, int dtype) {
    if (!xg_mlp_small_supported(dims, layers, dtype)) return 0;
    int64_t weights = 0;
    for (int l = 0; l < layers; ++l) weights += (dims[l] + 3) / 4 * 4 * dims[l + 1];
    return M <= 2048 || weights <= 4096;
}

namespace {

using at::Tensor;
using std::optional;
template <typename T>
using Buf = c10::SmallVector<T, 32>;

// ---- Python side: errors and observers -----------------------------------------------------------
struct Gil {
    PyGILState_STATE s = PyGILState_Ensure();
    ~Gil() { PyGILState_Release(s); }
};

[[noreturn]] void throw_python_error() {
    python_error e;
    e.persist();
    throw std::move(e);
}

// XgLibraryError, as lib.check raises it
[[noreturn]] void raise_library_error(const char* what, int rc) {
    Gil gil;
    const char* msg = xg_last_error();
    PyObject* mod = PyImport_ImportModule("xpu_graph_b200.lib");
    PyObject* names = mod ? PyObject_GetAttrString(mod, "ERR_NAMES") : nullptr;
    PyObject* type = mod ? PyObject_GetAttrString(mod, "XgLibraryError") : nullptr;
    PyObject* key = PyLong_FromLong(rc);
    PyObject* name = names ? PyDict_GetItem(names, key) : nullptr;
    if (type) PyErr_Format(type, "%s failed: %S: %s", what, name ? name : key, msg ? msg : "");
    Py_XDECREF(key);
    Py_XDECREF(names);
    Py_XDECREF(type);
    Py_XDECREF(mod);
    throw_python_error();
}

PyObject* g_before = nullptr;  // observers, guarded by the GIL
PyObject* g_after = nullptr;
std::atomic<bool> g_hooked{false};

PyObject* to_py(const void* p) { return p ? PyLong_FromVoidPtr(const_cast<void*>(p)) : Py_NewRef(Py_None); }
PyObject* to_py(int64_t v) { return PyLong_FromLongLong(v); }
PyObject* to_py(int v) { return PyLong_FromLong(v); }
PyObject* to_py(float v) { return PyFloat_FromDouble(v); }

void report(PyObject* fn, const char* name, PyObject* args, const int* rc) {
    if (!fn) return;
    PyObject* res = rc ? PyObject_CallFunction(fn, "sOi", name, args, *rc) : PyObject_CallFunction(fn, "sO", name, args);
    if (!res) throw_python_error();
    Py_DECREF(res);
}

template <typename... P, typename... A>
int observed_call(const char* name, int (*fn)(P...), A... a) {
    Gil gil;
    PyObject* args = PyTuple_New(sizeof...(A));
    Py_ssize_t i = 0;
    (PyTuple_SET_ITEM(args, i++, to_py(static_cast<P>(a))), ...);
    report(g_before, name, args, nullptr);
    const int rc = fn(static_cast<P>(a)...);
    report(g_after, name, args, &rc);
    Py_DECREF(args);
    return rc;
}

template <typename... P, typename... A>
void call(const char* name, int (*fn)(P...), A... a) {
    const int rc = g_hooked.load(std::memory_order_relaxed) ? observed_call(name, fn, a...) : fn(static_cast<P>(a)...);
    if (C10_UNLIKELY(rc != XG_OK)) raise_library_error(name, rc);
}
#define XG_CALL(fn, ...) call(#fn, fn, __VA_ARGS__)

// ---- tensors ---------------------------------------------------------------------------------------
int code_of(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return XG_F32;
        case at::kBFloat16: return XG_BF16;
        case at::kHalf: return XG_F16;
        default: TORCH_CHECK_TYPE(false, "xg_sm100: unsupported dtype ", t);
    }
}

int act_code(c10::string_view a) {
    if (a == "none") return XG_ACT_NONE;
    if (a == "gelu") return XG_ACT_GELU;
    if (a == "relu") return XG_ACT_RELU;
    if (a == "silu") return XG_ACT_SILU;
    if (a == "sigmoid") return XG_ACT_SIGMOID;
    TORCH_CHECK_VALUE(false, "xg_sm100: unknown activation ", std::string(a));
}

// The device of the call's tensors is made current (a no-op when it already is), its current stream carries the launch.
struct On {
    c10::cuda::CUDAGuard guard;
    void* stream;
    explicit On(const Tensor& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
};

Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType dtype, const Tensor& like) {
    return at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt);
}

const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* mut(const Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
const void* ptr(const optional<Tensor>& t) { return t.has_value() ? ptr(*t) : nullptr; }

// The kernels read operands by address and know one set of extents: a tensor on another device, of another dtype or with fewer
// elements than the extents say would be read past its end. These checks are host compares of a few ns.
bool elsewhere(const Tensor& x, const Tensor& t) { return t.defined() && t.device() != x.device(); }
bool elsewhere(const Tensor& x, const optional<Tensor>& t) { return t.has_value() && elsewhere(x, *t); }
template <typename... T>
void one_device(const char* who, const Tensor& x, const T&... others) {
    TORCH_CHECK_VALUE(!(elsewhere(x, others) || ...), "xg_sm100::", who, ": all tensors must be on ", x.device());
}

// A tensor seen as [rows, cols] with contiguous rows; copied only when its strides do not allow that.
struct Rows {
    Tensor t;
    int64_t rows, cols, ld;
    explicit Rows(const Tensor& x) : t(x) {
        cols = x.size(-1);
        if (x.dim() == 2 && x.stride(1) == 1) {
            rows = x.size(0);
            ld = rows > 1 ? x.stride(0) : std::max(x.stride(0), cols);
            return;
        }
        t = x.contiguous();
        rows = cols ? t.numel() / cols : 0;
        ld = cols;
    }
};

Tensor unit_rows(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
int64_t row_stride(const Tensor& x) { return x.size(0) > 1 ? x.stride(0) : std::max(x.stride(0), x.size(1)); }
Tensor cast(const Tensor& t, at::ScalarType dtype) { return t.scalar_type() == dtype ? t : t.to(dtype); }

// Affine coefficients are passed as fp32 or as the activation dtype.
Tensor coef(const Tensor& w, at::ScalarType dtype) {
    return (w.scalar_type() == at::kFloat || w.scalar_type() == dtype ? w : w.to(at::kFloat)).contiguous();
}

// [B, H, S, D] output in the order of x's memory: a [B, S, H, D] buffer with dims 1 and 2 swapped when x's heads lie closer
// together than its positions, as in projections and packed QKV buffers (so that the transpose + reshape after attention
// stays a view); contiguous otherwise.
Tensor empty_like_layout(const Tensor& x) {
    const int64_t B = x.size(0), H = x.size(1), S = x.size(2), D = x.size(3);
    if (x.stride(3) == 1 && x.stride(1) < x.stride(2) && H > 1 && S > 1)
        return new_tensor({B, S, H, D}, x.scalar_type(), x).transpose(1, 2);
    return new_tensor({B, H, S, D}, x.scalar_type(), x);
}

// ---- normalisation -----------------------------------------------------------------------------------
template <bool RMS>
std::pair<Tensor, Tensor> norm(const Tensor& x, const Tensor& residual, const Tensor& weight, const Tensor& bias, double eps,
                               bool want_sum) {
    const On on(x);
    one_device(RMS ? "rms_norm" : "layer_norm", x, residual, weight, bias);
    const Rows x2(x);
    TORCH_CHECK_VALUE(weight.numel() == x2.cols && (!bias.defined() || bias.numel() == x2.cols),
                      "xg_sm100 norm: weight and bias must have one element per column of x");
    optional<Rows> r2;
    if (residual.defined()) {
        TORCH_CHECK_VALUE(residual.sizes() == x.sizes() && residual.scalar_type() == x.scalar_type(),
                          "xg_sm100 norm: residual must match x in shape and dtype");
        r2.emplace(residual);
    }
    const Tensor w = coef(weight, x.scalar_type());
    Tensor y = new_tensor(x.sizes(), x.scalar_type(), x);
    Tensor s = want_sum ? new_tensor(x.sizes(), x.scalar_type(), x) : Tensor();
    const void* rp = r2 ? ptr(r2->t) : nullptr;
    const int64_t rld = r2 ? r2->ld : 0;
    const int dt = code_of(x.scalar_type()), wdt = code_of(w.scalar_type());
    if (RMS) {
        XG_CALL(xg_rmsnorm, ptr(x2.t), rp, ptr(w), mut(y), mut(s), x2.rows, x2.cols, x2.ld, rld, eps, dt, wdt, on.stream);
    } else {
        const Tensor b = bias.defined() ? cast(coef(bias, x.scalar_type()), w.scalar_type()) : Tensor();
        XG_CALL(xg_layernorm, ptr(x2.t), rp, ptr(w), ptr(b), mut(y), mut(s), x2.rows, x2.cols, x2.ld, rld, eps, dt, wdt, on.stream);
    }
    return {std::move(y), std::move(s)};
}

Tensor or_none(const optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }

Tensor rms_norm(const Tensor& x, const Tensor& weight, double eps) { return norm<true>(x, {}, weight, {}, eps, false).first; }
std::vector<Tensor> add_rms_norm(const Tensor& x, const Tensor& residual, const Tensor& weight, double eps) {
    auto r = norm<true>(x, residual, weight, {}, eps, true);
    return {r.first, r.second};
}
Tensor add_rms_norm_y(const Tensor& x, const Tensor& residual, const Tensor& weight, double eps) {
    return norm<true>(x, residual, weight, {}, eps, false).first;
}
Tensor layer_norm(const Tensor& x, const Tensor& weight, const optional<Tensor>& bias, double eps) {
    return norm<false>(x, {}, weight, or_none(bias), eps, false).first;
}
std::vector<Tensor> add_layer_norm(const Tensor& x, const Tensor& residual, const Tensor& weight, const optional<Tensor>& bias, double eps) {
    auto r = norm<false>(x, residual, weight, or_none(bias), eps, true);
    return {r.first, r.second};
}
Tensor add_layer_norm_y(const Tensor& x, const Tensor& residual, const Tensor& weight, const optional<Tensor>& bias, double eps) {
    return norm<false>(x, residual, weight, or_none(bias), eps, false).first;
}

// ---- elementwise -------------------------------------------------------------------------------------
// A cos / sin table as contiguous [S, D]; any shape of that many elements.
Tensor table(const Tensor& t, int64_t S, int64_t D, at::ScalarType dtype) {
    if (t.dim() == 2 && t.size(0) == S && t.size(1) == D) return cast(t, dtype).contiguous();
    return cast(t.reshape({S, D}), dtype).contiguous();
}

Tensor rope(const Tensor& x_in, const Tensor& cos, const Tensor& sin) {
    TORCH_CHECK_VALUE(x_in.dim() == 4, "xg_sm100::rope expects [B, H, S, D]");
    const On on(x_in);
    one_device("rope", x_in, cos, sin);
    const Tensor x = x_in.stride(3) == 1 ? x_in : x_in.contiguous();
    const int64_t S = x.size(2), D = x.size(3);
    const Tensor c = table(cos, S, D, x.scalar_type()), s = table(sin, S, D, x.scalar_type());
    Tensor y = empty_like_layout(x);
    XG_CALL(xg_rope, ptr(x), ptr(c), ptr(s), mut(y), x.size(0), x.size(1), S, D, x.stride(0), x.stride(1), x.stride(2), y.stride(0),
            y.stride(1), y.stride(2), code_of(x.scalar_type()), on.stream);
    return y;
}

Tensor swiglu(const Tensor& gate, const Tensor& up) {
    TORCH_CHECK_VALUE(gate.sizes() == up.sizes() && gate.scalar_type() == up.scalar_type(), "xg_sm100::swiglu: gate and up must match");
    const On on(gate);
    one_device("swiglu", gate, up);
    const Rows g(gate), u(up);
    Tensor out = new_tensor(gate.sizes(), gate.scalar_type(), gate);
    XG_CALL(xg_swiglu, ptr(g.t), ptr(u.t), mut(out), g.rows, g.cols, g.ld, u.ld, g.cols, code_of(gate.scalar_type()), on.stream);
    return out;
}

// ---- dense layers --------------------------------------------------------------------------------------
struct Weight {
    Tensor t;
    bool trans;
};
// A 2-D weight with contiguous rows and the orientation flag that goes with it. A transposed view of a contiguous matrix
// (w.T, what F.linear(x, w.T) or x @ w.t() hand over) is read through its base in the other orientation - the kernels take
// both [N, K] and [K, N] - instead of being copied on every call.
Weight weight_rows(const Tensor& w, bool trans) {
    if (w.dim() == 2 && w.stride(1) != 1 && w.stride(0) == 1 && w.size(0) > 1) return {w.t(), !trans};
    return {unit_rows(w), trans};
}

bool f32_on_tensor_cores(int64_t M, int64_t N, int64_t K) { return xg_torch_f32_on_tensor_cores(M, N, K) != 0; }

bool same_ints(PyObject* tuple, at::IntArrayRef v) {
    if (!PyTuple_Check(tuple) || (size_t)PyTuple_GET_SIZE(tuple) != v.size()) return false;
    for (size_t i = 0; i < v.size(); ++i)
        if (PyLong_AsLongLong(PyTuple_GET_ITEM(tuple, i)) != v[i]) return false;
    return true;
}

// What a kept set of planes was made by: the context of its tensor's storage, so that it lives and goes with the planes (and a
// copy or an unpickled set, which lacks it, is never taken for one).
struct PlanesOrigin {
    Tensor memory;
    at::cuda::CUDAEvent written;  // recorded behind the split
    c10::cuda::CUDAStream stream;  // the one that split the weight
    static void release(void* p) { delete static_cast<PlanesOrigin*>(p); }
};

Tensor with_origin(const Tensor& planes, const c10::cuda::CUDAStream& stream) {
    auto origin = std::make_unique<PlanesOrigin>(PlanesOrigin{planes, {}, stream});
    origin->written.record(stream);
    void* data = planes.mutable_data_ptr();
    at::DataPtr hold(data, origin.release(), &PlanesOrigin::release, planes.device());
    Tensor t = at::detail::make_tensor<at::TensorImpl>(at::Storage(at::Storage::use_byte_size_t(), planes.nbytes(), std::move(hold), nullptr, false),
                                                       planes.key_set(), planes.dtype());
    t.unsafeGetTensorImpl()->set_sizes_contiguous(planes.sizes());
    return t;
}

bool capturing(void* stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(static_cast<cudaStream_t>(stream), &status) != cudaSuccess) {
        (void)cudaGetLastError();  // the default stream while a stream that blocks it is captured
        return true;
    }
    return status != cudaStreamCaptureStatusNone;
}

// The three bf16 planes of an fp32 weight, [N, 3*Kp]. They ride on the weight's Python object (attribute _xg_bf16_planes =
// (tag, planes)) and are rebuilt when the tag - version counter, address, layout, orientation - changes, so a dense layer's
// weight is split once in inference and the planes go away with the tensor; a fresh view of a weight is simply split again.
// A call on another stream than the one that split the weight waits for the split and is recorded with the allocator.
// In-place updates through weight.data do not move the counter: ops.invalidate_weight_planes drops the planes after those.
// While a CUDA graph is captured no kept planes are used and none are kept: the split becomes part of the graph, which so
// follows the weight (planes made in a capture hold nothing before the first replay, and a graph does not keep tensors alive).
// Tensors made under torch.inference_mode() have no version counter; their planes are not kept.
// `keep`: !capturing(stream), asked once per call.
Tensor weight_planes(const Tensor& w, bool trans, int64_t N, int64_t K, void* stream, bool keep) {
    const bool tracked = keep && !w.is_inference();
    if (tracked) {
        Tensor hit;
        {
            Gil gil;
            PyObject* obj = THPVariable_Wrap(w);
            PyObject* kept = obj ? PyObject_GetAttrString(obj, "_xg_bf16_planes") : nullptr;
            if (!kept) PyErr_Clear();
            if (kept && PyTuple_Check(kept) && PyTuple_GET_SIZE(kept) == 2 && PyTuple_Check(PyTuple_GET_ITEM(kept, 0)) &&
                PyTuple_GET_SIZE(PyTuple_GET_ITEM(kept, 0)) == 5 && THPVariable_Check(PyTuple_GET_ITEM(kept, 1))) {
                PyObject* tag = PyTuple_GET_ITEM(kept, 0);
                if (PyLong_AsLongLong(PyTuple_GET_ITEM(tag, 0)) == (int64_t)w._version() &&
                    PyLong_AsVoidPtr(PyTuple_GET_ITEM(tag, 1)) == w.const_data_ptr() && same_ints(PyTuple_GET_ITEM(tag, 2), w.sizes()) &&
                    same_ints(PyTuple_GET_ITEM(tag, 3), w.strides()) && (PyTuple_GET_ITEM(tag, 4) == Py_True) == trans)
                    hit = THPVariable_Unpack(PyTuple_GET_ITEM(kept, 1));
                PyErr_Clear();
            }
            Py_XDECREF(kept);
            Py_XDECREF(obj);
        }
        PlanesOrigin* origin = hit.defined() ? hit.storage().data_ptr().cast_context<PlanesOrigin>(&PlanesOrigin::release) : nullptr;
        if (origin) {
            if (origin->stream.stream() != stream) {
                const c10::cuda::CUDAStream current = c10::cuda::getCurrentCUDAStream(w.device().index());
                origin->written.block(current);
                c10::cuda::CUDACachingAllocator::recordStream(origin->memory.storage().data_ptr(), current);
            }
            return hit;
        }
    }
    Tensor w3 = new_tensor({N, 3 * xg_gemm_f32x3_padded_k(K)}, at::kBFloat16, w);
    XG_CALL(xg_split_bf16x3, ptr(w), N, K, row_stride(w), trans ? 0 : 1, mut(w3), stream);
    if (tracked) {
        w3 = with_origin(w3, c10::cuda::getCurrentCUDAStream(w.device().index()));
        Gil gil;
        PyObject* obj = THPVariable_Wrap(w);
        PyObject* mod = PyImport_ImportModule("xpu_graph_b200.ops");
        PyObject* tag = obj && mod ? PyObject_CallMethod(mod, "_planes_tag", "OO", obj, trans ? Py_True : Py_False) : nullptr;
        PyObject* planes = tag ? THPVariable_Wrap(w3) : nullptr;
        PyObject* pair = planes ? PyTuple_Pack(2, tag, planes) : nullptr;
        if (pair) PyObject_SetAttrString(obj, "_xg_bf16_planes", pair);  // a tensor type without instance attributes: no reuse
        PyErr_Clear();
        Py_XDECREF(pair);
        Py_XDECREF(planes);
        Py_XDECREF(tag);
        Py_XDECREF(mod);
        Py_XDECREF(obj);
    }
    return w3;
}

Tensor dense(const Tensor& x_in, const Tensor& weight, bool weight_trans, const optional<Tensor>& bias_in,
             const optional<Tensor>& residual_in, c10::string_view act) {
    TORCH_CHECK_VALUE(x_in.dim() == 2 && weight.dim() == 2, "xg_sm100::dense expects 2-D x and weight");
    const On on(x_in);
    const at::ScalarType dt = x_in.scalar_type();
    const Tensor x = unit_rows(x_in);
    const Weight w = weight_rows(weight, weight_trans);
    const int64_t M = x.size(0), K = x.size(1), N = w.trans ? w.t.size(0) : w.t.size(1);
    TORCH_CHECK_VALUE((w.trans ? w.t.size(1) : w.t.size(0)) == K, "xg_sm100::dense: inner dimensions differ");
    one_device("dense", x_in, weight, bias_in, residual_in);
    TORCH_CHECK_VALUE(weight.scalar_type() == dt, "xg_sm100::dense: x and the weight must share a dtype");
    TORCH_CHECK_VALUE(!bias_in || bias_in->numel() == N, "xg_sm100::dense: the bias must have one element per output column");
    TORCH_CHECK_VALUE(!residual_in || (residual_in->dim() == 2 && residual_in->size(0) == M && residual_in->size(1) == N),
                      "xg_sm100::dense: the residual must have the result's shape");
    const Tensor bias = bias_in ? cast(*bias_in, dt).contiguous() : Tensor();
    const Tensor residual = residual_in ? unit_rows(cast(*residual_in, dt)) : Tensor();
    const int64_t ldr = residual.defined() ? row_stride(residual) : 0;
    const int code = code_of(dt), a = act_code(act);
    Tensor out = new_tensor({M, N}, dt, x);
    if (dt == at::kFloat && f32_on_tensor_cores(M, N, K)) {
        const Tensor w3 = weight_planes(w.t, w.trans, N, K, on.stream, !capturing(on.stream));
        const Tensor a3 = new_tensor({M, 3 * xg_gemm_f32x3_padded_k(K)}, at::kBFloat16, x);
        XG_CALL(xg_split_bf16x3, ptr(x), M, K, row_stride(x), 0, mut(a3), on.stream);
        XG_CALL(xg_gemm_f32x3, ptr(a3), ptr(w3), ptr(bias), ptr(residual), mut(out), M, N, K, N, ldr, a, 0, on.stream);
        return out;
    }
    // scratch: split-K partial sums of weight-streaming shapes (small M), copies of operands no tensor map addresses
    int64_t ws_bytes = dt != at::kFloat && M <= 128 ? xg_gemm_workspace_bytes(M, N, K, code) : 0;
    ws_bytes += xg_gemm_copy_bytes(ptr(x), ptr(w.t), M, N, K, row_stride(x), row_stride(w.t), w.trans ? 1 : 0, code);
    const Tensor ws = ws_bytes > 0 ? new_tensor({ws_bytes}, at::kByte, x) : Tensor();
    XG_CALL(xg_gemm_bias_act_ws, ptr(x), ptr(w.t), ptr(bias), ptr(residual), mut(out), M, N, K, row_stride(x), row_stride(w.t), N, ldr,
            w.trans ? 1 : 0, a, code, mut(ws), ws_bytes, on.stream);
    return out;
}

Tensor batch_dense(const Tensor& x_in, const Tensor& weight_in, bool weight_trans, const optional<Tensor>& bias_in,
                   const optional<Tensor>& residual_in, c10::string_view act) {
    TORCH_CHECK_VALUE(x_in.dim() == 3 && weight_in.dim() == 3, "xg_sm100::batch_dense expects 3-D x and weight");
    const On on(x_in);
    one_device("batch_dense", x_in, weight_in, bias_in, residual_in);
    const at::ScalarType dt = x_in.scalar_type();
    const Tensor x = x_in.contiguous(), w = weight_in.contiguous();
    const int64_t b = x.size(0), M = x.size(1), K = x.size(2), N = weight_trans ? w.size(1) : w.size(2);
    TORCH_CHECK_VALUE(w.scalar_type() == dt && w.size(0) == b && w.size(weight_trans ? 2 : 1) == K,
                      "xg_sm100::batch_dense: x and the weight must share a dtype, the batch and the inner dimension");
    const Tensor bias = bias_in ? cast(*bias_in, dt).broadcast_to({b, 1, N}).contiguous() : Tensor();
    const Tensor residual = residual_in ? cast(*residual_in, dt).broadcast_to({b, M, N}).contiguous() : Tensor();
    Tensor out = new_tensor({b, M, N}, dt, x);
    XG_CALL(xg_bgemm_bias_act, ptr(x), ptr(w), ptr(bias), ptr(residual), mut(out), b, M, N, K, K, w.size(2), N, N, M * K,
            w.size(1) * w.size(2), bias.defined() ? N : 0, residual.defined() ? M * N : 0, M * N, weight_trans ? 1 : 0, act_code(act),
            code_of(dt), on.stream);
    return out;
}

Tensor dense_swiglu(const Tensor& x_in, const Tensor& w_gate, const Tensor& w_up) {
    TORCH_CHECK_VALUE(x_in.dim() == 2 && w_gate.dim() == 2 && w_gate.sizes() == w_up.sizes() && w_gate.size(1) == x_in.size(1),
                      "xg_sm100::dense_swiglu expects 2-D x [M, K] and two weights [N, K]");
    TORCH_CHECK_VALUE(w_gate.scalar_type() == x_in.scalar_type() && w_up.scalar_type() == x_in.scalar_type(),
                      "xg_sm100::dense_swiglu: x and the weights must share a dtype");
    const On on(x_in);
    one_device("dense_swiglu", x_in, w_gate, w_up);
    const Tensor x = unit_rows(x_in);
    Tensor g = unit_rows(w_gate), u = unit_rows(w_up);
    if (row_stride(g) != row_stride(u)) {
        g = g.contiguous();
        u = u.contiguous();
    }
    const int64_t M = x.size(0), K = x.size(1), N = g.size(0);
    Tensor out = new_tensor({M, N}, x.scalar_type(), x);
    XG_CALL(xg_gemm_swiglu, ptr(x), ptr(g), ptr(u), mut(out), M, N, K, row_stride(x), row_stride(g), N, code_of(x.scalar_type()), on.stream);
    return out;
}

Tensor dense_rope(const Tensor& x_in, const Tensor& weight, const Tensor& cos, const Tensor& sin, int64_t seq_len, int64_t head_dim) {
    TORCH_CHECK_VALUE(x_in.dim() == 2 && weight.dim() == 2 && weight.size(1) == x_in.size(1) && weight.scalar_type() == x_in.scalar_type(),
                      "xg_sm100::dense_rope expects 2-D x [M, K] and a weight [N, K] of one dtype");
    const On on(x_in);
    one_device("dense_rope", x_in, weight, cos, sin);
    const Tensor x = unit_rows(x_in), w = unit_rows(weight);
    const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
    const Tensor c = table(cos, seq_len, head_dim, x.scalar_type()), s = table(sin, seq_len, head_dim, x.scalar_type());
    Tensor out = new_tensor({M, N}, x.scalar_type(), x);
    XG_CALL(xg_gemm_rope, ptr(x), ptr(w), ptr(c), ptr(s), mut(out), M, N, K, row_stride(x), row_stride(w), N, seq_len, head_dim,
            code_of(x.scalar_type()), on.stream);
    return out;
}

// ---- chained dense layers --------------------------------------------------------------------------------
using Weights = Buf<Tensor>;

// Layer widths of a chain; weight l is [N, K] unless bit l of weights_kn says [K, N].
Buf<int64_t> chain_dims(const Tensor& x, const Weights& ws, int64_t weights_kn, const char* who) {
    Buf<int64_t> dims{x.size(1)};
    for (size_t l = 0; l < ws.size(); ++l) {
        const bool kn = (weights_kn >> l) & 1;
        TORCH_CHECK_VALUE(ws[l].size(kn ? 0 : 1) == dims.back(), "xg_sm100::", who, ": inner dimensions differ");
        TORCH_CHECK_VALUE(ws[l].scalar_type() == x.scalar_type(), "xg_sm100::", who, ": x and the weights must share a dtype");
        one_device(who, x, ws[l]);
        dims.push_back(ws[l].size(kn ? 1 : 0));
    }
    return dims;
}

Tensor chain_bias(const optional<Tensor>& b, const Tensor& x, int64_t n, const char* who) {
    if (!b) return {};
    TORCH_CHECK_VALUE(b->numel() == n, "xg_sm100::", who, ": a bias does not match its layer's width");
    one_device(who, x, b);
    return cast(*b, x.scalar_type()).contiguous();
}

Tensor mlp2(const Tensor& x_in, const Tensor& w1, const optional<Tensor>& b1, const Tensor& w2, const optional<Tensor>& b2,
            c10::string_view act1, c10::string_view act2, int64_t weights_kn) {
    TORCH_CHECK_VALUE(x_in.dim() == 2 && w1.dim() == 2 && w2.dim() == 2, "xg_sm100::mlp2 expects 2-D x, w1 and w2");
    const On on(x_in);
    const Tensor x = unit_rows(x_in);
    const Weights w{unit_rows(w1), unit_rows(w2)};
    const auto d = chain_dims(x, w, weights_kn, "mlp2");
    const Tensor c1 = chain_bias(b1, x, d[1], "mlp2"), c2 = chain_bias(b2, x, d[2], "mlp2");
    const int64_t M = x.size(0);
    Tensor out = new_tensor({M, d[2]}, x.scalar_type(), x);
    if (M == 0) return out;
    XG_CALL(xg_mlp2_bias_act, ptr(x), ptr(w[0]), ptr(c1), ptr(w[1]), ptr(c2), mut(out), M, d[0], d[1], d[2], row_stride(x),
            row_stride(w[0]), row_stride(w[1]), d[2], act_code(act1), act_code(act2), weights_kn, code_of(x.scalar_type()), on.stream);
    return out;
}

Tensor mlp3(const Tensor& x_in, const Tensor& w1, const optional<Tensor>& b1, const Tensor& w2, const optional<Tensor>& b2,
            const Tensor& w3, const optional<Tensor>& b3, c10::string_view act1, c10::string_view act2, c10::string_view act3,
            int64_t weights_kn) {
    TORCH_CHECK_VALUE(x_in.dim() == 2 && w1.dim() == 2 && w2.dim() == 2 && w3.dim() == 2, "xg_sm100::mlp3 expects 2-D x and weights");
    const On on(x_in);
    const Tensor x = unit_rows(x_in);
    const Weights w{unit_rows(w1), unit_rows(w2), unit_rows(w3)};
    const auto d = chain_dims(x, w, weights_kn, "mlp3");
    const Tensor c1 = chain_bias(b1, x, d[1], "mlp3"), c2 = chain_bias(b2, x, d[2], "mlp3"), c3 = chain_bias(b3, x, d[3], "mlp3");
    const int64_t M = x.size(0);
    Tensor out = new_tensor({M, d[3]}, x.scalar_type(), x);
    if (M == 0) return out;
    XG_CALL(xg_mlp3_bias_act, ptr(x), ptr(w[0]), ptr(c1), ptr(w[1]), ptr(c2), ptr(w[2]), ptr(c3), mut(out), M, d[0], d[1], d[2], d[3],
            row_stride(x), row_stride(w[0]), row_stride(w[1]), row_stride(w[2]), d[3], act_code(act1), act_code(act2), act_code(act3),
            weights_kn, code_of(x.scalar_type()), on.stream);
    return out;
}

Buf<c10::string_view> split_names(c10::string_view names) {
    Buf<c10::string_view> out;
    while (true) {
        const auto at = names.find(',');
        out.push_back(names.substr(0, at));
        if (at == c10::string_view::npos) return out;
        names = names.substr(at + 1);
    }
}

using OptList = Buf<optional<Tensor>>;

Tensor mlp_small_impl(const Tensor& x_in, const Weights& weights, const OptList& biases, const Buf<c10::string_view>& acts, int64_t weights_kn) {
    const size_t n = weights.size();
    const On on(x_in);
    const Tensor x = unit_rows(x_in);
    Weights w;
    for (const Tensor& t : weights) w.push_back(unit_rows(t));
    const auto dims = chain_dims(x, w, weights_kn, "mlp_small");
    Weights b;
    Buf<const void*> wp, bp;
    Buf<int64_t> ldw;
    Buf<int> codes;
    for (size_t l = 0; l < n; ++l) {
        b.push_back(biases[l] ? chain_bias(biases[l]->reshape({-1}), x, dims[l + 1], "mlp_small") : Tensor());
        wp.push_back(ptr(w[l]));
        bp.push_back(ptr(b[l]));
        ldw.push_back(row_stride(w[l]));
        codes.push_back(act_code(acts[l]));
    }
    const int64_t M = x.size(0);
    Tensor out = new_tensor({M, dims.back()}, x.scalar_type(), x);
    if (M == 0) return out;
    XG_CALL(xg_mlp_small_bias_act, ptr(x), wp.data(), bp.data(), mut(out), M, dims.data(), (int)n, row_stride(x), ldw.data(), dims.back(),
            codes.data(), weights_kn, code_of(x.scalar_type()), on.stream);
    return out;
}

Tensor mlp_small(const Tensor& x, at::TensorList weights, const c10::List<optional<Tensor>>& biases, c10::string_view act_names, int64_t weights_kn) {
    const auto acts = split_names(act_names);
    const size_t n = weights.size();
    bool ok = x.dim() == 2 && biases.size() == n && acts.size() == n;
    for (const Tensor& w : weights) ok = ok && w.dim() == 2;
    TORCH_CHECK_VALUE(ok, "xg_sm100::mlp_small expects a 2-D x and one 2-D weight, bias and activation per layer");
    OptList b;
    for (size_t l = 0; l < n; ++l) b.push_back(biases.get(l));
    return mlp_small_impl(x, Weights(weights.begin(), weights.end()), b, acts, weights_kn);
}

Tensor dense_tower(const Tensor& x_in, at::TensorList weights_in, const c10::List<bool>& trans_in, const c10::List<optional<Tensor>>& biases_in,
                   c10::string_view act_names) {
    const auto acts = split_names(act_names);
    const int n = (int)weights_in.size();
    TORCH_CHECK_VALUE(n > 0 && acts.size() == (size_t)n && trans_in.size() == (size_t)n && biases_in.size() == (size_t)n,
                      "xg_sm100::dense_tower: one weight, orientation, bias and activation per layer");
    const at::ScalarType dt = x_in.scalar_type();
    TORCH_CHECK_VALUE(x_in.dim() == 2 && (dt == at::kFloat || dt == at::kBFloat16 || dt == at::kHalf),
                      "xg_sm100::dense_tower expects a 2-D floating-point input");
    const int code = code_of(dt);
    const int64_t M = x_in.size(0);
    Weights w;
    Buf<bool> trans;
    OptList b;
    Buf<int64_t> dims{x_in.size(1)};
    bool tensor_cores = dt == at::kFloat;  // every layer qualifies for the fp32 tensor-core path
    for (int i = 0; i < n; ++i) {
        Weight r{weights_in[i], trans_in.get(i)};
        TORCH_CHECK_VALUE(r.t.dim() == 2 && r.t.size(r.trans ? 1 : 0) == dims.back(), "xg_sm100::dense_tower: inner dimensions differ");
        TORCH_CHECK_VALUE(r.t.scalar_type() == dt, "xg_sm100::dense_tower: x and the weights must share a dtype");
        dims.push_back(r.trans ? r.t.size(0) : r.t.size(1));
        const auto bias = biases_in.get(i);
        TORCH_CHECK_VALUE(!bias || bias->numel() == dims.back(), "xg_sm100::dense_tower: a bias does not match its layer's width");
        one_device("dense_tower", x_in, r.t, bias);
        if (dt != at::kFloat) r = weight_rows(r.t, r.trans);
        w.push_back(r.t);
        trans.push_back(r.trans);
        b.push_back(bias);
        tensor_cores = tensor_cores && f32_on_tensor_cores(M, dims[i + 1], dims[i]);
    }
    if (!tensor_cores) {
        // 16-bit towers: runs of three or two neighbouring layers that fit the chained-layer kernel run as one launch each;
        // narrow layers of any dtype run with their weights in shared memory; the rest goes layer by layer
        Tensor y = x_in;
        for (int i = 0; i < n;) {
            auto kn = [&](int layers) {
                int64_t bits = 0;
                for (int l = 0; l < layers; ++l) bits |= (int64_t)(trans[i + l] ? 0 : 1) << l;
                return bits;
            };
            auto fits = [&](int layer) { return trans[i + layer] || dims[i + layer + 1] % 8 == 0; };
            if (dt != at::kFloat && M > 0 && i + 2 < n && fits(0) && fits(1) && fits(2) &&
                xg_mlp3_supported(M, dims[i], dims[i + 1], dims[i + 2], dims[i + 3], code)) {
                y = mlp3(y, w[i], b[i], w[i + 1], b[i + 1], w[i + 2], b[i + 2], acts[i], acts[i + 1], acts[i + 2], kn(3));
                i += 3;
                continue;
            }
            if (dt != at::kFloat && M > 0 && i + 1 < n && fits(0) && fits(1) &&
                xg_mlp2_supported(M, dims[i], dims[i + 1], dims[i + 2], code)) {
                y = mlp2(y, w[i], b[i], w[i + 1], b[i + 1], acts[i], acts[i + 1], kn(2));
                i += 2;
                continue;
            }
            int run = 1;
            for (int r = 3; r >= 2 && run == 1; --r)
                if (i + r <= n && xg_torch_small_tower_worth_it(M, &dims[i], r, code)) run = r;
            if (run > 1)
                y = mlp_small_impl(y, Weights(w.begin() + i, w.begin() + i + run), OptList(b.begin() + i, b.begin() + i + run),
                                   Buf<c10::string_view>(acts.begin() + i, acts.begin() + i + run), kn(run));
            else
                y = dense(y, w[i], trans[i], b[i], std::nullopt, acts[i]);
            i += run;
        }
        return y;
    }
    // fp32 on the tensor cores: every inner layer's epilogue writes its result straight as the next layer's three bf16
    // planes, so no fp32 activation is stored or re-read between layers; the last layer stores fp32
    const On on(x_in);
    const Tensor x = unit_rows(x_in);
    Tensor a3 = new_tensor({M, 3 * xg_gemm_f32x3_padded_k(dims[0])}, at::kBFloat16, x);
    XG_CALL(xg_split_bf16x3, ptr(x), M, dims[0], row_stride(x), 0, mut(a3), on.stream);
    const bool keep = !capturing(on.stream);
    for (int i = 0; i < n; ++i) {
        const int64_t K = dims[i], N = dims[i + 1];
        const Tensor wi = unit_rows(w[i]);
        const Tensor w3 = weight_planes(wi, trans[i], N, K, on.stream, keep);
        const Tensor bias = b[i] ? cast(*b[i], at::kFloat).contiguous() : Tensor();
        const bool last = i == n - 1;
        Tensor out = last ? new_tensor({M, N}, at::kFloat, x) : new_tensor({M, 3 * xg_gemm_f32x3_padded_k(N)}, at::kBFloat16, x);
        XG_CALL(xg_gemm_f32x3, ptr(a3), ptr(w3), ptr(bias), nullptr, mut(out), M, N, K, N, 0, act_code(acts[i]), last ? 0 : 1, on.stream);
        a3 = out;
    }
    return a3;
}

// ---- attention -------------------------------------------------------------------------------------------
Tensor sdpa(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const optional<Tensor>& mask_in, double scale, bool is_causal) {
    TORCH_CHECK_VALUE(q_in.dim() == 4 && k_in.dim() == 4 && v_in.dim() == 4, "xg_sm100::sdpa expects 4-D q/k/v");
    TORCH_CHECK_VALUE(k_in.sizes() == v_in.sizes() && k_in.size(0) == q_in.size(0) && k_in.size(1) == q_in.size(1) && k_in.size(3) == q_in.size(3),
                      "xg_sm100::sdpa: k and v must be [B, H, Skv, D] with q's batch, heads and head dim");
    TORCH_CHECK_VALUE(k_in.scalar_type() == q_in.scalar_type() && v_in.scalar_type() == q_in.scalar_type(), "xg_sm100::sdpa: q, k and v must share a dtype");
    const On on(q_in);
    one_device("sdpa", q_in, k_in, v_in, mask_in);
    const Tensor q = unit_rows(q_in), k = unit_rows(k_in), v = unit_rows(v_in);
    const int64_t B = q.size(0), H = q.size(1), Sq = q.size(2), D = q.size(3), Skv = k.size(2);
    Tensor m;
    bool mask_bool = false;
    if (mask_in) {
        mask_bool = mask_in->scalar_type() == at::kBool;
        m = mask_bool ? *mask_in : cast(*mask_in, q.scalar_type());
        while (m.dim() < 4) m = m.unsqueeze(0);
        m = m.expand({B, H, Sq, Skv});
    }
    Tensor out = empty_like_layout(q);
    const int code = code_of(q.scalar_type());
    const int64_t ws_bytes = xg_sdpa_workspace_bytes(B, H, Sq, Skv, D, code);
    const int64_t* mstr = m.defined() ? m.strides().data() : nullptr;
    if (ws_bytes == 0 && !mask_bool) {
        XG_CALL(xg_sdpa_fwd, ptr(q), ptr(k), ptr(v), ptr(m), mut(out), B, H, Sq, Skv, D, q.strides().data(), k.strides().data(),
                v.strides().data(), out.strides().data(), mstr, scale, is_causal ? 1 : 0, code, on.stream);
        return out;
    }
    const Tensor ws = ws_bytes > 0 ? new_tensor({ws_bytes}, at::kByte, q) : Tensor();
    XG_CALL(xg_sdpa_fwd_ws, ptr(q), ptr(k), ptr(v), ptr(m), mut(out), B, H, Sq, Skv, D, q.strides().data(), k.strides().data(),
            v.strides().data(), out.strides().data(), mstr, scale, is_causal ? 1 : 0, code, mask_bool ? 1 : 0, mut(ws), ws_bytes, on.stream);
    return out;
}

// ---- copy fusions (bit-exact) ------------------------------------------------------------------------------
struct Segments {
    Buf<const void*> src;
    Buf<void*> dst;
    Buf<int64_t> src_ld, dst_ld, len;
    void add(const void* s, int64_t s_off, int64_t s_ld, void* d, int64_t d_off, int64_t d_ld, int64_t bytes) {
        src.push_back(static_cast<const char*>(s) + s_off);
        dst.push_back(static_cast<char*>(d) + d_off);
        src_ld.push_back(s_ld);
        dst_ld.push_back(d_ld);
        len.push_back(bytes);
    }
    void copy(int64_t rows, const Tensor& mask, bool zero_when, void* stream) const {
        XG_CALL(xg_seg_copy, src.data(), dst.data(), src_ld.data(), dst_ld.data(), len.data(), (int64_t)src.size(), rows,
                static_cast<const uint8_t*>(ptr(mask)), zero_when ? 1 : 0, stream);
    }
};

Tensor mask_bytes(const optional<Tensor>& mask, int64_t rows, const Tensor& like) {
    if (!mask) return {};
    one_device("row mask", like, mask);
    TORCH_CHECK_VALUE(mask->numel() == rows, "xg_sm100: row mask must have one entry per row");
    const Tensor m = mask->contiguous();
    // a bool holds 0 or 1 in one byte: read as it is
    return m.scalar_type() == at::kBool || m.scalar_type() == at::kByte ? m : m.to(at::kByte);
}

Buf<std::pair<int64_t, int64_t>> clamp_slices(int64_t width, at::IntArrayRef starts, at::IntArrayRef ends) {
    Buf<std::pair<int64_t, int64_t>> out;
    for (size_t i = 0; i < std::min(starts.size(), ends.size()); ++i) {
        int64_t s = starts[i] < 0 ? starts[i] + width : starts[i], e = ends[i] < 0 ? ends[i] + width : ends[i];
        s = std::min(std::max<int64_t>(s, 0), width);
        e = std::min(std::max(e, s), width);
        out.emplace_back(s, e);
    }
    return out;
}

Tensor rows_2d(const Tensor& src) {
    TORCH_CHECK_NOT_IMPLEMENTED(src.dim() == 2, "input must be 2d");
    return src.stride(1) == 1 ? src : src.contiguous();
}

// cat of slices of a 2-D source; `masked` (one flag per slice) limits the row mask to the flagged ones: the masked and the
// unmasked slices are then two passes of the segmented copy into one output buffer
Tensor slice_cat_impl(const Tensor& src_in, at::IntArrayRef starts, at::IntArrayRef ends, const c10::List<bool>* masked,
                      const optional<Tensor>& row_mask, bool zero_when) {
    const Tensor src = rows_2d(src_in);
    TORCH_CHECK_VALUE(!masked || masked->size() == starts.size(), "xg_sm100::slice_cat_partly_masked: one flag per slice");
    const On on(src);
    const int64_t rows = src.size(0), es = src.element_size(), ld = row_stride(src) * es;
    const auto segs = clamp_slices(src.size(1), starts, ends);
    int64_t total = 0, off = 0;
    for (const auto& s : segs) total += s.second - s.first;
    Tensor out = new_tensor({rows, total}, src.scalar_type(), src);
    Segments parts[2];
    for (size_t i = 0; i < segs.size(); ++i) {
        const int64_t len = segs[i].second - segs[i].first;
        parts[masked && !masked->get(i) ? 0 : 1].add(ptr(src), segs[i].first * es, ld, mut(out), off * es, total * es, len * es);
        off += len;
    }
    const Tensor mask = mask_bytes(row_mask, rows, src);
    if (!parts[0].src.empty()) parts[0].copy(rows, {}, zero_when, on.stream);
    if (!parts[1].src.empty()) parts[1].copy(rows, mask, zero_when, on.stream);
    return out;
}

Tensor slice_cat(const Tensor& src, at::IntArrayRef starts, at::IntArrayRef ends, const optional<Tensor>& row_mask, bool zero_when) {
    return slice_cat_impl(src, starts, ends, nullptr, row_mask, zero_when);
}
Tensor slice_cat_partly_masked(const Tensor& src, at::IntArrayRef starts, at::IntArrayRef ends, const c10::List<bool>& masked,
                               const Tensor& row_mask, bool zero_when) {
    return slice_cat_impl(src, starts, ends, &masked, row_mask, zero_when);
}

// Slice starts with negative values wrapped; every slice has to lie inside the row (a slice that aten.slice would have
// clamped arrives here with a length the row does not have: refused instead of read past the row).
Buf<int64_t> checked_starts(int64_t width, at::IntArrayRef starts, int64_t slice_len) {
    TORCH_CHECK_VALUE(slice_len >= 0, "xg_sm100::multi_slice: negative slice length ", slice_len);
    Buf<int64_t> out;
    for (int64_t s : starts) {
        s = s < 0 ? s + width : s;
        TORCH_CHECK_VALUE(s >= 0 && slice_len <= width && s <= width - slice_len, "xg_sm100::multi_slice: slice at ", s, " of length ",
                          slice_len, " is outside a row of ", width, " elements");
        out.push_back(s);
    }
    return out;
}

Tensor multi_slice_impl(const Tensor& src, at::IntArrayRef starts_in, int64_t slice_len, const c10::List<bool>* masked,
                        const optional<Tensor>& row_mask, bool zero_when) {
    const auto starts = checked_starts(src.size(-1), starts_in, slice_len);
    const On on(src);
    const Rows s(src);
    const int64_t es = src.element_size(), num = (int64_t)starts.size(), slab = s.rows * slice_len * es;
    Buf<int64_t> shape{num};
    for (int64_t d = 0; d + 1 < src.dim(); ++d) shape.push_back(src.size(d));
    shape.push_back(slice_len);
    Tensor out = new_tensor(shape, src.scalar_type(), src);
    Segments parts[2];
    for (int64_t k = 0; k < num; ++k)
        parts[masked && !masked->get(k) ? 0 : 1].add(ptr(s.t), starts[k] * es, s.ld * es, mut(out), k * slab, slice_len * es, slice_len * es);
    const Tensor mask = mask_bytes(row_mask, s.rows, src);
    if (!parts[0].src.empty()) parts[0].copy(s.rows, {}, zero_when, on.stream);
    if (!parts[1].src.empty()) parts[1].copy(s.rows, mask, zero_when, on.stream);
    return out;
}

Tensor multi_slice(const Tensor& src, at::IntArrayRef starts, int64_t slice_len) {
    return multi_slice_impl(src, starts, slice_len, nullptr, std::nullopt, false);
}
Tensor multi_slice_masked(const Tensor& src, at::IntArrayRef starts, int64_t slice_len, const c10::List<bool>& masked, const Tensor& row_mask,
                          bool zero_when) {
    TORCH_CHECK_NOT_IMPLEMENTED(src.dim() == 2, "input must be 2d");
    TORCH_CHECK_VALUE(masked.size() == starts.size(), "xg_sm100::multi_slice_masked: one flag per slice");
    return multi_slice_impl(src, starts, slice_len, &masked, row_mask, zero_when);
}

std::vector<Tensor> slice_cat_multi(const Tensor& src_in, at::IntArrayRef starts, at::IntArrayRef ends, at::IntArrayRef counts) {
    const Tensor src = rows_2d(src_in);
    const On on(src);
    const int64_t rows = src.size(0), es = src.element_size(), ld = row_stride(src) * es;
    const auto segs = clamp_slices(src.size(1), starts, ends);
    std::vector<Tensor> outs;
    Segments all;
    size_t pos = 0;
    for (int64_t c : counts) {
        const size_t end = std::min(pos + (size_t)c, segs.size());
        int64_t total = 0, off = 0;
        for (size_t i = pos; i < end; ++i) total += segs[i].second - segs[i].first;
        Tensor o = new_tensor({rows, total}, src.scalar_type(), src);
        for (size_t i = pos; i < end; ++i) {
            const int64_t len = segs[i].second - segs[i].first;
            all.add(ptr(src), segs[i].first * es, ld, mut(o), off * es, total * es, len * es);
            off += len;
        }
        outs.push_back(std::move(o));
        pos = end;
    }
    all.copy(rows, {}, false, on.stream);
    return outs;
}

Tensor cat_lastdim(at::TensorList xs, const optional<Tensor>& row_mask, bool zero_when) {
    TORCH_CHECK_VALUE(!xs.empty(), "xg_sm100::cat_lastdim: nothing to concatenate");
    const On on(xs[0]);
    std::vector<Rows> parts;
    parts.reserve(xs.size());
    int64_t total = 0, off = 0;
    for (const Tensor& x : xs) {
        parts.emplace_back(x);
        TORCH_CHECK_VALUE(x.scalar_type() == xs[0].scalar_type() && parts.back().rows == parts[0].rows,
                          "xg_sm100::cat_lastdim: inputs must agree in dtype and leading dims");
        one_device("cat_lastdim", xs[0], x);
        total += parts.back().cols;
    }
    Buf<int64_t> shape(xs[0].sizes().begin(), xs[0].sizes().end());
    shape.back() = total;
    Tensor out = new_tensor(shape, xs[0].scalar_type(), xs[0]);
    const int64_t es = out.element_size(), rows = parts[0].rows;
    Segments all;
    for (const Rows& p : parts) {
        all.add(ptr(p.t), 0, p.ld * es, mut(out), off * es, total * es, p.cols * es);
        off += p.cols;
    }
    all.copy(rows, mask_bytes(row_mask, rows, xs[0]), zero_when, on.stream);
    return out;
}

Tensor gather_stack(at::TensorList tables, const Tensor& idx, const optional<Tensor>& row_mask, bool zero_when) {
    const int64_t F = (int64_t)tables.size();
    TORCH_CHECK_VALUE(F > 0 && idx.dim() == 2 && idx.size(1) == F && idx.scalar_type() == at::kLong,
                      "xg_sm100::gather_stack: idx must be int64 [rows, F]");
    const On on(idx);
    const int64_t D = tables[0].dim() == 2 ? tables[0].size(1) : 0, rows = idx.size(0);
    std::vector<Tensor> copies;  // contiguous copies live until the launch is enqueued (frees are stream-ordered)
    Buf<const void*> ptrs;
    Buf<int64_t> table_rows;
    for (const Tensor& t : tables) {
        TORCH_CHECK_VALUE(t.dim() == 2 && t.size(1) == D && t.scalar_type() == tables[0].scalar_type(),
                          "xg_sm100::gather_stack: tables must be 2-D with one embedding dim and dtype");
        one_device("gather_stack", idx, t);
        if (t.is_contiguous()) {
            ptrs.push_back(ptr(t));
        } else {
            copies.push_back(t.contiguous());
            ptrs.push_back(ptr(copies.back()));
        }
        table_rows.push_back(t.size(0));
    }
    Tensor out = new_tensor({rows, F * D}, tables[0].scalar_type(), idx);
    const Tensor mask = mask_bytes(row_mask, rows, idx);
    XG_CALL(xg_gather_rows, ptrs.data(), table_rows.data(), F, static_cast<const int64_t*>(ptr(idx)), idx.stride(0), idx.stride(1),
            static_cast<const uint8_t*>(ptr(mask)), zero_when ? 1 : 0, mut(out), rows, D, F * D, (int)out.element_size(), on.stream);
    return out;
}

// ---- sums --------------------------------------------------------------------------------------------------
std::vector<Tensor> sum3d(at::TensorList inputs, int64_t dim) {
    std::vector<Tensor> xs, outs;
    Buf<const void*> in;
    Buf<void*> out;
    Buf<int64_t> shapes;
    if (inputs.empty()) return outs;
    const On on(inputs[0]);
    for (const Tensor& x_in : inputs) {
        TORCH_CHECK_VALUE(x_in.dim() == 3, "xg_sm100::sum3d expects 3-D tensors");
        TORCH_CHECK_VALUE(x_in.scalar_type() == inputs[0].scalar_type(), "xg_sm100::sum3d: inputs must share a dtype");
        one_device("sum3d", inputs[0], x_in);
        xs.push_back(x_in.contiguous());
        const int64_t s0 = x_in.size(0), s1 = x_in.size(1), s2 = x_in.size(2);
        shapes.append({s0, s1, s2});
        outs.push_back(new_tensor({dim == 0 ? s1 : s0, dim == 2 ? s1 : s2}, x_in.scalar_type(), x_in));
        in.push_back(ptr(xs.back()));
        out.push_back(mut(outs.back()));
    }
    XG_CALL(xg_sum3d, in.data(), out.data(), shapes.data(), (int64_t)xs.size(), (int)dim, code_of(xs[0].scalar_type()), on.stream);
    return outs;
}

// Row sums written side by side: range k of [B, R_k, C] operand k (times a second operand) summed over its rows.
struct RowSums {
    std::vector<Tensor> keep;
    Buf<const void*> a, b;
    Buf<int64_t> a_bs, b_bs, ranges;
    int64_t batch, C;
    at::ScalarType dtype;
    RowSums(int64_t batch, const Tensor& first) : batch(batch), C(first.size(-1)), dtype(first.scalar_type()) {}

    void add(const Tensor& x_in, const Tensor& y_in, int64_t r0, int64_t r1) {
        const Tensor x = x_in.contiguous();
        TORCH_CHECK_VALUE(x.dim() == 3 && x.size(2) == C && x.scalar_type() == dtype && (x.size(0) == 1 || x.size(0) == batch),
                          "xg_sm100::rowsum_cat: operands must be [batch or 1, rows, C] tensors of one dtype");
        if (!keep.empty()) one_device("rowsum_cat", keep[0], x, y_in);
        else one_device("rowsum_cat", x, y_in);
        a.push_back(ptr(x));
        a_bs.push_back(x.size(0) == 1 && batch != 1 ? 0 : x.size(1) * C);
        keep.push_back(x);
        if (y_in.defined()) {
            const Tensor y = y_in.contiguous();
            TORCH_CHECK_VALUE(y.dim() == 3 && y.size(1) == x.size(1) && y.size(2) == C && y.scalar_type() == dtype &&
                                  (y.size(0) == 1 || y.size(0) == batch),
                              "xg_sm100::rowsum_cat: second operands must match the first in rows, C and dtype");
            b.push_back(ptr(y));
            b_bs.push_back(y.size(0) == 1 && batch != 1 ? 0 : y.size(1) * C);
            keep.push_back(y);
        }
        TORCH_CHECK_VALUE(0 <= r0 && r0 <= r1 && r1 <= x.size(1), "xg_sm100::rowsum_cat: row range outside the operand");
        ranges.append({r0, r1});
    }

    Tensor run() const {
        const On on(keep[0]);
        const int64_t n = (int64_t)a.size();
        Tensor out = new_tensor({batch, n * C}, dtype, keep[0]);
        XG_CALL(xg_rowsum_cat, a.data(), b.empty() ? nullptr : b.data(), a_bs.data(), b.empty() ? nullptr : b_bs.data(), ranges.data(), n,
                batch, C, mut(out), n * C, code_of(dtype), on.stream);
        return out;
    }
};

Tensor slice_sum_cat(const Tensor& src, at::IntArrayRef starts, at::IntArrayRef ends) {
    TORCH_CHECK_VALUE(src.dim() == 3, "xg_sm100::slice_sum_cat expects a 3-D tensor");
    TORCH_CHECK_VALUE(!starts.empty() && starts.size() <= ends.size(), "xg_sm100::slice_sum_cat: one end per start, and at least one of them");
    RowSums sums(src.size(0), src);
    const Tensor x = src.contiguous();
    for (const auto& r : clamp_slices(src.size(1), starts, ends)) sums.add(x, {}, r.first, r.second);
    return sums.run();
}

Tensor sum_cat(at::TensorList inputs) {
    TORCH_CHECK_VALUE(!inputs.empty(), "xg_sm100::sum_cat: no inputs");
    RowSums sums(inputs[0].size(0), inputs[0]);
    for (const Tensor& x : inputs) sums.add(x, {}, 0, x.size(1));
    return sums.run();
}

Tensor mul_sum_cat(at::TensorList lhs, at::TensorList rhs) {
    TORCH_CHECK_VALUE(!lhs.empty() && lhs.size() <= rhs.size(), "xg_sm100::mul_sum_cat: one second operand per first, and at least one of them");
    const size_t n = lhs.size();
    int64_t batch = 0;
    for (size_t i = 0; i < n; ++i) batch = std::max({batch, lhs[i].size(0), rhs[i].size(0)});
    RowSums sums(batch, lhs[0]);
    for (size_t i = 0; i < n; ++i) sums.add(lhs[i], rhs[i], 0, lhs[i].size(1));
    return sums.run();
}

// ---- whole graphs --------------------------------------------------------------------------------------------
// The fused op sequences of fused_graphs.py as one operator each. With a Python frame, a module call, an operator dispatch
// and several tensor views per kernel the host needed 90-105 us for the seven to nine launches of a small graph, more than
// the kernels; from here a launch costs 4 us. The operators are for inference only: nothing below is seen by autograd.
// Part `part` of `parts` side by side (packed q, k, v) of the rows of a projection as [B, H, S, D].
Tensor heads_view(const Tensor& rows, int64_t B, int64_t S, int64_t H, int64_t D, int part = 0, int parts = 1) {
    TORCH_CHECK(rows.size(0) == B * S && rows.size(1) == parts * H * D, "xg_sm100: a projection of ", rows.size(1), " columns is not ", parts, " x ", H,
                " heads of ", D);
    const int64_t ld = rows.stride(0);
    return rows.as_strided({B, H, S, D}, {S * ld, D, ld, 1}, rows.storage_offset() + part * H * D);
}
int64_t head_dim(int64_t hidden, int64_t heads, const char* who) {
    TORCH_CHECK_VALUE(heads > 0 && hidden % heads == 0, "xg_sm100::", who, ": ", hidden, " columns are not ", heads, " heads");
    return hidden / heads;
}
Tensor heads_to_rows(const Tensor& a, int64_t rows, int64_t cols) { return a.transpose(1, 2).reshape({rows, cols}); }

// LayerNorm | dense | attention | dense + residual | LayerNorm | dense + GELU | dense + residual.
// params: (weight, bias) of ln1, qkv, proj, ln2, fc1, fc2
Tensor encoder_block(const Tensor& x, const c10::List<optional<Tensor>>& params, double eps1, double eps2, int64_t heads) {
    at::AutoDispatchBelowADInplaceOrView no_grad;
    TORCH_CHECK_VALUE(x.dim() == 3 && params.size() == 12, "xg_sm100::encoder_block: x is [B, S, hidden], params are six (weight, bias) pairs");
    auto weight = [&](int i) -> Tensor { return params.get(2 * i).value(); };
    auto bias = [&](int i) -> optional<Tensor> { return params.get(2 * i + 1); };
    const int64_t B = x.size(0), S = x.size(1), C = x.size(2), D = head_dim(C, heads, "encoder_block"), T = B * S;
    const Tensor x0 = x.reshape({T, C});
    const Tensor qkv = dense(norm<false>(x0, {}, weight(0), or_none(bias(0)), eps1, false).first, weight(1), true, bias(1), std::nullopt, "none");
    const Tensor a = sdpa(heads_view(qkv, B, S, heads, D, 0, 3), heads_view(qkv, B, S, heads, D, 1, 3), heads_view(qkv, B, S, heads, D, 2, 3),
                          std::nullopt, 1.0 / std::sqrt((double)D), false);
    const Tensor x1 = dense(heads_to_rows(a, T, C), weight(2), true, bias(2), x0, "none");
    const Tensor h = dense(norm<false>(x1, {}, weight(3), or_none(bias(3)), eps2, false).first, weight(4), true, bias(4), std::nullopt, "gelu");
    return dense(h, weight(5), true, bias(5), x1, "none").view({B, S, C});
}

// Whether dense() adds up an output's products in one chain over K, as the grouped kernel does. Where it splits K (split-K through
// scratch, clusters of several CTA pairs) the partial sums round differently.
bool dense_sums_in_one_chain(int64_t M, int64_t N, int64_t K, int code) {
    int splits = 0, tile_n = 0;
    return xg_gemm_workspace_bytes(M, N, K, code) == 0 && !(xg_gemm_cluster_plan(M, N, K, code, &splits, &tile_n) && splits > 1);
}

// The q and k projections of one hidden state in one launch where that is the faster way (false: not taken), and v with them
// where the result is bit for bit that of a launch of its own: a graph rewritten op by op gives the same numbers.
bool qkv_rope(const Tensor& x_in, const Tensor& wq, const Tensor& wk, const Tensor& wv, const Tensor& cos, const Tensor& sin, int64_t S, int64_t D,
              Tensor* q, Tensor* k, Tensor* v) {
    const at::ScalarType dt = x_in.scalar_type();
    if ((dt != at::kHalf && dt != at::kBFloat16) || (D != 64 && D != 128) || wq.dim() != 2 || x_in.size(0) == 0) return false;
    const int code = code_of(dt);
    const int64_t M = x_in.size(0), K = x_in.size(1), N = wq.size(0), ldw = row_stride(wq);
    if (wq.size(1) != K || K == 0 || N == 0 || K % 8 != 0 || ldw % 8 != 0 || N % D != 0 || N % 8 != 0) return false;
    const int count = dense_sums_in_one_chain(M, N, K, code) ? 3 : 2;
    const Tensor* ws[3] = {&wq, &wk, &wv};
    for (int i = 0; i < count; ++i) {
        const Tensor& w = *ws[i];
        if (w.dim() != 2 || w.scalar_type() != dt || w.sizes() != wq.sizes() || w.strides() != wq.strides() || w.stride(1) != 1 ||
            (reinterpret_cast<uintptr_t>(ptr(w)) & 15u) != 0)
            return false;
    }
    if (!xg_gemm_rope_group_worth_it(count, M, N, K)) return false;
    const On on(x_in);
    one_device("decoder_layer", x_in, wq, wk, wv, cos, sin);
    const Tensor x = unit_rows(x_in);
    if ((reinterpret_cast<uintptr_t>(ptr(x)) & 15u) != 0 || row_stride(x) % 8 != 0) return false;
    const Tensor c = table(cos, S, D, dt), s = table(sin, S, D, dt);
    if (((reinterpret_cast<uintptr_t>(ptr(c)) | reinterpret_cast<uintptr_t>(ptr(s))) & 15u) != 0) return false;
    Tensor* outs[3] = {q, k, v};
    const void* wp[3];
    void* op[3];
    for (int i = 0; i < count; ++i) {
        *outs[i] = new_tensor({M, N}, dt, x);
        wp[i] = ptr(*ws[i]);
        op[i] = mut(*outs[i]);
    }
    XG_CALL(xg_gemm_rope_group, ptr(x), wp, ptr(c), ptr(s), op, count, 2, M, N, K, row_stride(x), ldw, N, S, D, code, on.stream);
    return true;
}

// RMSNorm | q, k with RoPE, v | causal attention | dense + residual | RMSNorm | SwiGLU | dense + residual.
// weights: input norm, q, k, v, o, post norm, gate, up, down
Tensor decoder_layer(const Tensor& x, const Tensor& cos, const Tensor& sin, at::TensorList w, double eps1, double eps2, int64_t heads,
                     bool fuse_rope, bool fuse_swiglu) {
    at::AutoDispatchBelowADInplaceOrView no_grad;
    TORCH_CHECK_VALUE(x.dim() == 3 && w.size() == 9, "xg_sm100::decoder_layer: x is [B, S, hidden], nine weights");
    const int64_t B = x.size(0), S = x.size(1), C = x.size(2), D = head_dim(C, heads, "decoder_layer"), T = B * S;
    const Tensor x0 = x.reshape({T, C});
    auto linear = [&](const Tensor& in, const Tensor& weight, const optional<Tensor>& residual) {
        return dense(in, weight, true, std::nullopt, residual, "none");
    };
    const Tensor h = norm<true>(x0, {}, w[0], {}, eps1, false).first;
    Tensor q, k, v;
    if (fuse_rope && qkv_rope(h, w[1], w[2], w[3], cos, sin, S, D, &q, &k, &v)) {
        q = heads_view(q, B, S, heads, D);
        k = heads_view(k, B, S, heads, D);
        if (v.defined()) v = heads_view(v, B, S, heads, D);
    } else if (fuse_rope) {
        q = heads_view(dense_rope(h, w[1], cos, sin, S, D), B, S, heads, D);
        k = heads_view(dense_rope(h, w[2], cos, sin, S, D), B, S, heads, D);
    } else {
        q = rope(heads_view(linear(h, w[1], std::nullopt), B, S, heads, D), cos, sin);
        k = rope(heads_view(linear(h, w[2], std::nullopt), B, S, heads, D), cos, sin);
    }
    if (!v.defined()) v = heads_view(linear(h, w[3], std::nullopt), B, S, heads, D);
    const Tensor a = sdpa(q, k, v, std::nullopt, 1.0 / std::sqrt((double)D), true);
    const Tensor x1 = linear(heads_to_rows(a, T, C), w[4], x0);
    const Tensor h2 = norm<true>(x1, {}, w[5], {}, eps2, false).first;
    const Tensor g = fuse_swiglu ? dense_swiglu(h2, w[6], w[7]) : swiglu(linear(h2, w[6], std::nullopt), linear(h2, w[7], std::nullopt));
    return linear(g, w[8], x1).view({B, S, C});
}

// The fp32 input of a recommender's first layer - slices of the features, then the masked lookups - as that layer's three bf16
// planes, in one kernel. Undefined where the inputs are not what the kernel takes (whole 16-byte units throughout); they then
// go through slice_cat, gather_stack and cat_lastdim, which also report what is wrong with them.
Tensor recommender_planes(const Tensor& features, const Tensor& idx, const Tensor& mask, at::TensorList tables, at::IntArrayRef starts,
                          at::IntArrayRef ends, int64_t* K) {
    const int64_t F = (int64_t)tables.size();
    if (features.dim() != 2 || features.scalar_type() != at::kFloat || (features.size(1) > 1 && features.stride(1) != 1) || F < 1 || F > 64 || starts.size() > 64 ||
        starts.size() != ends.size() || idx.dim() != 2 || idx.size(1) != F || idx.scalar_type() != at::kLong)
        return {};
    const int64_t rows = features.size(0), ld = row_stride(features), D = tables[0].dim() == 2 ? tables[0].size(1) : 0;
    auto aligned = [](const Tensor& t) { return (reinterpret_cast<uintptr_t>(ptr(t)) & 15u) == 0; };
    one_device("recommender", features, idx, mask);
    if (features.numel() == 0 || idx.size(0) != rows || mask.numel() != rows || D == 0 || D % 4 != 0 || D > 1 << 20 || ld % 4 != 0 || !aligned(features)) return {};
    Buf<const void*> ptrs;
    Buf<int64_t> table_rows, first, len;
    for (const Tensor& t : tables) {
        one_device("recommender", features, t);
        if (t.dim() != 2 || t.size(1) != D || t.scalar_type() != at::kFloat || !t.is_contiguous() || !aligned(t) || t.size(0) > 0x7fffffff ||
            t.numel() == 0)
            return {};
        ptrs.push_back(ptr(t));
        table_rows.push_back(t.size(0));
    }
    int64_t cols = 0;
    for (const auto& s : clamp_slices(features.size(1), starts, ends)) {
        if (s.first % 4 != 0 || s.second % 4 != 0) return {};
        first.push_back(s.first);
        len.push_back(s.second - s.first);
        cols += s.second - s.first;
    }
    if (cols > 4096 || (rows > 1 && ld < features.size(1))) return {};
    *K = cols + F * D;
    const On on(features);
    const Tensor hide = mask_bytes(mask, rows, features);
    Tensor out = new_tensor({rows, 3 * xg_gemm_f32x3_padded_k(*K)}, at::kBFloat16, features);
    XG_CALL(xg_gather_planes, ptr(features), ld, first.data(), len.data(), (int64_t)first.size(), ptrs.data(), table_rows.data(), F,
            static_cast<const int64_t*>(ptr(idx)), idx.stride(0), idx.stride(1), static_cast<const uint8_t*>(ptr(hide)), 1, mut(out), rows, D,
            on.stream);
    return out;
}

// Slices of the dense features and the masked lookups side by side in one buffer, then the dense layers (ReLU). Neighbouring
// layers on the tensor cores hand their result over as bf16 planes.
Tensor recommender(const Tensor& features, const Tensor& idx, const Tensor& mask, at::TensorList tables, at::IntArrayRef starts,
                   at::IntArrayRef ends, at::TensorList weights, const c10::List<optional<Tensor>>& biases) {
    at::AutoDispatchBelowADInplaceOrView no_grad;
    TORCH_CHECK_VALUE(!weights.empty() && biases.size() == weights.size(), "xg_sm100::recommender: one bias entry per weight");
    const int64_t M = features.dim() == 2 ? features.size(0) : 0;
    auto on_tensor_cores = [&](size_t i, int64_t k) {
        return i < weights.size() && weights[i].dim() == 2 && weights[i].scalar_type() == at::kFloat && weights[i].size(1) == k &&
               f32_on_tensor_cores(M, weights[i].size(0), k);
    };
    size_t i = 0;
    Tensor h;
    int64_t k = 0;
    // (the first weight's own width stands for the assembled row's: it has to be that)
    if (on_tensor_cores(0, weights[0].dim() == 2 ? weights[0].size(1) : 0))
        h = recommender_planes(features, idx, mask, tables, starts, ends, &k);
    if (h.defined()) {
        TORCH_CHECK_VALUE(weights[0].size(1) == k, "xg_sm100::dense: inner dimensions differ");
        const On on(features);
        const bool keep = !capturing(on.stream);
        for (bool planes = true; planes; ++i) {
            const int64_t N = weights[i].size(0);
            const Tensor w = unit_rows(weights[i]);
            one_device("recommender", features, w);
            const Tensor w3 = weight_planes(w, true, N, k, on.stream, keep);
            const Tensor bias = chain_bias(biases.get(i), features, N, "recommender");
            planes = on_tensor_cores(i + 1, N);
            Tensor out = planes ? new_tensor({M, 3 * xg_gemm_f32x3_padded_k(N)}, at::kBFloat16, h) : new_tensor({M, N}, at::kFloat, h);
            XG_CALL(xg_gemm_f32x3, ptr(h), ptr(w3), ptr(bias), nullptr, mut(out), M, N, k, N, 0, act_code("relu"), planes ? 1 : 0, on.stream);
            h = out;
            k = N;
        }
    } else {
        h = cat_lastdim({slice_cat(features, starts, ends, std::nullopt, false), gather_stack(tables, idx, mask, true)}, std::nullopt, false);
    }
    for (; i < weights.size(); ++i) h = dense(h, weights[i], true, biases.get(i), std::nullopt, "relu");
    return h;
}

// The autograd kernels of the graph operators: inference only, like the other operators, so that a backward through one of them
// is an error instead of a gradient that is missing without a word. By hand, since the general fallback boxes its arguments:
// some forty tensors, a tenth of what a small graph costs.
void collect(at::TensorList& all, std::vector<Tensor>& out) { out.insert(out.end(), all.begin(), all.end()); }
void collect(const Tensor& t, std::vector<Tensor>& out) { out.push_back(t); }
void collect(const c10::List<optional<Tensor>>& all, std::vector<Tensor>& out) {
    for (size_t i = 0; i < all.size(); ++i) out.push_back(or_none(all.get(i)));
}
template <typename T>
void collect(const T&, std::vector<Tensor>&) {}

template <auto Op>
struct GraphAutograd;
template <typename... A, Tensor (*Op)(A...)>
struct GraphAutograd<Op> {
    static inline const char* name = nullptr;
    static Tensor call(c10::DispatchKeySet keys, A... args) {
        static auto op = c10::Dispatcher::singleton().findSchemaOrThrow(name, "").template typed<Tensor(A...)>();
        Tensor out = [&] {
            at::AutoDispatchBelowAutograd below;
            return op.redispatch(keys & c10::after_autograd_keyset, args...);
        }();
        const bool forward_mode = torch::autograd::ForwardADLevel::try_get_by_idx(0) != nullptr;
        if (at::GradMode::is_enabled() || forward_mode) {
            std::vector<Tensor> inputs;
            (collect(args, inputs), ...);
            for (const Tensor& t : inputs)
                TORCH_CHECK_NOT_IMPLEMENTED(!forward_mode || !t.defined() || !t._fw_grad(0).defined(), name, " has no forward-mode derivative");
            if (torch::autograd::compute_requires_grad(inputs))
                torch::autograd::set_history(out, std::make_shared<torch::autograd::NotImplemented>(name, torch::autograd::collect_next_edges(inputs)));
        }
        return out;
    }
};

// ---- registration --------------------------------------------------------------------------------------------
const char* const kSchemas[] = {
    "rms_norm(Tensor x, Tensor weight, float eps) -> Tensor",
    "add_rms_norm(Tensor x, Tensor residual, Tensor weight, float eps) -> Tensor[]",
    "add_rms_norm_y(Tensor x, Tensor residual, Tensor weight, float eps) -> Tensor",
    "layer_norm(Tensor x, Tensor weight, Tensor? bias, float eps) -> Tensor",
    "add_layer_norm(Tensor x, Tensor residual, Tensor weight, Tensor? bias, float eps) -> Tensor[]",
    "add_layer_norm_y(Tensor x, Tensor residual, Tensor weight, Tensor? bias, float eps) -> Tensor",
    "rope(Tensor x, Tensor cos, Tensor sin) -> Tensor",
    "swiglu(Tensor gate, Tensor up) -> Tensor",
    "dense(Tensor x, Tensor weight, bool weight_trans, Tensor? bias, Tensor? residual, str act) -> Tensor",
    "batch_dense(Tensor x, Tensor weight, bool weight_trans, Tensor? bias, Tensor? residual, str act) -> Tensor",
    "dense_swiglu(Tensor x, Tensor w_gate, Tensor w_up) -> Tensor",
    "dense_rope(Tensor x, Tensor weight, Tensor cos, Tensor sin, SymInt seq_len, SymInt head_dim) -> Tensor",
    "mlp2(Tensor x, Tensor w1, Tensor? b1, Tensor w2, Tensor? b2, str act1, str act2, SymInt weights_kn=0) -> Tensor",
    "mlp3(Tensor x, Tensor w1, Tensor? b1, Tensor w2, Tensor? b2, Tensor w3, Tensor? b3, str act1, str act2, str act3, "
    "SymInt weights_kn=0) -> Tensor",
    "mlp_small(Tensor x, Tensor[] weights, Tensor?[] biases, str act_names, SymInt weights_kn) -> Tensor",
    "dense_tower(Tensor x, Tensor[] weights, bool[] weight_trans, Tensor?[] biases, str act_names) -> Tensor",
    "sdpa(Tensor q, Tensor k, Tensor v, Tensor? attn_mask, float scale, bool is_causal) -> Tensor",
    "slice_cat(Tensor src, SymInt[] starts, SymInt[] ends, Tensor? row_mask, bool zero_when) -> Tensor",
    "slice_cat_partly_masked(Tensor src, SymInt[] starts, SymInt[] ends, bool[] masked, Tensor row_mask, bool zero_when) -> Tensor",
    "multi_slice(Tensor src, SymInt[] starts, SymInt slice_len) -> Tensor",
    "multi_slice_masked(Tensor src, SymInt[] starts, SymInt slice_len, bool[] masked, Tensor row_mask, bool zero_when) -> Tensor",
    "slice_cat_multi(Tensor src, SymInt[] starts, SymInt[] ends, SymInt[] counts) -> Tensor[]",
    "cat_lastdim(Tensor[] xs, Tensor? row_mask, bool zero_when) -> Tensor",
    "gather_stack(Tensor[] tables, Tensor idx, Tensor? row_mask, bool zero_when) -> Tensor",
    "sum3d(Tensor[] inputs, SymInt dim) -> Tensor[]",
    "slice_sum_cat(Tensor src, SymInt[] starts, SymInt[] ends) -> Tensor",
    "sum_cat(Tensor[] inputs) -> Tensor",
    "mul_sum_cat(Tensor[] lhs, Tensor[] rhs) -> Tensor",
};

const char* const kGraphSchemas[] = {
    "encoder_block(Tensor x, Tensor?[] params, float eps1, float eps2, SymInt heads) -> Tensor",
    "decoder_layer(Tensor x, Tensor cos, Tensor sin, Tensor[] weights, float eps1, float eps2, SymInt heads, bool fuse_rope, "
    "bool fuse_swiglu) -> Tensor",
    "recommender(Tensor features, Tensor idx, Tensor mask, Tensor[] tables, SymInt[] starts, SymInt[] ends, Tensor[] weights, "
    "Tensor?[] biases) -> Tensor",
};

}  // namespace

TORCH_LIBRARY(xg_sm100, m) {
    for (const char* s : kSchemas) m.def(s, {at::Tag::pt2_compliant_tag});
    for (const char* s : kGraphSchemas) m.def(s, {at::Tag::pt2_compliant_tag});
}

TORCH_LIBRARY_IMPL(xg_sm100, CUDA, m) {
#define XG_IMPL(op) m.impl(#op, &op)
    XG_IMPL(rms_norm);
    XG_IMPL(add_rms_norm);
    XG_IMPL(add_rms_norm_y);
    XG_IMPL(layer_norm);
    XG_IMPL(add_layer_norm);
    XG_IMPL(add_layer_norm_y);
    XG_IMPL(rope);
    XG_IMPL(swiglu);
    XG_IMPL(dense);
    XG_IMPL(batch_dense);
    XG_IMPL(dense_swiglu);
    XG_IMPL(dense_rope);
    XG_IMPL(mlp2);
    XG_IMPL(mlp3);
    XG_IMPL(mlp_small);
    XG_IMPL(dense_tower);
    XG_IMPL(sdpa);
    XG_IMPL(slice_cat);
    XG_IMPL(slice_cat_partly_masked);
    XG_IMPL(multi_slice);
    XG_IMPL(multi_slice_masked);
    XG_IMPL(slice_cat_multi);
    XG_IMPL(cat_lastdim);
    XG_IMPL(gather_stack);
    XG_IMPL(sum3d);
    XG_IMPL(slice_sum_cat);
    XG_IMPL(sum_cat);
    XG_IMPL(mul_sum_cat);
    XG_IMPL(encoder_block);
    XG_IMPL(decoder_layer);
    XG_IMPL(recommender);
#undef XG_IMPL
}

// Inference operators: a backward through one of them is an error.
TORCH_LIBRARY_IMPL(xg_sm100, Autograd, m) {
    for (const char* s : kSchemas) {
        const std::string schema(s);
        m.impl(schema.substr(0, schema.find('(')).c_str(), torch::autograd::autogradNotImplementedFallback());
    }
#define XG_GRAPH_IMPL(op) GraphAutograd<&op>::name = "xg_sm100::" #op, m.impl(#op, TORCH_FN(GraphAutograd<&op>::call))
    XG_GRAPH_IMPL(encoder_block);
    XG_GRAPH_IMPL(decoder_layer);
    XG_GRAPH_IMPL(recommender);
#undef XG_GRAPH_IMPL
}

// lib.call_hook: Python callables (or None) that see every C-ABI call made from this file. Called with the GIL held.
extern "C" void xg_torch_set_hook(PyObject* before, PyObject* after) {
    auto set = [](PyObject*& slot, PyObject* fn) {
        PyObject* old = slot;
        slot = fn && fn != Py_None ? Py_NewRef(fn) : nullptr;
        Py_XDECREF(old);
    };
    set(g_before, before);
    set(g_after, after);
    g_hooked.store(g_before || g_after);
}
