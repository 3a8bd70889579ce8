"""The custom ops of the ``cuda_sm100`` target (namespace ``xg_sm100``) as Python sees them.

The operators are native: libxg_sm100_torch.so (csrc/torch_ops.cpp) defines their schemas and CUDA kernels, which validate
the tensors, allocate the outputs and hand raw pointers, extents and the current CUDA stream to the C ABI of libxg_sm100.so.
This module loads that library, adds the fake implementations through which the graph compiler propagates shapes, and holds
the two grouped operators whose work is mostly list handling. Ops are functional and have CUDA kernels only (there is no CPU
implementation on purpose).

Registration pattern follows passes/patterns/targets/mlu/triton_kernel/fused_slice_where_cat.py:75,132
(``custom_op`` + ``register_fake``) of the reference.
"""
from __future__ import annotations

import sys
import types
from typing import List, Optional, Sequence

import torch

from . import lib as _lib

NS = "xg_sm100"

_lib.load_torch_ops()

_DTYPE_CODE = {torch.float32: _lib.XG_F32, torch.bfloat16: _lib.XG_BF16, torch.float16: _lib.XG_F16}


class NativeOp:
    """One operator of libxg_sm100_torch.so: callable, and open for fake and further device kernels."""

    def __init__(self, name: str):
        self.qualname = f"{NS}::{name}"
        self._overload = getattr(getattr(torch.ops, NS), name).default

    def __call__(self, *args, **kwargs):
        return self._overload(*args, **kwargs)

    def register_fake(self, fn):
        return torch.library.register_fake(self.qualname, fn)

    def register_kernel(self, device_types):
        return torch.library.impl(self.qualname, device_types)


def _code(dtype: torch.dtype) -> int:
    try:
        return _DTYPE_CODE[dtype]
    except KeyError:
        raise TypeError(f"xg_sm100: unsupported dtype {dtype}") from None


def _stream(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


def _row_stride(x2: torch.Tensor) -> int:
    return x2.stride(0) if x2.shape[0] > 1 else max(x2.stride(0), x2.shape[1])


def _empty_like_layout(x: torch.Tensor) -> torch.Tensor:
    """[B, H, S, D] output in the order of x's memory: a [B, S, H, D] buffer with dims 1 and 2 swapped when x's heads lie
    closer together than its positions (so that the transpose + reshape after attention stays a view); contiguous
    otherwise."""
    B, H, S, D = x.shape
    if x.stride(3) == 1 and x.stride(1) < x.stride(2) and H > 1 and S > 1:
        return torch.empty((B, S, H, D), dtype=x.dtype, device=x.device).transpose(1, 2)
    return torch.empty((B, H, S, D), dtype=x.dtype, device=x.device)


# --------------------------------------------------------------------------------------------
# normalisation
# --------------------------------------------------------------------------------------------
rms_norm = NativeOp("rms_norm")


@rms_norm.register_fake
def _(x, weight, eps):
    return torch.empty(x.shape, dtype=x.dtype, device=x.device)


add_rms_norm = NativeOp("add_rms_norm")


@add_rms_norm.register_fake
def _(x, residual, weight, eps):
    return [torch.empty(x.shape, dtype=x.dtype, device=x.device), torch.empty(x.shape, dtype=x.dtype, device=x.device)]


add_rms_norm_y = NativeOp("add_rms_norm_y")


@add_rms_norm_y.register_fake
def _(x, residual, weight, eps):
    return torch.empty(x.shape, dtype=x.dtype, device=x.device)


layer_norm = NativeOp("layer_norm")


@layer_norm.register_fake
def _(x, weight, bias, eps):
    return torch.empty(x.shape, dtype=x.dtype, device=x.device)


add_layer_norm = NativeOp("add_layer_norm")


@add_layer_norm.register_fake
def _(x, residual, weight, bias, eps):
    return [torch.empty(x.shape, dtype=x.dtype, device=x.device), torch.empty(x.shape, dtype=x.dtype, device=x.device)]


add_layer_norm_y = NativeOp("add_layer_norm_y")


@add_layer_norm_y.register_fake
def _(x, residual, weight, bias, eps):
    return torch.empty(x.shape, dtype=x.dtype, device=x.device)


# --------------------------------------------------------------------------------------------
# elementwise
# --------------------------------------------------------------------------------------------
# x: [B, H, S, D] (any strides with D contiguous); cos/sin broadcastable from [S, D].
rope = NativeOp("rope")


@rope.register_fake
def _(x, cos, sin):
    return _empty_like_layout(x)


swiglu = NativeOp("swiglu")


@swiglu.register_fake
def _(gate, up):
    return torch.empty(gate.shape, dtype=gate.dtype, device=gate.device)


# --------------------------------------------------------------------------------------------
# dense layers
# --------------------------------------------------------------------------------------------
def _mat(t: torch.Tensor) -> torch.Tensor:
    return t if t.stride(-1) == 1 else t.contiguous()


def _weight_rows(w: torch.Tensor, weight_trans: bool):
    """A 2-D weight with contiguous rows and the orientation flag that goes with it. A transposed view of a contiguous
    matrix (``w.T``, what F.linear(x, w.T) or x @ w.t() hand over) is read through its base in the other orientation -
    the kernels take both [N, K] and [K, N] - instead of being copied on every call."""
    if w.dim() == 2 and w.stride(-1) != 1 and w.stride(0) == 1 and w.shape[0] > 1:
        return w.t(), not weight_trans
    return _mat(w), weight_trans


# Which fp32 dense layers run on the tensor cores is decided in one place, csrc/torch_ops.cpp; F32_TENSOR_MIN_FLOPS and
# F32_TENSOR_MAX_K are its variables under these names (see _Settings below), so that setting one moves operators and rewrites alike.
def _f32_on_tensor_cores(M: int, N: int, K: int) -> bool:
    return bool(_lib.load_torch_ops().xg_torch_f32_on_tensor_cores(int(M), int(N), int(K)))


class _Settings(types.ModuleType):
    """This module's type."""

    @property
    def F32_TENSOR_MIN_FLOPS(self) -> int:
        return _lib.torch_setting("xg_torch_f32_min_flops").value

    @F32_TENSOR_MIN_FLOPS.setter
    def F32_TENSOR_MIN_FLOPS(self, value: int) -> None:
        _lib.torch_setting("xg_torch_f32_min_flops").value = int(value)

    @property
    def F32_TENSOR_MAX_K(self) -> int:
        return _lib.torch_setting("xg_torch_f32_max_k").value

    @F32_TENSOR_MAX_K.setter
    def F32_TENSOR_MAX_K(self, value: int) -> None:
        _lib.torch_setting("xg_torch_f32_max_k").value = int(value)


sys.modules[__name__].__class__ = _Settings


def _planes_tag(weight: torch.Tensor, weight_trans: bool):
    """Key under which a weight's bf16 planes are kept, or None when the tensor cannot be tracked: tensors made under
    torch.inference_mode() have no version counter, so their planes are rebuilt on every call."""
    try:
        version = weight._version
    except RuntimeError:
        return None
    return (version, weight.data_ptr(), tuple(weight.shape), tuple(weight.stride()), bool(weight_trans))


def invalidate_weight_planes(weight: torch.Tensor) -> None:
    """Drop the bf16 planes kept for an fp32 weight. Needed after the weight was rewritten through ``.data`` (or any
    other route that does not bump its version counter): the planes are keyed on the counter and would go stale."""
    try:
        del weight._xg_bf16_planes
    except AttributeError:
        pass


def dense_tower_eligible(M: int, dims: Sequence[int]) -> bool:
    """Every layer of an fp32 tower [K0 -> K1 -> ... -> Kn] over M rows qualifies for the tensor-core path."""
    return all(_f32_on_tensor_cores(M, dims[i + 1], dims[i]) for i in range(len(dims) - 1))


def mlp2_eligible(M: int, K1: int, N1: int, N2: int, dtype: torch.dtype, trans1: bool = True, trans2: bool = True) -> bool:
    """Two chained 16-bit dense layers [K1 -> N1 -> N2] fit the single-kernel form: 16 <= N1 <= 256 with N1 % 8 == 0,
    N2 <= 256, K1 % 8 == 0 (the limits of xg_mlp2_supported); a weight stored [K, N] (not transposed) needs N % 8 == 0."""
    return (dtype in (torch.bfloat16, torch.float16) and M > 0 and K1 >= 8 and K1 % 8 == 0
            and 16 <= N1 <= 256 and N1 % 8 == 0 and 1 <= N2 <= 256 and (bool(trans2) or N2 % 8 == 0))


# act2(act1(x @ W1 + b1) @ W2 + b2) in one kernel; weight l is given as [N, K] (nn.Linear's layout) or, if bit l of
# weights_kn is set, as [K, N]; the hidden activation stays on chip (rounded to the tensors' 16-bit dtype between
# the layers, as the unfused graph does).
mlp2 = NativeOp("mlp2")


@mlp2.register_fake
def _(x, w1, b1, w2, b2, act1, act2, weights_kn=0):
    return torch.empty((x.shape[0], w2.shape[1] if (weights_kn >> 1) & 1 else w2.shape[0]), dtype=x.dtype, device=x.device)


def mlp3_eligible(M: int, K1: int, N1: int, N2: int, N3: int, dtype: torch.dtype, trans=(True, True, True)) -> bool:
    """Three chained 16-bit dense layers fit the single-kernel form (the limits of xg_mlp3_supported)."""
    return (mlp2_eligible(M, K1, N1, N2, dtype, trans[0], trans[1]) and 16 <= N2 and N2 % 8 == 0
            and 1 <= N3 <= 256 and (bool(trans[2]) or N3 % 8 == 0))


# Three chained dense layers in one kernel (see mlp2).
mlp3 = NativeOp("mlp3")


@mlp3.register_fake
def _(x, w1, b1, w2, b2, w3, b3, act1, act2, act3, weights_kn=0):
    return torch.empty((x.shape[0], w3.shape[1] if (weights_kn >> 2) & 1 else w3.shape[0]), dtype=x.dtype, device=x.device)


MLP_SMALL_MAX_DIM = 128
MLP_SMALL_MAX_WEIGHTS = 24576


def _small_run(dims: Sequence[int], i: int, n: int, dtype: torch.dtype, M: int) -> int:
    """How many layers starting at layer i (at most three) run together on the weights-in-shared-memory kernel."""
    for run in (3, 2):
        if i + run <= n and mlp_small_worth_it(M, dims[i:i + run + 1], dtype):
            return run
    return 1


def mlp_small_worth_it(M: int, dims: Sequence[int], dtype: torch.dtype) -> bool:
    """The one-launch FMA tower is the faster form where a launch per layer is mostly launch and latency: few rows, or
    very narrow layers. Measured on B200 (us, one kernel / a launch per layer): 16 rows of 20 -> 32 -> 16 -> 1 fp16
    8.3 / 26.5; 16384 rows of 64 -> 32 -> 16 -> 1 fp32 20.5 / 21.7; 16384 rows of 128 -> 64 -> 32 fp32 43.5 / 24.6."""
    if dtype not in _DTYPE_CODE or not 1 <= len(dims) - 1 <= 3:
        return False
    return bool(_lib.load_torch_ops().xg_torch_small_tower_worth_it(int(M), _lib.i64_array(list(dims)), len(dims) - 1, _DTYPE_CODE[dtype]))


def mlp_small_eligible(dims: Sequence[int], dtype: torch.dtype) -> bool:
    """A tower [K0 -> N1 -> ... ] of one to three layers fits the weights-in-shared-memory kernel (the limits of
    xg_mlp_small_supported: every width <= 128, at most 24576 weight elements with K padded to a multiple of 4)."""
    n = len(dims) - 1
    if dtype not in (torch.float32, torch.bfloat16, torch.float16) or not 1 <= n <= 3:
        return False
    if any(d < 1 or d > MLP_SMALL_MAX_DIM for d in dims):
        return False
    return sum(((dims[i] + 3) // 4 * 4) * dims[i + 1] for i in range(n)) <= MLP_SMALL_MAX_WEIGHTS


# One to three chained narrow dense layers in one launch with every weight resident in shared memory (FMA
# arithmetic, fp32 accumulation, any row length); weight l is [N, K] unless bit l of weights_kn says [K, N].
mlp_small = NativeOp("mlp_small")


@mlp_small.register_fake
def _(x, weights, biases, act_names, weights_kn):
    w = weights[-1]
    last = len(weights) - 1
    return torch.empty((x.shape[0], w.shape[1] if (weights_kn >> last) & 1 else w.shape[0]), dtype=x.dtype, device=x.device)


# A chain of fp32 dense layers y_i = act_i(y_{i-1} @ W_i + b_i); act_names = "relu,relu,none" (one per layer). On
# the tensor-core path every inner layer's epilogue writes its result straight as the next layer's three bf16
# planes, so no fp32 activation is stored or re-read between layers; the last layer stores fp32.
dense_tower = NativeOp("dense_tower")


@dense_tower.register_fake
def _(x, weights, weight_trans, biases, act_names):
    N = weights[-1].shape[0] if weight_trans[-1] else weights[-1].shape[1]
    return torch.empty((x.shape[0], N), dtype=x.dtype, device=x.device)


# act(x @ W + bias + residual); W = weight ([K, N]) or weight^T (weight is [N, K], weight_trans).
dense = NativeOp("dense")


@dense.register_fake
def _(x, weight, weight_trans, bias, residual, act):
    N = weight.shape[0] if weight_trans else weight.shape[1]
    return torch.empty((x.shape[0], N), dtype=x.dtype, device=x.device)


# Batched dense: x [b, M, K], weight [b, K, N] or [b, N, K]; bias [b, 1, N] / [b, N]; residual [b, M, N].
batch_dense = NativeOp("batch_dense")


@batch_dense.register_fake
def _(x, weight, weight_trans, bias, residual, act):
    N = weight.shape[1] if weight_trans else weight.shape[2]
    return torch.empty((x.shape[0], x.shape[1], N), dtype=x.dtype, device=x.device)


@torch.library.custom_op(f"{NS}::combo_dense", mutates_args=(), device_types="cuda")
def combo_dense(inputs: List[torch.Tensor], weights: List[torch.Tensor], weight_trans: bool,
                biases: List[Optional[torch.Tensor]], act: str) -> torch.Tensor:
    """T same-shape dense layers act(x_t @ W_t + b_t) in one launch; returns the stacked [T, M, N] result. Operands are
    used in place through the grouped kernels (a pointer per layer, no stacking copy: tensor-core kernel for 16-bit,
    FMA kernel for fp32); what those cannot address goes through the batched form, for which operands that are not
    consecutive slabs of one buffer are stacked first. b_t: None, a row of N, or a full [M, N] addend."""
    T = len(inputs)
    if T == 0 or len(weights) != T or len(biases) != T:
        raise ValueError("xg_sm100::combo_dense: one input, weight and bias entry per layer")
    if any(t is not None and t.device != inputs[0].device for t in (*inputs, *weights, *biases)):
        raise ValueError(f"xg_sm100::combo_dense: all tensors must be on {inputs[0].device}")
    grouped = _combo_dense_grouped(inputs, weights, weight_trans, biases, act)
    if grouped is not None:
        return grouped
    x = _stack_or_view(inputs)
    w = _stack_or_view(weights)
    M = inputs[0].shape[0]
    N = weights[0].shape[0] if weight_trans else weights[0].shape[1]
    kinds = {_bias_kind(b, M, N) for b in biases}
    if len(kinds) != 1:
        raise ValueError("xg_sm100::combo_dense: the layers' biases must be of one kind (none, a row of N, or [M, N])")
    kind = kinds.pop()
    b = torch.stack([bi.reshape(1, -1) for bi in biases]) if kind == 1 else None  # [T, 1, N]
    r = torch.stack([bi.reshape(M, N) for bi in biases]) if kind == 2 else None   # [T, M, N]
    return batch_dense(x, w, weight_trans, b, r, act)


def _bias_kind(b: Optional[torch.Tensor], M: int, N: int) -> int:
    """0: none; 1: a per-column bias ([N] or [1, N]); 2: a full [M, N] addend (dense_layer_modules.py:22-57)."""
    if b is None:
        return 0
    if b.numel() == N and (b.dim() == 1 or (b.dim() == 2 and b.shape[0] == 1)):
        return 1
    if b.dim() == 2 and tuple(b.shape) == (M, N):
        return 2
    raise ValueError(f"xg_sm100::combo_dense: bias of shape {tuple(b.shape)} for an [{M}, {N}] result")


def _combo_dense_grouped(inputs, weights, weight_trans: bool, biases, act: str) -> Optional[torch.Tensor]:
    """The grouped launch: every layer's operands are used where they are (a pointer per entry), the results land side
    by side in one [T, M, N] tensor. A bias is a row of N or a full [M, N] addend, layer by layer. Returns None when
    the operands do not qualify (shapes that differ; 16-bit rows a tensor map cannot address), and the caller falls back
    to the stacked batched form."""
    x0, w0 = inputs[0], weights[0]
    if x0.dtype not in (torch.bfloat16, torch.float16, torch.float32) or x0.dim() != 2 or w0.dim() != 2:
        return None
    tc = x0.dtype != torch.float32
    xs = [_mat(t) for t in inputs]
    rows = [_weight_rows(t, weight_trans) for t in weights]
    if any(r[1] != rows[0][1] for r in rows):
        return None
    ws, weight_trans = [r[0] for r in rows], rows[0][1]
    M, K = xs[0].shape
    N = ws[0].shape[0] if weight_trans else ws[0].shape[1]
    lda, ldw = _row_stride(xs[0]), _row_stride(ws[0])
    for x, w in zip(xs, ws):
        if (x.shape != xs[0].shape or w.shape != ws[0].shape or x.dtype != x0.dtype or w.dtype != x0.dtype
                or _row_stride(x) != lda or _row_stride(w) != ldw or (tc and (x.data_ptr() % 16 or w.data_ptr() % 16))):
            return None
    if (ws[0].shape[1] if weight_trans else ws[0].shape[0]) != K or (tc and (lda % 8 or ldw % 8)):
        return None
    kinds = [_bias_kind(b, M, N) for b in biases]
    bs = [b.reshape(-1).to(x0.dtype).contiguous() if k == 1 else None for b, k in zip(biases, kinds)]
    rs = [_mat(b.to(x0.dtype)) if k == 2 else None for b, k in zip(biases, kinds)]
    ldr = 0
    if any(r is not None for r in rs):
        strides = {_row_stride(r) for r in rs if r is not None}
        if len(strides) != 1:
            rs = [None if r is None else r.contiguous() for r in rs]
            strides = {N}
        ldr = strides.pop()
    out = torch.empty((len(xs), M, N), dtype=x0.dtype, device=x0.device)
    step = M * N * out.element_size()
    rc = _lib.load().xg_gemm_group_bias_act(
        _lib.ptr_array([x.data_ptr() for x in xs]), _lib.ptr_array([w.data_ptr() for w in ws]),
        _lib.ptr_array([0 if b is None else b.data_ptr() for b in bs]), _lib.ptr_array([0 if r is None else r.data_ptr() for r in rs]),
        _lib.ptr_array([out.data_ptr() + i * step for i in range(len(xs))]),
        len(xs), M, N, K, lda, ldw, N, ldr, 1 if weight_trans else 0, _lib.ACT_CODES[act], _code(x0.dtype), _stream(x0))
    _lib.check(rc, "xg_gemm_group_bias_act")
    return out


def _stack_or_view(ts: Sequence[torch.Tensor]) -> torch.Tensor:
    """[T, ...] tensor of the list's members: a view when they are equally spaced contiguous slabs of one storage
    (the outputs of an unbind / split), else a stacked copy."""
    t0 = ts[0]
    if len(ts) > 1 and all(t.is_contiguous() and t.shape == t0.shape and t.dtype == t0.dtype for t in ts):
        step = ts[1].data_ptr() - t0.data_ptr()
        same_store = all(t.untyped_storage().data_ptr() == t0.untyped_storage().data_ptr() for t in ts)
        if same_store and step == t0.numel() * t0.element_size() and all(
                ts[i].data_ptr() - t0.data_ptr() == i * step for i in range(len(ts))):
            return t0.as_strided((len(ts),) + tuple(t0.shape), (t0.numel(),) + tuple(t0.stride()), t0.storage_offset())
    return torch.stack(list(ts))


@combo_dense.register_fake
def _(inputs, weights, weight_trans, biases, act):
    N = weights[0].shape[0] if weight_trans else weights[0].shape[1]
    return torch.empty((len(inputs), inputs[0].shape[0], N), dtype=inputs[0].dtype, device=inputs[0].device)


@torch.library.custom_op(f"{NS}::combo_batch_dense", mutates_args=(), device_types="cuda")
def combo_batch_dense(inputs: List[torch.Tensor], weights: List[torch.Tensor], weight_trans: bool,
                      biases: List[Optional[torch.Tensor]], act: str) -> torch.Tensor:
    """T same-shape batched dense layers act(bmm(x_t, W_t) + b_t), x_t [S, M, K], W_t [S, K, N] (or [S, N, K]), in one
    grouped launch over the T * S matrix products (a pointer per product: batch entries of a member, also broadcast
    ones, are addressed where they lie); returns [T, S, M, N]. b_t: None, a full [S, M, N] addend, or anything that
    broadcasts to [S, 1, N]."""
    T = len(inputs)
    if T == 0 or len(weights) != T or len(biases) != T:
        raise ValueError("xg_sm100::combo_batch_dense: one input, weight and bias entry per layer")
    S, M, _ = inputs[0].shape
    N = weights[0].shape[1] if weight_trans else weights[0].shape[2]
    xs, ws, bs = [], [], []
    for x, w, b in zip(inputs, weights, biases):
        if x.dim() != 3 or w.dim() != 3 or x.shape[0] != S or w.shape[0] != S:
            raise ValueError("xg_sm100::combo_batch_dense: every member is [S, M, K] x [S, K, N] with one S")
        if b is not None:
            b = b if tuple(b.shape) == (S, M, N) else b.broadcast_to((S, 1, N))
        for i in range(S):
            xs.append(x[i])
            ws.append(w[i])
            bs.append(None if b is None else b[i])
    return combo_dense(xs, ws, weight_trans, bs, act).view(T, S, M, N)


@combo_batch_dense.register_fake
def _(inputs, weights, weight_trans, biases, act):
    S, M, _ = inputs[0].shape
    N = weights[0].shape[1] if weight_trans else weights[0].shape[2]
    return torch.empty((len(inputs), S, M, N), dtype=inputs[0].dtype, device=inputs[0].device)


# silu(x @ w_gate^T) * (x @ w_up^T); weights in Linear layout [N, K].
dense_swiglu = NativeOp("dense_swiglu")


@dense_swiglu.register_fake
def _(x, w_gate, w_up):
    return torch.empty((x.shape[0], w_gate.shape[0]), dtype=x.dtype, device=x.device)


# rope(x @ weight^T) with the rotation in the GEMM epilogue. x: [B*S, K] (row r is token r % seq_len of its
# sequence), weight: [H*D, K]; cos/sin broadcastable from [S, D]. Returns [B*S, H*D].
dense_rope = NativeOp("dense_rope")


@dense_rope.register_fake
def _(x, weight, cos, sin, seq_len, head_dim):
    return torch.empty((x.shape[0], weight.shape[0]), dtype=x.dtype, device=x.device)


# --------------------------------------------------------------------------------------------
# attention
# --------------------------------------------------------------------------------------------
# q [B,H,Sq,D], k/v [B,H,Skv,D]; attn_mask: additive (same dtype) or boolean, broadcastable to [B,H,Sq,Skv].
sdpa = NativeOp("sdpa")


@sdpa.register_fake
def _(q, k, v, attn_mask, scale, is_causal):
    return _empty_like_layout(q if q.stride(3) == 1 else q.contiguous())


# --------------------------------------------------------------------------------------------
# copy fusions (bit-exact)
# --------------------------------------------------------------------------------------------
def _norm_slices(width: int, starts: Sequence[int], ends: Sequence[int]):
    out = []
    for s, e in zip(starts, ends):
        s = s + width if s < 0 else s
        e = e + width if e < 0 else e
        s = min(max(s, 0), width)
        e = min(max(e, s), width)
        out.append((s, e))
    return out


# cat([src[:, s:e] for s, e in zip(starts, ends)], -1) of a 2-D src; rows where (row_mask != 0) == zero_when are
# written as zeros.
slice_cat = NativeOp("slice_cat")


@slice_cat.register_fake
def _(src, starts, ends, row_mask, zero_when):
    segs = _norm_slices(src.shape[1], starts, ends)
    return torch.empty((src.shape[0], sum(e - s for s, e in segs)), dtype=src.dtype, device=src.device)


# slice_cat where the row mask applies to the slices flagged in `masked` only (cat([x[:, a:b], where(m, 0, x[:,
# c:d]), ...], -1)): the masked and the unmasked slices are two passes of the segmented copy into one output buffer.
slice_cat_partly_masked = NativeOp("slice_cat_partly_masked")


@slice_cat_partly_masked.register_fake
def _(src, starts, ends, masked, row_mask, zero_when):
    segs = _norm_slices(src.shape[1], starts, ends)
    return torch.empty((src.shape[0], sum(e - s for s, e in segs)), dtype=src.dtype, device=src.device)


def _checked_starts(width: int, starts: Sequence[int], slice_len: int) -> List[int]:
    """Slice starts with negative values wrapped; every slice [s, s + slice_len) has to lie inside the row. The
    reference derives slice_len as end - start of the raw aten.slice arguments (structure/fuse_slice.py:28), so a slice
    that aten would have clamped (an end past the width, INT64_MAX) arrives here with a length the row does not
    have: that is refused instead of read past the row."""
    if slice_len < 0:
        raise ValueError(f"xg_sm100::multi_slice: negative slice length {slice_len}")
    out = []
    for s in starts:
        s = s + width if s < 0 else s
        if s < 0 or s + slice_len > width:
            raise ValueError(f"xg_sm100::multi_slice: slice [{s}, {s + slice_len}) is outside a row of {width} elements")
        out.append(s)
    return out


# stack([src[..., s:s+slice_len] for s in starts], 0) -> [num, *src.shape[:-1], slice_len].
multi_slice = NativeOp("multi_slice")


@multi_slice.register_fake
def _(src, starts, slice_len):
    _checked_starts(src.shape[-1], starts, slice_len)
    return torch.empty([len(starts)] + list(src.shape[:-1]) + [slice_len], dtype=src.dtype, device=src.device)


# multi_slice of a 2-D src where the slices flagged in `masked` are written as zeros in the rows where (row_mask !=
# 0) == zero_when: stack([x[:, a:a+L], where(m, 0, x[:, b:b+L]), ...], 0) -> [num, rows, L].
multi_slice_masked = NativeOp("multi_slice_masked")


@multi_slice_masked.register_fake
def _(src, starts, slice_len, masked, row_mask, zero_when):
    _checked_starts(src.shape[-1], starts, slice_len)
    return torch.empty((len(starts), src.shape[0], slice_len), dtype=src.dtype, device=src.device)


# Several slice_cat results of one 2-D src in one pass: output k concatenates the next counts[k] (start, end) pairs.
slice_cat_multi = NativeOp("slice_cat_multi")


@slice_cat_multi.register_fake
def _(src, starts, ends, counts):
    segs = _norm_slices(src.shape[1], starts, ends)
    outs, pos = [], 0
    for c in counts:
        outs.append(torch.empty((src.shape[0], sum(e - s for s, e in segs[pos:pos + c])), dtype=src.dtype, device=src.device))
        pos += c
    return outs


# cat(xs, -1) for tensors that agree on every leading dim (stack along a new trailing-but-one dim is the same copy
# followed by a view).
cat_lastdim = NativeOp("cat_lastdim")


@cat_lastdim.register_fake
def _(xs, row_mask, zero_when):
    return torch.empty(list(xs[0].shape[:-1]) + [sum(x.shape[-1] for x in xs)], dtype=xs[0].dtype, device=xs[0].device)


# out[r, f*D:(f+1)*D] = tables[f][idx[r, f]] (zeros where the row mask says so): F embedding lookups, the where-mask
# and the stack in one pass. idx: int64 [rows, F].
gather_stack = NativeOp("gather_stack")


@gather_stack.register_fake
def _(tables, idx, row_mask, zero_when):
    return torch.empty((idx.shape[0], len(tables) * tables[0].shape[1]), dtype=tables[0].dtype, device=idx.device)


# [sum(x, dim) for x in inputs] for 3-D tensors, one launch for the whole list.
sum3d = NativeOp("sum3d")


@sum3d.register_fake
def _(inputs, dim):
    outs = []
    for x in inputs:
        s0, s1, s2 = x.shape
        oshape = (s1, s2) if dim == 0 else ((s0, s2) if dim == 1 else (s0, s1))
        outs.append(torch.empty(oshape, dtype=x.dtype, device=x.device))
    return outs


# ---- row sums written side by side -----------------------------------------------------------------
# cat([src[:, s:e, :].sum(1) for s, e in zip(starts, ends)], -1) for a [B, R, C] tensor.
slice_sum_cat = NativeOp("slice_sum_cat")


@slice_sum_cat.register_fake
def _(src, starts, ends):
    return torch.empty((src.shape[0], len(starts) * src.shape[2]), dtype=src.dtype, device=src.device)


# cat([x.sum(1) for x in inputs], -1) for [B, R_k, C] tensors.
sum_cat = NativeOp("sum_cat")


@sum_cat.register_fake
def _(inputs):
    return torch.empty((inputs[0].shape[0], len(inputs) * inputs[0].shape[2]), dtype=inputs[0].dtype, device=inputs[0].device)


# cat([(a * b).sum(1) for a, b in zip(lhs, rhs)], -1) for [B or 1, R, C] tensors (batch broadcast).
mul_sum_cat = NativeOp("mul_sum_cat")


@mul_sum_cat.register_fake
def _(lhs, rhs):
    batch = max(max(a.shape[0], b.shape[0]) for a, b in zip(lhs, rhs))
    return torch.empty((batch, len(lhs) * lhs[0].shape[2]), dtype=lhs[0].dtype, device=lhs[0].device)


# ---- whole graphs (fused_graphs.py) -----------------------------------------------------------------
encoder_block = NativeOp("encoder_block")
decoder_layer = NativeOp("decoder_layer")
recommender = NativeOp("recommender")


@encoder_block.register_fake
def _(x, params, eps1, eps2, heads):
    return torch.empty(x.shape, dtype=x.dtype, device=x.device)


@decoder_layer.register_fake
def _(x, cos, sin, weights, eps1, eps2, heads, fuse_rope, fuse_swiglu):
    return torch.empty(x.shape, dtype=x.dtype, device=x.device)


@recommender.register_fake
def _(features, idx, mask, tables, starts, ends, weights, biases):
    return torch.empty((features.shape[0], weights[-1].shape[0]), dtype=features.dtype, device=features.device)


OP_NAMES = tuple(name for name, op in list(globals().items()) if isinstance(op, (NativeOp, torch.library.CustomOpDef)))
