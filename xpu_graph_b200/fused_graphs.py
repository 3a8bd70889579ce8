"""The benchmark graphs after the ``cuda_sm100`` rewrite, assembled directly from the target's operators.

Each class takes the eager model from ``workloads.py``, shares its parameters (no copies) and runs, in ``forward``, the fused-op
sequence that xpu_graph's pattern pass produces for that model with this target, as one native operator (csrc/torch_ops.cpp): bit
for bit the results of the replacement modules called one after the other, with fewer launches where the operator joins two (q
and k of few rows; the recommender's copies and lookups). A compiled graph calls the modules; no pattern emits these operators.
They let the fused path run (and be measured) where the xpu_graph package itself is not installed; tests/test_target_patterns.py
checks, where it is, that compiling the eager model through XpuGraph yields that op sequence. Inference only: results carry no
gradient.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from . import ops  # noqa: F401  (registers torch.ops.xg_sm100.*)
from .workloads import EncoderBlock, LlamaDecoderLayer, RecsysGraph

_X = torch.ops.xg_sm100
_encoder_block, _decoder_layer, _recommender = _X.encoder_block.default, _X.decoder_layer.default, _X.recommender.default


class FusedLlamaDecoderLayer(nn.Module):
    """RMSNorm | 2x dense with the RoPE epilogue (q, k) | dense (v) | flash SDPA | dense(+residual) | RMSNorm |
    dual-GEMM SwiGLU | dense(+residual). The two residual adds ride in the GEMM epilogues (the [M, N] addend
    form of the dense layer) and RoPE in the q/k projections' epilogues, so the block is 9 kernels; with few rows
    the q and k projections are one launch (8 kernels), and v with them where the dense layer would not split K for it
    (7 kernels): every result has the bits that the op sequence gives."""

    def __init__(self, layer: LlamaDecoderLayer, fuse_swiglu_gemm: bool = True, fuse_rope_gemm: bool = True):
        super().__init__()
        self.layer = layer
        self.fuse_rope_gemm = fuse_rope_gemm and layer.head_dim in (64, 128)
        self.heads, self.head_dim = layer.heads, layer.head_dim
        self.eps1, self.eps2 = layer.input_norm.eps, layer.post_norm.eps
        self.fuse_swiglu_gemm = fuse_swiglu_gemm

    def forward(self, x, cos, sin):
        L = self.layer
        weights = [L.input_norm.weight, L.q_proj.weight, L.k_proj.weight, L.v_proj.weight, L.o_proj.weight, L.post_norm.weight,
                   L.gate_proj.weight, L.up_proj.weight, L.down_proj.weight]
        with torch.no_grad():
            return _decoder_layer(x, cos, sin, weights, self.eps1, self.eps2, self.heads, self.fuse_rope_gemm, self.fuse_swiglu_gemm)


class FusedEncoderBlock(nn.Module):
    """LayerNorm | dense+bias | SDPA | dense+bias(+residual) | LayerNorm | dense+bias+GELU | dense+bias(+residual)."""

    def __init__(self, block: EncoderBlock):
        super().__init__()
        self.block = block

    def forward(self, x):
        b = self.block
        params = []
        for m in (b.ln1, b.qkv, b.proj, b.ln2, b.fc1, b.fc2):
            params += (m.weight, m.bias)
        with torch.no_grad():
            return _encoder_block(x, params, b.ln1.eps, b.ln2.eps, b.heads)


class FusedRecsysGraph(nn.Module):
    """slice+cat of the dense features (one copy kernel) | 26 embedding lookups + where + stack (one
    gather kernel) | cat | 3x dense+bias+ReLU. Where the first layer is large enough for the fp32 tensor-core path
    the three copies are one kernel that writes that layer's operand."""

    def __init__(self, graph: RecsysGraph):
        super().__init__()
        self.graph = graph
        w = graph.n_dense // graph.n_groups
        self.starts = [g * w for g in graph.perm]
        self.ends = [s + w for s in self.starts]

    def forward(self, dense, idx, mask):
        G = self.graph
        # (iterating a ParameterList looks every member up by name: 16 us for 26 tables)
        tables = list(G.tables._parameters.values())
        if len(tables) != len(G.tables):
            tables = list(G.tables)
        weights, biases = [m.weight for m in G.layers], [m.bias for m in G.layers]
        with torch.no_grad():
            return _recommender(dense, idx, mask, tables, self.starts, self.ends, weights, biases)
