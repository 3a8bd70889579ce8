"""The work that programs hand to this package, as cases to be timed: whole fused graphs (decoder layer, encoder block,
recommender) and the fused patterns that a compiled graph calls on its own (dense layer, attention, residual + norm,
feature pooling), each through its public module.

``listed()`` names twelve of them, ``draw(rng)`` makes another one of the same ranges. A case is a dict of plain values;
``prepare`` makes its inputs and weights on the GPU from a seed, ``run`` makes one call, ``work`` counts the bytes and
operations the call cannot do without, ``tolerance`` says how far another correct result of the same precision may be off.
"""
from __future__ import annotations

import math

import torch

from xpu_graph_b200 import modules as M
from xpu_graph_b200.fused_graphs import FusedEncoderBlock, FusedLlamaDecoderLayer, FusedRecsysGraph
from xpu_graph_b200.workloads import EncoderBlock, LlamaDecoderLayer, RecsysGraph, rope_tables

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SIZE = {"f32": 4, "bf16": 2, "f16": 2}

# encoder block and recommender: the sizes of the package's own workloads
ENC_HIDDEN, ENC_HEADS, ENC_FFN = 256, 4, 1024
N_DENSE, N_SPARSE, EMB, TABLE_ROWS, MLP = 64, 26, 64, 100000, (1024, 512, 256)
MASKED_SHARE = 0.3  # rows whose lookups are masked out


def listed():
    return [
        # The decoder layer at the benchmark's size: a full prefill batch.
        {"name": "decoder 8x2048 bf16", "kind": "decoder", "batch": 8, "seq": 2048, "hidden": 4096, "heads": 32, "ffn": 11008},
        # The same layer on one short prompt of no particular length: latency of a request that arrives alone.
        {"name": "decoder 1x333 bf16", "kind": "decoder", "batch": 1, "seq": 333, "hidden": 4096, "heads": 32, "ffn": 11008},
        # The small encoder block in fp32: seven small launches, the latency of the host path and of each kernel.
        {"name": "encoder 2x128 f32", "kind": "encoder", "batch": 2, "seq": 128, "dtype": "f32"},
        # A serving batch of the same block in 16 bits, with a sequence length that is no multiple of a tile.
        {"name": "encoder 24x197 f16", "kind": "encoder", "batch": 24, "seq": 197, "dtype": "f16"},
        # The recommender at its offline batch: lookups, feature copies and the fp32 tower.
        {"name": "recommender 16384 f32", "kind": "recommender", "rows": 16384},
        # The recommender on one online request with some hundred candidates.
        {"name": "recommender 500 f32", "kind": "recommender", "rows": 500},
        # Residual + RMSNorm with both results kept, as every decoder layer has it, at a prefill batch.
        {"name": "norm rms 16384x4096 bf16", "kind": "norm", "norm": "rms", "rows": 16384, "hidden": 4096, "dtype": "bf16",
         "residual": True, "keep_sum": True},
        # Dense layer + activation with some hundred rows: a mixed serving batch.
        {"name": "dense 256x4096x11008 bf16", "kind": "dense", "m": 256, "k": 4096, "n": 11008, "dtype": "bf16", "act": "gelu",
         "residual": False},
        # Dense layer + residual with one row per sequence: a decoding step, bound by reading the weights.
        {"name": "dense 16x4096x4096 bf16", "kind": "dense", "m": 16, "k": 4096, "n": 4096, "dtype": "bf16", "act": "none",
         "residual": True},
        # Attention of padded sequences: every sequence of the batch has its own number of valid keys.
        {"name": "attention padded 4x32x500 f16", "kind": "attention", "batch": 4, "heads": 32, "sq": 500, "skv": 500, "d": 64,
         "dtype": "f16", "mask": "padding"},
        # Attention of a decoding step: one query per sequence against the keys so far.
        {"name": "attention 8x32x1x2048 bf16", "kind": "attention", "batch": 8, "heads": 32, "sq": 1, "skv": 2048, "d": 128,
         "dtype": "bf16", "mask": "none"},
        # Feature pooling in front of a recommender's tower: sums over ranges of a history, interaction sums, slices.
        {"name": "features 16384 f32", "kind": "features", "rows": 16384, "history": 50, "dim": 64, "pairs": 3, "pair_rows": 10,
         "slices": 16, "slice_len": 32, "dtype": "f32"},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], evenly spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi):
    """A row width: usually a multiple of 8 elements, now and then any number."""
    w = _log_int(rng, lo, hi)
    return w if rng.random() < 0.2 else max(8, w // 8 * 8)


def draw(rng):
    kind = rng.choice(["decoder", "encoder", "recommender", "norm", "dense", "dense", "attention", "attention", "features"])
    if kind == "decoder":
        small = rng.random() < 0.3
        return {"kind": kind, "batch": rng.randint(1, 8), "seq": _log_int(rng, 16, 2048), "hidden": 512 if small else 4096,
                "heads": 4 if small else 32, "ffn": 1376 if small else 11008}
    if kind == "encoder":
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "seq": _log_int(rng, 16, 512), "dtype": rng.choice(["f32", "bf16", "f16"])}
    if kind == "recommender":
        return {"kind": kind, "rows": _log_int(rng, 64, 16384)}
    if kind == "norm":
        residual = rng.random() < 0.7
        return {"kind": kind, "norm": rng.choice(["rms", "layer"]), "rows": _log_int(rng, 16, 65536), "hidden": _width(rng, 256, 8192),
                "dtype": rng.choice(["bf16", "bf16", "f16", "f32"]), "residual": residual, "keep_sum": residual and rng.random() < 0.6}
    if kind == "dense":
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        m, k, n = _log_int(rng, 1, 16384), _width(rng, 64, 11008), _width(rng, 64, 11008)
        # fp32 layers, and 16-bit ones whose rows are no multiples of 16 bytes, come to this package while they are small
        limit = 2 ** 37 if dtype == "f32" else 2 ** 26 if k % 8 else 2 ** 41
        m = max(1, min(m, limit // (2 * k * n)))
        if 2 * m * k * n > limit:
            k, n = min(k, 1001), min(n, 1001)
        return {"kind": kind, "m": m, "k": k, "n": n, "dtype": dtype, "act": rng.choice(["none", "gelu", "silu", "relu"]),
                "residual": rng.random() < 0.3}
    if kind == "attention":
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        mask = rng.choice(["none", "causal", "causal", "padding"])
        skv = _log_int(rng, 16, 512 if dtype == "f32" else 4096)
        sq = 1 if mask != "causal" and rng.random() < 0.3 else skv if rng.random() < 0.7 else _log_int(rng, 1, skv)
        return {"kind": kind, "batch": rng.randint(1, 8), "heads": rng.choice([4, 8, 16, 32]), "sq": sq, "skv": skv,
                "d": rng.choice([64, 128]), "dtype": dtype, "mask": mask}
    return {"kind": kind, "rows": _log_int(rng, 64, 32768), "history": rng.randint(5, 60), "dim": rng.choice([16, 32, 64, 100, 128]),
            "pairs": rng.randint(1, 4), "pair_rows": rng.randint(2, 16), "slices": rng.randint(4, 24), "slice_len": rng.randint(4, 64),
            "dtype": rng.choice(["f32", "f32", "bf16"])}


# ---- inputs ------------------------------------------------------------------------------------
def _history_ranges(history):
    """Pooling windows over a history, newest first: all of it, its half, its fifth, and the middle part."""
    return [(0, history), (0, max(1, history // 2)), (0, max(1, history // 5)), (history // 4, max(history // 4 + 1, history * 3 // 4))]


def _slices(case):
    """The blocks that a tower takes out of a wide row: equal widths, a gap of a few columns between them."""
    return [(i * (case["slice_len"] + 5), i * (case["slice_len"] + 5) + case["slice_len"]) for i in range(case["slices"])]


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    dtype = DTYPES[case.get("dtype", "bf16")]
    kind = case["kind"]

    def rn(*shape, std=1.0, dt=dtype):
        return torch.randn(*shape, generator=g, device=dev, dtype=torch.float32).mul_(std).to(dt)

    def fill(module, std, norms=()):
        with torch.no_grad():
            for p in module.parameters():
                p.normal_(0.0, std, generator=g)
            for norm in norms:
                norm.weight.normal_(1.0, 0.02, generator=g)
        return module.eval()

    with torch.no_grad(), torch.device(dev):
        if kind == "decoder":
            layer = LlamaDecoderLayer(case["hidden"], case["heads"], case["ffn"])
            layer = fill(layer, 0.02, (layer.input_norm, layer.post_norm)).to(dtype)
            cos, sin = rope_tables(case["seq"], case["hidden"] // case["heads"])
            return {"kind": kind, "graph": FusedLlamaDecoderLayer(layer),
                    "args": (rn(case["batch"], case["seq"], case["hidden"]), cos.to(dtype), sin.to(dtype))}
        if kind == "encoder":
            block = EncoderBlock(ENC_HIDDEN, ENC_HEADS, ENC_FFN)
            block = fill(block, 0.02, (block.ln1, block.ln2)).to(dtype)
            return {"kind": kind, "graph": FusedEncoderBlock(block), "args": (rn(case["batch"], case["seq"], ENC_HIDDEN),)}
        if kind == "recommender":
            graph = RecsysGraph(N_DENSE, 16, N_SPARSE, EMB, TABLE_ROWS, MLP)
            for t in graph.tables:
                t.normal_(0.0, 0.01, generator=g)
            for layer in graph.layers:
                fill(layer, 0.02)
            rows = case["rows"]
            idx = torch.randint(0, TABLE_ROWS, (rows, N_SPARSE), generator=g, device=dev, dtype=torch.int64)
            mask = torch.rand(rows, 1, generator=g, device=dev) < MASKED_SHARE
            return {"kind": kind, "graph": FusedRecsysGraph(graph), "args": (rn(rows, N_DENSE, dt=torch.float32), idx, mask)}
        if kind == "norm":
            rows, hidden = case["rows"], case["hidden"]
            x = rn(rows, hidden)
            residual = (rn(rows, hidden),) if case["residual"] else ()
            weight = (1.0 + rn(hidden, std=0.1, dt=torch.float32)).to(dtype)
            affine = (weight,) if case["norm"] == "rms" else (weight, rn(hidden, std=0.1))
            if case["norm"] == "rms":
                module = M.AddRMSNormModule(case["keep_sum"]) if residual else M.RMSNormModule()
            else:
                module = M.AddLayerNormModule(case["keep_sum"]) if residual else M.LayerNormModule()
            return {"kind": kind, "graph": module, "args": (x, *residual, *affine, 1e-5)}
        if kind == "dense":
            m, k, n = case["m"], case["k"], case["n"]
            x, w, b = rn(m, k), rn(n, k, std=0.02), rn(n, std=0.02)
            if case["residual"]:
                return {"kind": kind, "graph": M.DenseResidualModule(), "args": (x, w, True, b, rn(m, n), case["act"])}
            return {"kind": kind, "graph": M.DenseLayerModule(False), "args": (x, w, True, b, case["act"])}
        if kind == "attention":
            b, h, sq, skv, d = (case[key] for key in ("batch", "heads", "sq", "skv", "d"))
            # as the projections leave them: [batch, position, head, dim] buffers seen as [batch, head, position, dim]
            q, k, v = (rn(b, s, h, d).transpose(1, 2) for s in (sq, skv, skv))
            mask = None
            if case["mask"] == "padding":
                lengths = torch.randint((skv + 1) // 2, skv + 1, (b, 1, 1, 1), generator=g, device=dev)
                mask = torch.arange(skv, device=dev).view(1, 1, 1, skv) < lengths
            return {"kind": kind, "graph": M.SDPAModule(), "args": (q, k, v, mask, None, case["mask"] == "causal")}
        rows, dim = case["rows"], case["dim"]
        slices = _slices(case)
        lhs = [rn(rows, case["pair_rows"], dim) for _ in range(case["pairs"])]
        rhs = [rn(rows, case["pair_rows"], dim) for _ in range(case["pairs"])]
        return {"kind": kind, "history": rn(rows, case["history"], dim), "pool": M.SliceSumCatModule(_history_ranges(case["history"])),
                "pairs": [t for pair in zip(lhs, rhs) for t in pair], "interact": M.MulSumCatModule(), "wide": rn(rows, slices[-1][1] + 5),
                "slices": slices, "slice_cat": M.FuseSliceCatSameInputModule()}


def run(state):
    if state["kind"] == "features":
        return [state["pool"](state["history"]), state["interact"](state["pairs"]), state["slice_cat"](state["wide"], state["slices"])]
    return state["graph"](*state["args"])


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "decoder":
        h, f, s = case["hidden"], case["ffn"], case["seq"]
        t = case["batch"] * s
        weights = 4 * h * h + 3 * h * f
        return {"bytes": 2 * (weights + 2 * h + 2 * t * h + 2 * s * (h // case["heads"])),
                "flops": 2 * t * weights + 2 * case["batch"] * s * s * h}  # causal: half of q k^T and p v
    es = SIZE[case.get("dtype", "f32")]
    if kind == "encoder":
        h, f = ENC_HIDDEN, ENC_FFN
        t = case["batch"] * case["seq"]
        weights = 4 * h * h + 2 * h * f
        return {"bytes": es * (weights + 9 * h + f + 2 * t * h), "flops": 2 * t * weights + 4 * t * case["seq"] * h}
    if kind == "recommender":
        rows = case["rows"]
        dims = (N_DENSE + N_SPARSE * EMB,) + MLP
        weights = sum(a * b + b for a, b in zip(dims, dims[1:]))
        lookups = (1 - MASKED_SHARE) * N_SPARSE * (8 + 4 * EMB)  # a masked row's indices and table rows are not needed
        return {"bytes": rows * (4 * N_DENSE + lookups + 1 + 4 * MLP[-1]) + 4 * weights, "flops": 2 * rows * weights}
    if kind == "norm":
        per = 2 + case["residual"] + case["keep_sum"]
        return {"bytes": es * (per * case["rows"] * case["hidden"] + 2 * case["hidden"]), "flops": 8 * case["rows"] * case["hidden"]}
    if kind == "dense":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": es * (m * k + n * k + n + m * n * (2 if case["residual"] else 1)), "flops": 2 * m * k * n}
    if kind == "attention":
        b, h, sq, skv, d = (case[key] for key in ("batch", "heads", "sq", "skv", "d"))
        seen = sq * skv
        if case["mask"] == "causal":  # row i sees keys 0..i
            seen = sum(min(i + 1, skv) for i in range(sq))
            skv = min(skv, sq)
        elif case["mask"] == "padding":  # three quarters of the keys are valid on average
            seen, skv = seen * 3 // 4, skv * 3 // 4
        return {"bytes": es * b * h * d * (2 * sq + 2 * skv), "flops": 4 * b * h * seen * d}
    rows, dim = case["rows"], case["dim"]
    ranges = _history_ranges(case["history"])
    pooled = rows * dim * (case["history"] + len(ranges))
    pairs = rows * dim * case["pairs"] * (2 * case["pair_rows"] + 1)
    return {"bytes": es * (pooled + pairs + 2 * rows * case["slices"] * case["slice_len"]),
            "flops": rows * dim * (sum(b - a for a, b in ranges) + 2 * case["pairs"] * case["pair_rows"])}


def tolerance(case):
    # sums and products in 32 bits; results rounded to 16 bits with intermediate tensors rounded on the way
    if case["kind"] in ("recommender",):
        return {"rel": 1e-5}
    return {"rel": {"f32": 1e-5, "bf16": 1e-2, "f16": 2e-3}[case.get("dtype", "bf16")]}
