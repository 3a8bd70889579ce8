"""GPU parity of whole fused graphs against the eager (pattern-disabled) models on CPU."""
import pytest
import torch

from tests.helpers import assert_parity, error_stats

pytestmark = pytest.mark.gpu


def test_encoder_block_fp32(cuda_device):
    """Config 1: encoder block fp32, batch 2 x seq 128 x hidden 256, 4 heads, FFN 1024 GELU, seed 0."""
    from xpu_graph_b200.fused_graphs import FusedEncoderBlock
    from xpu_graph_b200.workloads import make_encoder

    model, x = make_encoder(seed=0)
    with torch.no_grad():
        want = model(x)
    got = FusedEncoderBlock(model.to(cuda_device))(x.to(cuda_device))
    assert_parity(got, want, "encoder block fp32")


@pytest.mark.parametrize("fuse_swiglu_gemm", [True, False])
def test_llama_layer_small(cuda_device, fuse_swiglu_gemm):
    """Config 4 at reduced size (hidden 512, 4 heads x 128, FFN 1376, batch 2 x seq 320), bf16, causal."""
    from xpu_graph_b200 import lib
    from xpu_graph_b200.fused_graphs import FusedLlamaDecoderLayer
    from xpu_graph_b200.workloads import make_llama_layer

    model, (x, cos, sin) = make_llama_layer(seed=3, batch=2, seq=320, hidden=512, heads=4, ffn=1376)
    with torch.no_grad():
        want = model(x, cos, sin)
        exact = model.float()(x.float(), cos.float(), sin.float())
    model = model.to(torch.bfloat16).to(cuda_device)
    got = FusedLlamaDecoderLayer(model, fuse_swiglu_gemm)(x.to(cuda_device), cos.to(cuda_device), sin.to(cuda_device))
    torch.cuda.synchronize()
    assert lib.tc_status() == 0
    assert_parity(got, want, "llama layer bf16")
    ours, theirs = error_stats(got, exact)[0], error_stats(want, exact)[0]
    print(f"max abs error vs fp32 math: fused {ours:.4g}, eager bf16 {theirs:.4g}")
    assert ours <= 2.0 * theirs + 1e-2


def test_llama_layer_benchmark_size(cuda_device):
    """Config 4 at the benchmark's size (hidden 4096, 32 heads x 128, FFN 11008, RoPE, causal, seed 3) on one
    2048-token sequence, against the eager (pattern-disabled) bf16 layer on CPU, in two parts.

    Op by op: each of the nine fused ops gets exactly the inputs its eager counterpart saw and must match it within
    the stated rel 2e-2 / abs 1e-2 (relative to the op's operands where a sum can cancel).

    End to end: two bf16 evaluations of a 4096 -> 11008 -> 4096 chain differ by more than that per element whichever
    two they are (the down projection adds up 11008 products whose bf16 inputs already differ in the last place: the
    noise is set by the row, not by the element, so small outputs miss any element-relative bound; measured here:
    eager bf16 itself is 0.011 mean / 0.093 max away from the same layer in fp32). The end-to-end gate is therefore
    against fp32 math: the fused layer must be at least as close to it as eager bf16 is. Max-abs and mean-rel against
    the eager result are printed."""
    from xpu_graph_b200 import lib
    from xpu_graph_b200 import modules as M
    from xpu_graph_b200.fused_graphs import FusedLlamaDecoderLayer
    from xpu_graph_b200.workloads import llama_layer_stages, make_llama_layer

    model, (x, cos, sin) = make_llama_layer(seed=3, batch=1, seq=2048, hidden=4096, heads=32, ffn=11008)
    B, S, Hd = x.shape
    H, D = model.heads, model.head_dim
    st = llama_layer_stages(model, x, cos, sin)
    with torch.no_grad():
        exact = model.float()(x.float(), cos.float(), sin.float())
    model = model.to(torch.bfloat16).to(cuda_device)
    dev = lambda t: t.to(cuda_device)  # noqa: E731
    rows = lambda t: dev(t).reshape(B * S, -1)  # noqa: E731
    cd, sd = dev(cos), dev(sin)
    norm, dense, drope = M.RMSNormModule(), M.DenseLayerModule(False), M.DenseRopeModule()
    eps = model.input_norm.eps

    assert_parity(norm(rows(x), model.input_norm.weight, eps).view(B, S, Hd), st["h1"], "op 1: RMSNorm")
    for name, w in (("q", model.q_proj.weight), ("k", model.k_proj.weight)):
        got = drope(rows(st["h1"]), w, cd, sd, B, S, H, D)
        assert_parity(got, st[name], f"op 2/3: {name} projection + RoPE", magnitude=st[name + "_proj"])
    got = dense(rows(st["h1"]), model.v_proj.weight, True, None, "none").view(B, S, H, D).transpose(1, 2)
    assert_parity(got, st["v_proj"], "op 4: v projection")
    got = M.SDPAModule()(dev(st["q"]), dev(st["k"]), dev(st["v_proj"]), None, None, True)
    assert_parity(got, st["attn"], "op 5: causal attention")
    got = dense(rows(st["attn_rows"]), model.o_proj.weight, True, rows(x), "none").view(B, S, Hd)
    assert_parity(got, st["x1"], "op 6: o projection + residual", magnitude=torch.maximum(x.float().abs(), st["o"].float().abs()))
    assert_parity(norm(rows(st["x1"]), model.post_norm.weight, eps).view(B, S, Hd), st["h2"], "op 7: RMSNorm")
    got = M.DenseSwiGLUModule()(rows(st["h2"]), model.gate_proj.weight, model.up_proj.weight).view(B, S, -1)
    assert_parity(got, st["ffn_h"], "op 8: gate/up dual GEMM + SwiGLU",
                  magnitude=torch.maximum(st["up"].float().abs(), (F_silu(st["gate"].float()) * st["up"].float()).abs()))
    got = dense(rows(st["ffn_h"]), model.down_proj.weight, True, rows(st["x1"]), "none").view(B, S, Hd)
    assert_parity(got, st["out"], "op 9: down projection + residual",
                  magnitude=torch.maximum(st["x1"].float().abs(), st["down"].float().abs()))

    got = FusedLlamaDecoderLayer(model)(dev(x), cd, sd)
    torch.cuda.synchronize()
    assert lib.tc_status() == 0
    _end_to_end_gate(got, st["out"], exact, "llama layer 1x2048x4096 bf16")


def F_silu(t):
    return torch.nn.functional.silu(t)


def _end_to_end_gate(got, want, exact, what):
    max_abs, mean_rel = error_stats(got, want)
    ours, theirs = (got.float().cpu() - exact).abs(), (want.float() - exact).abs()
    print(f"{what} vs the CPU oracle (eager bf16): max_abs={max_abs:.4g} mean_rel={mean_rel:.4g}; error vs fp32 math, "
          f"max / mean: this target {ours.max():.4g} / {ours.mean():.4g}, eager bf16 {theirs.max():.4g} / {theirs.mean():.4g}")
    assert ours.mean().item() <= 1.05 * theirs.mean().item(), "mean error vs fp32 math must not exceed eager bf16's"
    assert ours.max().item() <= 1.25 * theirs.max().item() + 1e-2, "max error vs fp32 math must stay at eager bf16's level"
    # and the two bf16 results agree to within a few units in the last place of the output scale
    scale = want.float().pow(2).mean().sqrt().item()
    assert max_abs <= 1e-2 + 5e-2 * scale, f"max |got - want| {max_abs} against an output RMS of {scale}"


def test_recsys_graph(cuda_device):
    """Config 5 at reduced size (batch 2048, tables of 5000 rows), fp32 values / int64 indices."""
    from xpu_graph_b200.fused_graphs import FusedRecsysGraph
    from xpu_graph_b200.workloads import make_recsys

    model, (dense, idx, mask) = make_recsys(seed=4, batch=2048, table_rows=5000)
    with torch.no_grad():
        want = model(dense, idx, mask)
    got = FusedRecsysGraph(model.to(cuda_device))(dense.to(cuda_device), idx.to(cuda_device), mask.to(cuda_device))
    assert_parity(got, want, "recsys graph fp32")


def test_recsys_graph_full_size(cuda_device):
    """Config 5 at its full size (batch 16384, 26 tables of 1e5 rows): here all three MLP layers are large enough for the
    fp32 tensor-core path, so the graph ends in one dense-tower call; checked against the eager model on the CPU."""
    from xpu_graph_b200 import ops
    from xpu_graph_b200.fused_graphs import FusedRecsysGraph
    from xpu_graph_b200.workloads import make_recsys

    model, (dense, idx, mask) = make_recsys(seed=4)
    assert dense.shape[0] == 16384
    with torch.no_grad():
        want = model(dense, idx, mask)
    assert ops.dense_tower_eligible(16384, [64 + 26 * 64, 1024, 512, 256])
    got = FusedRecsysGraph(model.to(cuda_device))(dense.to(cuda_device), idx.to(cuda_device), mask.to(cuda_device))
    assert_parity(got, want, "recsys graph fp32, full size")


def test_cuda_graph_replay_encoder(cuda_device):
    """Capture the fused encoder block once, replay it on new inputs (the reference's GraphRunner contract)."""
    from xpu_graph_b200.fused_graphs import FusedEncoderBlock
    from xpu_graph_b200.graph_runner import CUDAGraphRunner
    from xpu_graph_b200.workloads import make_encoder

    model, x = make_encoder(seed=0)
    cpu_model, _ = make_encoder(seed=0)  # same seed: an identical copy that stays on the CPU
    fused = FusedEncoderBlock(model.to(cuda_device))
    runner = CUDAGraphRunner(fused)
    xd = x.to(cuda_device)
    runner.capture(xd, clone_args=True)
    g = torch.Generator().manual_seed(99)
    for _ in range(2):
        x2 = torch.randn(x.shape, generator=g)
        with torch.no_grad():
            want = cpu_model(x2)
        got = runner(x2.to(cuda_device)).clone()
        assert_parity(got, want, "graph replay")


def test_cuda_graph_replay_llama_small(cuda_device):
    from xpu_graph_b200 import lib
    from xpu_graph_b200.fused_graphs import FusedLlamaDecoderLayer
    from xpu_graph_b200.graph_runner import CUDAGraphRunner
    from xpu_graph_b200.workloads import make_llama_layer

    model, (x, cos, sin) = make_llama_layer(seed=3, batch=1, seq=256, hidden=512, heads=4, ffn=1376)
    with torch.no_grad():
        want = model(x, cos, sin)
    fused = FusedLlamaDecoderLayer(model.to(cuda_device))
    runner = CUDAGraphRunner(fused)
    args = (x.to(cuda_device), cos.to(cuda_device), sin.to(cuda_device))
    runner.capture(*args, clone_args=True)
    got = runner(*args).clone()
    torch.cuda.synchronize()
    assert lib.tc_status() == 0
    assert_parity(got, want, "llama graph replay")


@pytest.mark.parametrize("batch,seq,hidden,splits_k", [(1, 16, 4096, True), (1, 128, 4096, True), (1, 333, 4096, True), (3, 37, 1024, False),
                                                       (2, 500, 512, False)])
def test_llama_layer_equals_its_op_sequence(cuda_device, batch, seq, hidden, splits_k):
    """The decoder layer's operator gives the bits of the replacement modules called one after the other, as a graph rewritten
    op by op calls them - at row counts where q and k share a launch, and where the dense kernels split K for the v projection."""
    import ctypes

    from tests.helpers import LaunchCounter
    from xpu_graph_b200 import lib
    from xpu_graph_b200 import modules as M
    from xpu_graph_b200.fused_graphs import FusedLlamaDecoderLayer
    from xpu_graph_b200.workloads import make_llama_layer

    heads = hidden // 128
    model, (x, cos, sin) = make_llama_layer(seed=3, batch=batch, seq=seq, hidden=hidden, heads=heads, ffn=1376)
    model = model.to(torch.bfloat16).to(cuda_device)
    x, cos, sin = x.to(cuda_device), cos.to(cuda_device), sin.to(cuda_device)
    rows, L = batch * seq, lib.load()
    S, tn = ctypes.c_int(0), ctypes.c_int(0)
    clusters = L.xg_gemm_cluster_plan(rows, hidden, hidden, lib.XG_BF16, ctypes.byref(S), ctypes.byref(tn)) and S.value > 1
    assert bool(clusters or L.xg_gemm_workspace_bytes(rows, hidden, hidden, lib.XG_BF16)) == splits_k
    with LaunchCounter() as calls:
        got = FusedLlamaDecoderLayer(model)(x, cos, sin)
    assert "xg_gemm_rope_group" in calls.names
    norm, dense, rope = M.RMSNormModule(), M.DenseLayerModule(False), M.DenseRopeModule()
    with torch.no_grad():
        x2 = x.reshape(rows, hidden)
        h = norm(x2, model.input_norm.weight, model.input_norm.eps)
        q, k = (rope(h, p.weight, cos, sin, batch, seq, heads, 128) for p in (model.q_proj, model.k_proj))
        v = dense(h, model.v_proj.weight, True, None, "none").view(batch, seq, heads, 128).transpose(1, 2)
        a = M.SDPAModule()(q, k, v, None, None, True).transpose(1, 2).reshape(rows, hidden)
        x2 = dense(a, model.o_proj.weight, True, x2, "none")
        h = norm(x2, model.post_norm.weight, model.post_norm.eps)
        want = dense(M.DenseSwiGLUModule()(h, model.gate_proj.weight, model.up_proj.weight), model.down_proj.weight, True, x2, "none")
    torch.cuda.synchronize()
    assert lib.tc_status() == 0
    assert torch.equal(got.view(rows, hidden), want)


def test_graph_operators_refuse_projections_of_another_width(cuda_device):
    """A q / k / v projection that is wider or narrower than its heads is an error (its columns used to be reinterpreted), and so
    is a number of heads that does not divide the width."""
    from xpu_graph_b200 import ops

    bf = dict(dtype=torch.bfloat16, device=cuda_device)
    x, cos, sin = torch.zeros(1, 16, 512, **bf), torch.zeros(16, 128, **bf), torch.zeros(16, 128, **bf)
    t = lambda *s: torch.zeros(*s, **bf)  # noqa: E731
    for i, width in ((1, 1024), (2, 256), (3, 1024), (3, 256)):
        w = [t(512), t(512, 512), t(512, 512), t(512, 512), t(512, 512), t(512), t(1376, 512), t(1376, 512), t(512, 1376)]
        w[i] = t(width, 512)
        with pytest.raises((RuntimeError, ValueError)):
            ops.decoder_layer(x, cos, sin, w, 1e-5, 1e-5, 4, True, True)
    for qkv, heads in ((2048, 4), (1024, 4), (1536, 0), (1536, 5)):
        p = [t(512), t(512), t(qkv, 512), t(qkv), t(512, 512), t(512), t(512), t(512), t(1024, 512), t(1024), t(512, 1024), t(512)]
        with pytest.raises((RuntimeError, ValueError)):
            ops.encoder_block(x, p, 1e-5, 1e-5, heads)
    w = [t(512), t(512, 512), t(512, 512), t(512, 512), t(512, 512), t(512), t(1376, 512), t(1376, 512), t(512, 1376)]
    with pytest.raises((RuntimeError, ValueError)):
        ops.decoder_layer(x, cos, sin, w, 1e-5, 1e-5, 0, True, True)


def test_graph_operators_are_inference_only(cuda_device):
    """A backward through a graph operator is an error, as through every other operator of the library; the fused classes run
    without gradients."""
    from xpu_graph_b200 import ops
    from xpu_graph_b200.fused_graphs import FusedEncoderBlock
    from xpu_graph_b200.workloads import make_encoder

    model, x = make_encoder(seed=0)
    model, x = model.to(cuda_device), x.to(cuda_device)
    params = []
    for m in (model.ln1, model.qkv, model.proj, model.ln2, model.fc1, model.fc2):
        params += (m.weight, m.bias)
    args = (params, model.ln1.eps, model.ln2.eps, model.heads)
    y = ops.encoder_block(x, *args)  # the parameters require gradients
    assert y.requires_grad
    with pytest.raises(RuntimeError, match="encoder_block"):
        y.sum().backward()
    fused = FusedEncoderBlock(model)(x.requires_grad_())
    assert not fused.requires_grad and torch.equal(fused, y.detach())
    with torch.no_grad():
        assert not ops.encoder_block(x, *args).requires_grad
    import torch.autograd.forward_ad as fwd

    with fwd.dual_level(), pytest.raises(NotImplementedError, match="forward-mode"):
        ops.encoder_block(fwd.make_dual(x.detach(), torch.ones_like(x)), *args)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_traced_layouts_are_the_real_ones(cuda_device, dtype):
    """What the compiler is told about attention's and RoPE's results (shape, strides, dtype) is what the operators return, for the
    layouts that projections leave: packed q, k, v, separate buffers, contiguous heads, one head, one position, broadcast heads."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    X = torch.ops.xg_sm100
    rnd = lambda *s: torch.randn(*s, device=cuda_device).to(dtype)  # noqa: E731
    packed = rnd(2, 40, 3, 4, 64)
    layouts = {
        "packed": [packed[:, :, i].transpose(1, 2) for i in range(3)],
        "packed by head": [rnd(2, 40, 4, 3, 64)[:, :, :, i].transpose(1, 2) for i in range(3)],
        "projections": [rnd(2, 40, 4, 64).transpose(1, 2) for _ in range(3)],
        "contiguous": [rnd(2, 4, 40, 64) for _ in range(3)],
        "one head": [rnd(2, 40, 1, 64).transpose(1, 2) for _ in range(3)],
        "one position": [rnd(2, 1, 4, 64).transpose(1, 2) for _ in range(3)],
        "broadcast heads": [rnd(2, 1, 40, 64).expand(2, 4, 40, 64) for _ in range(3)],
        "strided elements": [rnd(2, 4, 64, 40).transpose(2, 3) for _ in range(3)],
    }
    for name, (q, k, v) in layouts.items():
        cos, sin = rnd(q.shape[2], 64), rnd(q.shape[2], 64)
        mask = torch.rand(2, 1, 1, k.shape[2], device=cuda_device) < 0.9
        calls = [lambda q, k, v, c, s, m: X.sdpa(q, k, v, None, 0.125, False), lambda q, k, v, c, s, m: X.sdpa(q, k, v, m, 0.125, True),
                 lambda q, k, v, c, s, m: X.rope(q, c, s)]
        for i, call in enumerate(calls):
            real = call(q, k, v, cos, sin, mask)
            with FakeTensorMode() as mode:
                fake = call(*(mode.from_tensor(t) for t in (q, k, v, cos, sin, mask)))
            assert (fake.shape, fake.stride(), fake.dtype, fake.device) == (real.shape, real.stride(), real.dtype, real.device), (name, i)


@pytest.mark.parametrize("dynamic", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_modules_compile_to_the_same_bits(cuda_device, dtype, dynamic):
    """The replacement modules under torch.compile (traced through the operators' fake implementations, run by their CUDA
    kernels) give the bits of the same modules called one by one, also when the batch is a symbol."""
    from xpu_graph_b200 import modules as M

    H, D, S = 4, 64, 37
    C = H * D
    dense, norm, sdpa = M.DenseLayerModule(False), M.RMSNormModule(), M.SDPAModule()

    def block(x, g, w_qkv, b_qkv, w_o):
        B = x.shape[0]
        h = norm(x.reshape(B * S, C), g, 1e-5)
        qkv = dense(h, w_qkv, True, b_qkv, "none").view(B, S, 3, H, D)
        q, k, v = (qkv[:, :, i].transpose(1, 2) for i in range(3))
        a = sdpa(q, k, v, None, 0.125, True).transpose(1, 2).reshape(B * S, C)
        return dense(a, w_o, True, None, "gelu").view(B, S, C)

    rnd = lambda *s: torch.randn(*s, device=cuda_device).to(dtype) * 0.05  # noqa: E731
    weights = (rnd(C), rnd(3 * C, C), rnd(3 * C), rnd(C, C))
    torch._dynamo.reset()
    compiled = torch.compile(block, backend="aot_eager", fullgraph=True, dynamic=dynamic)
    with torch.no_grad():
        for B in (2, 5, 3) if dynamic else (2,):
            x = rnd(B, S, C)
            assert torch.equal(compiled(x, *weights), block(x, *weights))


@pytest.mark.parametrize("rows,mlp", [(500, (1024, 512, 256)), (4096, (1024, 512, 256)), (40, (64, 32))])
def test_recommender_equals_its_op_sequence(cuda_device, rows, mlp):
    """The recommender's operator gives the bits of the replacement modules called one after the other: all layers on the tensor
    cores, some of them, none."""
    from xpu_graph_b200 import modules as M
    from xpu_graph_b200.fused_graphs import FusedRecsysGraph
    from xpu_graph_b200.workloads import RecsysGraph

    torch.manual_seed(5)
    graph = RecsysGraph(64, 16, 26, 64, 1000, mlp).to(cuda_device)
    dense, idx = torch.randn(rows, 64, device=cuda_device), torch.randint(0, 1000, (rows, 26), device=cuda_device)
    mask = torch.rand(rows, 1, device=cuda_device) < 0.3
    fused = FusedRecsysGraph(graph)
    with torch.no_grad():
        h = M.CatLastDimModule()([M.FuseSliceCatSameInputModule()(dense, list(zip(fused.starts, fused.ends))),
                                  M.GatherStackModule()(list(graph.tables), idx, mask, True)])
        for layer in graph.layers:
            h = M.DenseLayerModule(False)(h, layer.weight, True, layer.bias, "relu")
    assert torch.equal(fused(dense, idx, mask), h)


@pytest.mark.parametrize("batch,seq,dtype", [(2, 128, torch.float32), (3, 197, torch.float16), (24, 197, torch.bfloat16)])
def test_encoder_block_equals_its_op_sequence(cuda_device, batch, seq, dtype):
    """The encoder block's operator gives the bits of the replacement modules called one after the other."""
    from xpu_graph_b200 import modules as M
    from xpu_graph_b200.fused_graphs import FusedEncoderBlock
    from xpu_graph_b200.workloads import make_encoder

    b, _ = make_encoder(seed=0)
    b = b.to(cuda_device).to(dtype)
    C, H, T = b.ln1.weight.shape[0], b.heads, batch * seq
    x = torch.randn(batch, seq, C, device=cuda_device).to(dtype)
    norm, dense, res = M.LayerNormModule(), M.DenseLayerModule(False), M.DenseResidualModule()
    with torch.no_grad():
        x0 = x.reshape(T, C)
        qkv = dense(norm(x0, b.ln1.weight, b.ln1.bias, b.ln1.eps), b.qkv.weight, True, b.qkv.bias, "none").view(batch, seq, 3, H, C // H)
        a = M.SDPAModule()(*(qkv[:, :, i].transpose(1, 2) for i in range(3)), None, None, False).transpose(1, 2).reshape(T, C)
        x1 = res(a, b.proj.weight, True, b.proj.bias, x0, "none")
        h = dense(norm(x1, b.ln2.weight, b.ln2.bias, b.ln2.eps), b.fc1.weight, True, b.fc1.bias, "gelu")
        want = res(h, b.fc2.weight, True, b.fc2.bias, x1, "none")
    assert torch.equal(FusedEncoderBlock(b)(x).view(T, C), want)
