"""Operands that do not fit each other are refused on the host, before anything is launched: the kernels read by address and
know one set of extents, so a tensor of another dtype, device or size would be read past its end."""
import pytest
import torch

from tests.helpers import LaunchCounter

pytestmark = pytest.mark.gpu


def _t(*shape, dt=torch.bfloat16, dev="cuda"):
    return torch.zeros(*shape, dtype=dt, device=dev)


F32 = torch.float32
BAD = {
    "mul_sum_cat: a second operand is missing": lambda X: X.mul_sum_cat([_t(4, 3, 8)] * 2, [_t(4, 3, 8)]),
    "slice_sum_cat: an end is missing": lambda X: X.slice_sum_cat(_t(4, 9, 8), [0, 3], [3]),
    "dense_tower: no layers": lambda X: X.dense_tower(_t(4, 8), [], [], [], ""),
    "norm: weight too short": lambda X: X.rms_norm(_t(4, 64), _t(32), 1e-5),
    "norm: bias too short": lambda X: X.layer_norm(_t(4, 64), _t(64), _t(1), 1e-5),
    "norm: weight on the host": lambda X: X.rms_norm(_t(4, 64), _t(64, dev="cpu"), 1e-5),
    "dense: weight of another dtype": lambda X: X.dense(_t(4, 64, dt=F32), _t(32, 64), True, None, None, "none"),
    "dense: one bias element": lambda X: X.dense(_t(4, 64), _t(32, 64), True, _t(1), None, "none"),
    "dense: residual of one row": lambda X: X.dense(_t(4, 64), _t(32, 64), True, None, _t(1, 32), "none"),
    "dense: residual too narrow": lambda X: X.dense(_t(4, 64), _t(32, 64), True, None, _t(4, 16), "none"),
    "dense: bias on the host": lambda X: X.dense(_t(4, 64), _t(32, 64), True, _t(32, dev="cpu"), None, "none"),
    "batch_dense: fewer weights": lambda X: X.batch_dense(_t(4, 8, 64), _t(2, 32, 64), True, None, None, "none"),
    "batch_dense: inner dimensions": lambda X: X.batch_dense(_t(4, 8, 64), _t(4, 32, 32), True, None, None, "none"),
    "batch_dense: weight of another dtype": lambda X: X.batch_dense(_t(4, 8, 64, dt=F32), _t(4, 32, 64), True, None, None, "none"),
    "dense_swiglu: up narrower": lambda X: X.dense_swiglu(_t(4, 64), _t(32, 64), _t(16, 64)),
    "dense_swiglu: inner dimensions": lambda X: X.dense_swiglu(_t(4, 64), _t(32, 32), _t(32, 32)),
    "dense_swiglu: dtypes": lambda X: X.dense_swiglu(_t(4, 64), _t(32, 64), _t(32, 64, dt=torch.float16)),
    "dense_rope: inner dimensions": lambda X: X.dense_rope(_t(4, 64), _t(64, 32), _t(4, 64), _t(4, 64), 4, 64),
    "dense_rope: tables on the host": lambda X: X.dense_rope(_t(4, 64), _t(64, 64), _t(4, 64, dev="cpu"), _t(4, 64), 4, 64),
    "sdpa: fewer key heads": lambda X: X.sdpa(_t(2, 4, 8, 64), _t(2, 2, 8, 64), _t(2, 2, 8, 64), None, 1.0, False),
    "sdpa: v shorter than k": lambda X: X.sdpa(_t(2, 4, 8, 64), _t(2, 4, 8, 64), _t(2, 4, 4, 64), None, 1.0, False),
    "sdpa: head dims": lambda X: X.sdpa(_t(2, 4, 8, 64), _t(2, 4, 8, 32), _t(2, 4, 8, 32), None, 1.0, False),
    "sdpa: dtypes": lambda X: X.sdpa(_t(2, 4, 8, 64, dt=F32), _t(2, 4, 8, 64), _t(2, 4, 8, 64), None, 1.0, False),
    "sdpa: mask on the host": lambda X: X.sdpa(_t(2, 4, 8, 64), _t(2, 4, 8, 64), _t(2, 4, 8, 64), _t(8, 8, dev="cpu"), 1.0, False),
    "rope: tables on the host": lambda X: X.rope(_t(1, 2, 4, 64), _t(4, 64, dev="cpu"), _t(4, 64)),
    "mlp_small: weight on the host": lambda X: X.mlp_small(_t(4, 32), [_t(16, 32, dev="cpu")], [None], "relu", 0),
    "dense_tower: weight of another dtype": lambda X: X.dense_tower(_t(8192, 512, dt=F32), [_t(512, 512)], [True], [None], "relu"),
    "dense_tower: bias too short": lambda X: X.dense_tower(_t(8192, 512, dt=F32), [_t(512, 512, dt=F32)], [True], [_t(8, dt=F32)], "relu"),
    "slice_cat: mask on the host": lambda X: X.slice_cat(_t(4, 64), [0], [8], _t(4, dt=torch.bool, dev="cpu"), True),
    "cat_lastdim: one input on the host": lambda X: X.cat_lastdim([_t(4, 8), _t(4, 8, dev="cpu")], None, True),
    "gather_stack: table on the host": lambda X: X.gather_stack([_t(9, 8, dev="cpu")], _t(4, 1, dt=torch.int64), None, True),
    "sum_cat: one input on the host": lambda X: X.sum_cat([_t(4, 3, 8), _t(4, 3, 8, dev="cpu")]),
    "sum3d: one input on the host": lambda X: X.sum3d([_t(4, 3, 8), _t(4, 3, 8, dev="cpu")], 1),
    "combo_dense: bias on the host": lambda X: X.combo_dense([_t(4, 64)] * 2, [_t(32, 64)] * 2, True, [_t(32, dev="cpu")] * 2, "none"),
}


@pytest.mark.parametrize("what", list(BAD))
def test_misfit_operands_are_refused_before_a_launch(cuda_device, what):
    from xpu_graph_b200 import ops  # noqa: F401

    with LaunchCounter() as calls:
        with pytest.raises((ValueError, RuntimeError)):
            BAD[what](torch.ops.xg_sm100)
    assert calls.names == []
