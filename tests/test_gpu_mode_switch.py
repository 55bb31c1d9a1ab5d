"""The math mode changed between the forward and the backward pass of a transformer block: tensors that exist as operand
planes alone are made whole, planes of the other mode are not read; against the f64 oracle."""
import numpy as np
import pytest

from neuralrs_b200 import _lib
from neuralrs_b200.cuda import backward_graph
from neuralrs_b200.cuda import runtime as gpu
from oracle import autograd as og
from .conftest import rel_l2
from .test_gpu_transformer import gpu_block, make_block_params, on_gpu

pytestmark = pytest.mark.gpu
MODES = {"fp32": _lib.MATH_FP32, "tf32": _lib.MATH_TF32, "3xtf32": _lib.MATH_3XTF32}
# 11-bit operands in either pass (a GELU network of six products); sums in f32 or 3xTF32 otherwise
TOL = {"fp32": 2e-5, "3xtf32": 2e-5, "tf32": 5e-3}


@pytest.mark.parametrize("forward,backward", [(a, b) for a in MODES for b in MODES if a != b])
def test_block_with_another_mode_backward(gpu_ctx, oracle64, forward, backward):
    B, S, D, H, F = 2, 64, 64, 2, 128
    rng = np.random.default_rng(11)
    p = make_block_params(rng, D, F)
    x, seed = (rng.standard_normal((B, S, D)).astype(np.float32) for _ in range(2))
    g = og.Graph(oracle64)
    cx, cp = og.Node(x), {k: og.Node(v) for k, v in p.items()}
    cout = g.transformer_block(cx, cp, H, 1e-5, "gelu", causal=True)
    cout.grad = seed.copy()
    og.backward_graph(cout)
    gx = on_gpu(x)
    block, gp = gpu_block(p, H, "gelu", True)
    try:
        gpu_ctx.set_math_mode(MODES[forward])
        out = block.forward(gx)
        gpu.set_grad(out, seed)
        gpu_ctx.set_math_mode(MODES[backward])
        backward_graph(out)
        tol = max(TOL[forward], TOL[backward])
        assert rel_l2(gpu.to_host(out), cout.data) <= TOL[forward]
        for k, gn, cn in [("x", gx, cx)] + [(k, gp[k], cp[k]) for k in gp]:
            assert rel_l2(gpu.read_grad(gn), cn.grad) <= tol, k
    finally:
        gpu_ctx.set_math_mode(_lib.MATH_3XTF32)
