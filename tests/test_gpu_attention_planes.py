"""Multi-head attention over operand planes: sequences inside, at and across the 128-row tiles and the 1024-column row
kernels, head sizes with padded column and K tiles, causal and not, separate weights and weights of one flat block,
gradients overwritten and added to; against the f64 oracle."""
import numpy as np
import pytest

from neuralrs_b200 import _lib
from neuralrs_b200.cuda import Node, backward_graph, nn
from neuralrs_b200.cuda import runtime as gpu
from oracle import autograd as og
from .conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = {_lib.MATH_3XTF32: 1e-4, _lib.MATH_TF32: 1e-2}
SHAPES = [(3, 7, 32, 4), (2, 128, 64, 2), (1, 129, 64, 4), (2, 250, 96, 4), (1, 500, 128, 2), (1, 1030, 32, 2)]   # batch, seq, d, heads


def on_gpu(a):
    n = Node.new(a, list(np.shape(a)))
    gpu.to_cuda(n)
    return n


@pytest.mark.parametrize("mode", list(TOL), ids=["3xtf32", "tf32"])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_mha_over_planes(gpu_ctx, oracle64, shape, causal, mode):
    B, S, D, H = shape
    rng = np.random.default_rng(S + D)
    w = [(rng.standard_normal((D, D)) / np.sqrt(D)).astype(np.float32) for _ in range(4)]
    x, seed = (rng.standard_normal((B, S, D)).astype(np.float32) for _ in range(2))
    g = og.Graph(oracle64)
    cx, cw = og.Node(x), [og.Node(a) for a in w]
    cout = g.mha_forward_batch(cx, *cw, H, causal)
    cout.grad = seed.copy()
    og.backward_graph(cout)
    gpu_ctx.set_math_mode(mode)
    try:
        gx, gw = on_gpu(x), [on_gpu(a) for a in w]
        mha = nn.MultiHeadAttention(*gw, D, H, causal)
        for total in (1, 2):   # the second pass adds to the gradients of the first
            out = mha.forward_batch(gx)
            assert rel_l2(gpu.to_host(out), cout.data) <= TOL[mode]
            gpu.set_grad(out, seed)
            backward_graph(out)
            for gn, cn in zip([gx] + gw, [cx] + cw):
                assert rel_l2(gpu.read_grad(gn), total * cn.grad) <= TOL[mode]
    finally:
        gpu_ctx.set_math_mode(_lib.MATH_3XTF32)
