"""Multi-head attention over operand planes: sequences inside, at and across the 128-row tiles and the 1024-column row
kernels, head sizes with padded column and K tiles, causal and not, separate weights and weights of one flat block,
gradients overwritten and added to; against the f64 oracle."""
import ctypes

import numpy as np
import pytest

from neuralrs_b200 import _lib
from neuralrs_b200.cuda import Context, Node, backward_graph, nn
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


def test_backward_memory_does_not_grow_with_the_square(gpu_ctx):
    """The weight gradients of Q, K and V wait for the end of the pass where the three lie side by side; what a layer holds for
    them until then is the planes of their operands, not its scores."""
    S, D, H = 2048, 128, 4
    libcuda = ctypes.CDLL("libcuda.so.1")

    def used(ctx):
        ctx.sync()
        free, total = ctypes.c_size_t(), ctypes.c_size_t()
        assert libcuda.cuMemGetInfo_v2(ctypes.byref(free), ctypes.byref(total)) == 0
        return total.value - free.value

    def grown(layers):
        ctx = Context(0)
        try:
            rng = np.random.default_rng(layers)
            new = lambda *shape: Node.new((rng.standard_normal(shape) / np.sqrt(D)).astype(np.float32), list(shape), ctx=ctx)  # noqa: E731
            w = [new(D, D) for _ in range(4 * layers)]
            h = x = new(1, S, D)
            for n in w + [x]:
                gpu.to_cuda(n)
            gpu.flatten_params(w)
            for i in range(layers):
                h = nn.MultiHeadAttention(*w[4 * i:4 * i + 4], D, H, True).forward_batch(h)
            gpu.set_grad(h, np.ones((1, S, D), np.float32))
            before = used(ctx)
            backward_graph(h)
            after = used(ctx)
            assert all(np.isfinite(gpu.read_grad(n)).all() for n in w[:4])
            return after - before
        finally:
            ctx.close()

    per_layer = (grown(9) - grown(3)) / 6
    assert per_layer <= 20 * S * D * 4, per_layer   # (scores and the planes of dS: 8 * H * S * S bytes, 128 times S * D * 4)


def test_weights_of_one_product_are_measured_together(gpu_ctx):
    """f16 pairs want exponents: of the input, of Q, K and V in one launch, of the output projection; nothing else is launched
    more than in TF32."""
    B, S, D, H = 2, 128, 256, 8
    rng = np.random.default_rng(1)
    w, x = [on_gpu((rng.standard_normal((D, D)) / 16).astype(np.float32)) for _ in range(4)], rng.standard_normal((B, S, D)).astype(np.float32)
    mha, launches = nn.MultiHeadAttention(*w, D, H, True), {}
    try:
        for mode in TOL:
            gpu_ctx.set_math_mode(mode)
            gx = on_gpu(x)
            before = gpu_ctx.launch_count()
            mha.forward_batch(gx)
            launches[mode] = gpu_ctx.launch_count() - before
    finally:
        gpu_ctx.set_math_mode(_lib.MATH_3XTF32)
    assert launches[_lib.MATH_3XTF32] <= launches[_lib.MATH_TF32] + 3, launches
