"""The queue that collects a backward pass's second-stage reductions into one launch: a weight whose gradient has one
share in the joint product of Q, K and V and one in another product, before or after it, and more reductions than one
launch takes; against the f64 oracle."""
import numpy as np
import pytest

from neuralrs_b200 import _lib
from neuralrs_b200.cuda import Context, Node, backward_graph, graph, nn
from neuralrs_b200.cuda import runtime as gpu
from oracle import autograd as og
from .conftest import rel_l2

pytestmark = pytest.mark.gpu


def on_gpu(a):
    n = Node.new(a, list(np.shape(a)))
    gpu.to_cuda(n)
    return n


@pytest.mark.parametrize("attention_first", [True, False])
@pytest.mark.parametrize("shared", [0, 1, 2], ids=["w_q", "w_k", "w_v"])
def test_weight_of_attention_and_of_another_product(gpu_ctx, oracle64, shared, attention_first):
    B, S, D, H = 3, 100, 64, 2
    rng = np.random.default_rng(shared)
    w = [(rng.standard_normal((D, D)) / np.sqrt(D)).astype(np.float32) for _ in range(4)]
    x = rng.standard_normal((B, S, D)).astype(np.float32)
    x2, seed = (rng.standard_normal((B * S, D)).astype(np.float32) for _ in range(2))
    g = og.Graph(oracle64)
    cx, cx2, cw = og.Node(x), og.Node(x2), [og.Node(a) for a in w]
    ca, cz = g.reshape(g.mha_forward_batch(cx, *cw, H), (B * S, D)), g.matmul(cx2, cw[shared])
    cout = g.add(cz, ca) if attention_first else g.add(ca, cz)   # the later operand's backward pass runs first
    cout.grad = seed.copy()
    og.backward_graph(cout)
    gx, gx2, gw = on_gpu(x), on_gpu(x2), [on_gpu(a) for a in w]
    gpu.flatten_params(gw)
    mha = nn.MultiHeadAttention(*gw, D, H, False)
    gpu.zero_grad(gw)
    for total in (1, 2):   # the second pass adds to the gradients of the first
        ga, gz = graph.reshape(mha.forward_batch(gx), (B * S, D)), graph.matmul(gx2, gw[shared])
        out = graph.add(gz, ga) if attention_first else graph.add(ga, gz)
        gpu.set_grad(out, seed)
        backward_graph(out)
        for i, (gn, cn) in enumerate(zip([gx, gx2] + gw, [cx, cx2] + cw)):
            assert rel_l2(gpu.read_grad(gn), total * cn.grad) <= 1e-4, i


def test_more_reductions_than_one_launch_takes(gpu_ctx, oracle64):
    rows, d, layers = 4500, 32, 20   # a product's gradient over 4500 rows is split; 20 of them and 20 LayerNorm pairs
    rng = np.random.default_rng(9)
    w = [(np.eye(d) + 0.1 * rng.standard_normal((d, d))).astype(np.float32) for _ in range(layers)]
    gamma, beta = ([(k + 0.1 * rng.standard_normal(d)).astype(np.float32) for _ in range(layers)] for k in (1, 0))
    x, seed = (rng.standard_normal((rows, d)).astype(np.float32) for _ in range(2))
    g = og.Graph(oracle64)
    cx, cp = og.Node(x), [og.Node(a) for a in w + gamma + beta]
    gx, gp = on_gpu(x), [on_gpu(a) for a in w + gamma + beta]
    ch, gh = cx, gx
    for i in range(layers):
        ch = g.layernorm(g.matmul(ch, cp[i]), cp[layers + i], cp[2 * layers + i], 1e-5)
        gh = nn.layernorm(graph.matmul(gh, gp[i]), gp[layers + i], gp[2 * layers + i], 1e-5)
    ch.grad = seed.copy()
    og.backward_graph(ch)
    gpu.set_grad(gh, seed)
    before = gpu_ctx.launch_count()
    backward_graph(gh)
    assert gpu_ctx.launch_count() - before > 2 * layers
    for i, (gn, cn) in enumerate(zip([gx] + gp, [cx] + cp)):
        assert rel_l2(gpu.read_grad(gn), cn.grad) <= 2e-4, i   # twenty 3xTF32 products deep, some 1e-5 each


def test_idle_memory_goes_back_before_an_allocation_fails():
    ctx = Context(0)
    try:
        assert _lib.lib().nrs_selftest_memory_pressure(ctx.h) == 0
    finally:
        ctx.close()
