"""3xTF32 products as f16 pairs (one power-of-two exponent a tensor) and the kernels around them: magnitudes and ranges,
zeros, infinities, many live ranges; convolutions by slabs at the edges of their tiles; weight gradients in column blocks, by
slabs and collected to the end of a pass; the small kernels' second stages.  Against f64."""
import ctypes

import numpy as np
import pytest

from neuralrs_b200 import _lib, cuda, workloads
from neuralrs_b200.cuda import Node, backward_graph, graph, nn
from neuralrs_b200.cuda import runtime as gpu
from oracle import autograd as og
from oracle import models
from .conftest import rel_l2
from .gpu_util import Dev, call
from .test_gpu_transformer import gpu_block, make_block_params, on_gpu

pytestmark = pytest.mark.gpu


def gemm(ctx, ta, tb, a, b, c=None):
    m, k = (a.shape[1], a.shape[0]) if ta else a.shape
    n = b.shape[0] if tb else b.shape[1]
    out = Dev(ctx, c) if c is not None else Dev(ctx, shape=(m, n))
    call(ctx, "nrs_gemm", ta, tb, m, n, k, Dev(ctx, a), Dev(ctx, b), out, None, 0, _lib.C.c_float(0.0 if c is None else 1.0))
    return out.get()


def entry_bound(a, b, k, chain=4096):
    """What an entry of a @ b may be off by.  A pair holds a value to 2^-22 of itself, or to 2^-51 of its tensor's largest;
    the product of the two low halves is left out (2^-22); the tensor core adds 16 values at a time and cuts what lies
    2^-23 below the largest of a step, in two accumulators; sums of chunks and the end round once each."""
    a, b = np.abs(a.astype(np.float64)), np.abs(b.astype(np.float64))
    rel = 3 * 2.0**-22 + (2 * min(k, chain) / 16 + k // chain + 4) * 2.0**-23
    floor = 2.0**-50 * (a.max() * b.sum(0)[None, :] + a.sum(1)[:, None] * b.max())
    return rel * (a @ b) + floor


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("ea,eb", [(0, 0), (-100, 0), (60, 60), (-60, -55), (-90, 100)])
def test_products_at_any_magnitude(gpu_ctx, ta, tb, ea, eb):
    m, n, k = 136, 72, 200
    rng = np.random.default_rng(abs(ea) + 3 * abs(eb))
    a = (rng.standard_normal((m, k)) * 2.0**ea).astype(np.float32)
    b = (rng.standard_normal((k, n)) * 2.0**eb).astype(np.float32)
    got = gemm(gpu_ctx, ta, tb, a.T if ta else a, b.T if tb else b)
    err = np.abs(got - a.astype(np.float64) @ b.astype(np.float64))
    assert (err <= entry_bound(a, b, k)).all(), float((err / entry_bound(a, b, k)).max())


@pytest.mark.parametrize("spread", [12, 24, 28])
def test_values_far_below_the_largest(gpu_ctx, spread):
    """Values down to 2^-spread of the tensor's largest keep their 22 bits."""
    m, n, k = 128, 64, 160
    rng = np.random.default_rng(spread)
    a = (rng.choice([-1.0, 1.0], (m, k)) * rng.uniform(1, 2, (m, k)) * 2.0 ** -rng.integers(0, spread, m)[:, None]).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    err = np.abs(gemm(gpu_ctx, 0, 0, a, b) - a.astype(np.float64) @ b.astype(np.float64))
    assert (err <= entry_bound(a, b, k)).all(), float((err / entry_bound(a, b, k)).max())


def test_zeros_infinities_and_nans(gpu_ctx):
    m, n, k = 128, 64, 96
    rng = np.random.default_rng(1)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    assert not gemm(gpu_ctx, 0, 0, np.zeros_like(a), b).any()
    assert not gemm(gpu_ctx, 0, 0, a, np.zeros_like(b)).any()
    bad = a.copy()
    bad[3, 5], bad[70, 0] = np.inf, np.nan
    got = gemm(gpu_ctx, 0, 0, bad, b)
    rows = np.setdiff1d(np.arange(m), [3, 70])
    assert not np.isfinite(got[[3, 70]]).any()
    err = np.abs(got - a.astype(np.float64) @ b.astype(np.float64))[rows]
    assert (err <= entry_bound(a, b, k)[rows]).all()   # the others as if those values were not there


def test_more_ranges_than_a_page(gpu_ctx):
    """300 tensors with planes at a time, of different magnitudes, dropped and made again."""
    n, ci, h, w, co = 1, 32, 6, 6, 32
    rng = np.random.default_rng(2)
    wt = (rng.standard_normal((co, ci, 3, 3)) / 17).astype(np.float32)
    wd, bd, y = Dev(gpu_ctx, wt), Dev(gpu_ctx, np.zeros(co, np.float32)), Dev(gpu_ctx, shape=(n, co, h, w))
    x = rng.standard_normal((n, ci, h, w)).astype(np.float32)
    outs = []
    for scale in (1.0, 1e-6, 1e5):
        xs = [Dev(gpu_ctx, (x * np.float32(scale * (i + 1))).astype(np.float32)) for i in range(300)]
        for d in xs:
            call(gpu_ctx, "nrs_planes_cache", d, n, ci, h, w)
        for i in (0, 1, 255, 256, 299):
            call(gpu_ctx, "nrs_conv2d_fwd", xs[i], wd, bd, y, n, ci, h, w, co, 3, 3, 1, 1, 0)
            outs.append((scale * (i + 1), y.get()))
        for d in xs:
            call(gpu_ctx, "nrs_planes_drop", d)
    ref = outs[0][1].astype(np.float64)
    for s, out in outs:   # the same product up to a factor: two roundings of the input, the chain of 288 values twice
        assert rel_l2(out / s, ref) <= 2 * (2.0**-22 + (288 / 16 + 4) * 2.0**-23), s


def chain_tolerance(k):
    """Relative to the result (2-norm): operands to 2^-21 together, the cut of each step of 16 values relative to a partial
    sum, which is no larger than the result; in two accumulators."""
    return 2.0**-20 + (2 * k / 16 + 4) * 2.0**-23


SLABS = [(n, ci, h, w, co, k) for n, ci, h, co, k in [(5, 64, 9, 64, 3)] for w in (7, 8, 9, 14, 16, 17, 24, 28, 31, 32, 33, 57)] + [
    (3, 32, 12, 28, 128, 3),      # one 32-channel block
    (4, 96, 7, 16, 72, 3),        # blocks of 32 only; ragged columns
    (2, 128, 5, 32, 256, 3),      # two column tiles
    (33, 64, 4, 4, 64, 3),        # many images in a tile, an odd count of them
    (2, 200, 11, 9, 40, 5),       # 5x5, a last block of 8 channels
    (2, 64, 13, 12, 130, 5),      # a column tile of two
    (2, 200, 20, 17, 96, 5),      # few pixels and 5000 values a chain: chunks
    (1, 64, 3, 64, 64, 3),        # fewer rows than taps reach
]


@pytest.mark.parametrize("cfg", SLABS, ids=lambda c: "x".join(map(str, c)))
def test_convolutions_by_slabs(gpu_ctx, oracle64, cfg):
    n, ci, h, w, co, k = cfg
    rng = np.random.default_rng(sum(cfg))
    x = rng.standard_normal((n, ci, h, w)).astype(np.float32)
    wt = (rng.standard_normal((co, ci, k, k)) * np.sqrt(2.0 / (ci * k * k))).astype(np.float32)
    b = (rng.standard_normal(co) * 0.1).astype(np.float32)
    dy = rng.standard_normal((n, co, h, w)).astype(np.float32)
    yref, refs = oracle64.conv2d_fwd(x, wt, b, 1, k // 2), oracle64.conv2d_bwd(x, wt, dy, 1, k // 2)
    xd, wd, bd, dyd = (Dev(gpu_ctx, a) for a in (x, wt, b, dy))
    y, grads = Dev(gpu_ctx, shape=yref.shape), [Dev(gpu_ctx, shape=a.shape) for a in (x, wt, b)]
    args = (n, ci, h, w, co, k, k, 1, k // 2)
    call(gpu_ctx, "nrs_planes_cache", xd, n, ci, h, w)
    call(gpu_ctx, "nrs_planes_cache", dyd, n, co, h, w)
    call(gpu_ctx, "nrs_conv2d_fwd", xd, wd, bd, y, *args, 0)
    call(gpu_ctx, "nrs_conv2d_bwd", xd, wd, dyd, *grads, *args, 0)
    call(gpu_ctx, "nrs_planes_drop", xd)
    call(gpu_ctx, "nrs_planes_drop", dyd)
    for name, got, ref, chain in zip(("y", "dx", "dw", "db"), [y] + grads, (yref, *refs), (min(4096, ci * k * k), min(4096, co * k * k), n * h * w, 1)):
        assert rel_l2(got.get(), ref) <= chain_tolerance(chain), name


@pytest.mark.parametrize("m,n,k", [(64, 64, 32), (130, 72, 40), (256, 1000, 4096), (1000, 130, 515), (48, 520, 9000), (512, 512, 64)])
@pytest.mark.parametrize("add", [False, True])
def test_linear_weight_gradients(gpu_ctx, m, n, k, add):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((k, m)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    c = rng.standard_normal((m, n)).astype(np.float32) if add else None
    ref = a.T.astype(np.float64) @ b.astype(np.float64) + (c if add else 0.0)
    assert rel_l2(gemm(gpu_ctx, 1, 0, a, b, c), ref) <= chain_tolerance(min(k, 8192))


@pytest.mark.parametrize("passes", [1, 2])
def test_collected_weight_gradients(gpu_ctx, oracle64, passes):
    """More products than one launch takes, some with the same weight, and a second pass that adds."""
    rows, d, layers = 520, 64, 22
    rng = np.random.default_rng(passes)
    w = [(np.eye(d) + 0.1 * rng.standard_normal((d, d))).astype(np.float32) for _ in range(layers - 2)]
    order = list(range(layers - 2)) + [0, 5]
    x, seed = (rng.standard_normal((rows, d)).astype(np.float32) for _ in range(2))
    g = og.Graph(oracle64)
    cw = [og.Node(a) for a in w]
    ch = cx = og.Node(x)
    for i in order:
        ch = g.gelu(g.matmul(ch, cw[i]))
    ch.grad = seed.copy()
    og.backward_graph(ch)
    gx, gw = on_gpu(x), [on_gpu(a) for a in w]
    gpu.zero_grad(gw)
    for _ in range(passes):
        gh = gx
        for i in order:
            gh = graph.gelu(graph.matmul(gh, gw[i]))
        gpu.set_grad(gh, seed)
        backward_graph(gh)
    for i, (gn, cn) in enumerate(zip([gx] + gw, [cx] + cw)):   # up to 22 products deep, each with the error of its own chain
        assert rel_l2(gpu.read_grad(gn), passes * cn.grad) <= layers * chain_tolerance(d) + chain_tolerance(rows), i


# Convolutions in a trainer: 14 weight gradients of one kind, pooling at its tiles' edges (a window of two columns, 40 and 72
# channels, positions that fill no block), planes and channel sums that one layer leaves for the next.
NETS = {
    "deep": ((3, 8, 8), [("conv", 3, 32, 3, 1, 1), ("relu",)] + [("conv", 32, 32, 3, 1, 1), ("relu",)] * 14 + [("flatten",), ("linear", 2048, 10)]),
    "pools": ((2, 24, 16), [("conv", 2, 40, 3, 1, 1), ("relu",), ("maxpool", 2, 2), ("conv", 40, 72, 3, 1, 1), ("relu",), ("maxpool", 2, 2),
                            ("conv", 72, 64, 3, 1, 1), ("relu",), ("maxpool", 2, 2), ("conv", 64, 8, 3, 1, 1), ("relu",), ("flatten",),
                            ("linear", 48, 10)]),
    "two_columns": ((16, 6, 2), [("conv", 16, 48, 3, 1, 1), ("relu",), ("maxpool", 2, 2), ("conv", 48, 32, 3, 1, 1), ("relu",), ("flatten",),
                                 ("linear", 96, 10)]),
}


@pytest.mark.parametrize("net", list(NETS))
def test_trainer_convolutions(gpu_ctx, oracle64, net):
    shape, layers = NETS[net]
    rng = np.random.default_rng(len(net))
    x = rng.standard_normal((13, *shape)).astype(np.float32)
    t = np.eye(10, dtype=np.float32)[rng.integers(0, 10, 13)]
    tr = cuda.Trainer(layers, shape, 10, ctx=gpu_ctx)
    params = workloads.he_init(layers, 7)
    tr.set_params([p.ravel() for p in params])
    loss = tr.forward_backward(x, t)
    got = [tr.get_grad(i) for i in range(tr.n_params)]
    ref_loss, ref, _ = models.forward_backward(oracle64, layers, params, x, t, buffers=workloads.bn_buffers(layers))
    assert np.isclose(loss, ref_loss, rtol=1e-5)
    convs = sum(ly[0] == "conv" for ly in layers)
    for i, (a, b) in enumerate(zip(got, ref)):   # each layer adds its chain's error, forward and backward, then the gradient's own
        assert rel_l2(a, b) <= 2 * convs * chain_tolerance(648) + chain_tolerance(13 * 24 * 16), i


@pytest.mark.parametrize("c,n,hw", [(96, 9, 32), (96, 100, 8), (160, 20, 16), (160, 5, 32)])
def test_masked_data_gradients_with_a_ragged_column_tile(gpu_ctx, oracle64, c, n, hw):
    """64-column tiles by pairs of CTAs, 32 live channels in the last one, and the mask of the ReLU below.  Whole inputs and
    weights and a bias of a half: no pre-activation is near zero, whatever the rounding."""
    layers = [("conv", 3, c, 3, 1, 1), ("relu",), ("conv", c, 32, 3, 1, 1), ("flatten",), ("linear", 32 * hw * hw, 10)]
    rng = np.random.default_rng(c + n)
    x = rng.integers(-3, 4, (n, 3, hw, hw)).astype(np.float32)
    t = np.eye(10, dtype=np.float32)[rng.integers(0, 10, n)]
    params = workloads.he_init(layers, 7)
    params[0][:] = rng.integers(-1, 2, params[0].shape)
    params[1][:] = 0.5
    tr = cuda.Trainer(layers, (3, hw, hw), 10, ctx=gpu_ctx)
    tr.set_params([p.ravel() for p in params])
    tr.forward_backward(x, t)
    _, ref, _ = models.forward_backward(oracle64, layers, params, x, t, buffers={})
    for i, b in enumerate(ref):   # three products in a row each way, then the gradient's own
        assert rel_l2(tr.get_grad(i), b) <= 6 * chain_tolerance(9 * c) + chain_tolerance(min(8192, n * hw * hw)), i


@pytest.mark.parametrize("told", ["root", "view", "sibling"])
def test_views_of_rewritten_values(gpu_ctx, oracle64, told):
    """Values a hundred times the bound their operator left, written through the device pointer and announced through any
    node that shares them: whoever shares them multiplies the new ones."""
    n, ci, hw, co, out = 32, 32, 4, 32, 64
    rng = np.random.default_rng(3)
    x, wt = rng.standard_normal((n, ci, hw, hw)).astype(np.float32), (rng.standard_normal((co, ci, 3, 3)) / 17).astype(np.float32)
    w = (rng.standard_normal((co * hw * hw, out)) / 23).astype(np.float32)
    h = nn.conv2d(on_gpu(x), on_gpu(wt), on_gpu(np.zeros(co, np.float32)), 1, 1)
    views = [nn.flatten(h), graph.reshape(h, [n, co * hw * hw])]
    new = (100 * rng.standard_normal((n, co * hw * hw))).astype(np.float32)
    call(gpu_ctx, "nrs_d2d", _lib.VP(h.data_ptr()), Dev(gpu_ctx, new), new.nbytes)
    {"root": h, "view": views[0], "sibling": views[1]}[told].invalidate()
    got = gpu.to_host(graph.matmul(views[0], on_gpu(w))).reshape(n, out)
    err = np.abs(got - new.astype(np.float64) @ w.astype(np.float64))
    assert (err <= entry_bound(new, w, co * hw * hw)).all(), float(np.abs(got).max())


def test_batchnorm_whose_variance_is_lost(gpu_ctx):
    """Channels that are constant but for their first value, over 2^21 values: what is left of the variance is the rounding of
    its sums, and the first value lies up to thousands of times sqrt(count) away.  As planes for the next convolution it stays
    finite: the layer's statistics are the same in both modes, its products are not."""
    layers = [("batchnorm", 8), ("conv", 8, 32, 3, 1, 1), ("flatten",), ("linear", 32 * 64 * 64, 10)]
    rng = np.random.default_rng(4)
    x = np.zeros((512, 8, 64, 64), np.float32)
    x[0, :, 0, 0] = [100.1, 37.3, 211.7, 5.9, 1e4, 777.7, 3.3e-3, 63.1]
    t = np.eye(10, dtype=np.float32)[rng.integers(0, 10, 512)]
    params = workloads.he_init(layers, 7)
    got = {}
    try:
        for mode in (_lib.MATH_3XTF32, _lib.MATH_FP32):
            gpu_ctx.set_math_mode(mode)
            tr = cuda.Trainer(layers, (8, 64, 64), 10, ctx=gpu_ctx)
            tr.set_params([p.ravel() for p in params])
            tr.forward_backward(x, t)
            got[mode] = [tr.get_grad(2), tr.get_grad(4)]   # what the planes are multiplied with, and what they make
    finally:
        gpu_ctx.set_math_mode(_lib.MATH_3XTF32)
    for a, b in zip(*got.values()):   # a chain of 72, then of at most 8192 pixels; in f32 as many roundings again
        assert np.isfinite(a).all() and rel_l2(a, b) <= 2 * chain_tolerance(72) + 2 * chain_tolerance(8192)


@pytest.mark.parametrize("training", [True, False])
def test_batchnorm_channels_over_many_octaves(gpu_ctx, oracle64, training):
    """Gradients of channels down to 2^-23 of the largest: as planes, below a batch normalisation, they keep their bits."""
    n, c, hw = 8, 64, 8
    layers = [("conv", 16, c, 3, 1, 1), ("batchnorm", c), ("conv", c, 32, 3, 1, 1), ("flatten",), ("linear", 32 * hw * hw, 10)]
    rng = np.random.default_rng(6)
    x = rng.standard_normal((n, 16, hw, hw)).astype(np.float32)
    t = np.eye(10, dtype=np.float32)[rng.integers(0, 10, n)]
    params = workloads.he_init(layers, 7)
    params[2] = (2.0 ** -(np.arange(c) % 24)).astype(np.float32).reshape(params[2].shape)
    tr = cuda.Trainer(layers, (16, hw, hw), 10, ctx=gpu_ctx)
    tr.set_params([p.ravel() for p in params])
    tr.set_training(training)
    tr.forward_backward(x, t)
    _, ref, _ = models.forward_backward(oracle64, layers, params, x, t, buffers=workloads.bn_buffers(layers), training=training)
    got, want = np.asarray(tr.get_grad(0)).reshape(c, -1), np.asarray(ref[0]).reshape(c, -1)
    # two products forward and one back, twice for what is taken off again in between, then the gradient's own
    bound = 2 * (chain_tolerance(144) + 2 * chain_tolerance(9 * c)) + chain_tolerance(n * hw * hw)
    err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert (err <= bound).all(), float((err / bound).max())


@pytest.mark.parametrize("d,rows", [(64, 12), (256, 700), (512, 90)])
def test_bias_gradient_from_the_layernorm_above(gpu_ctx, oracle64, d, rows):
    """The column sums that LayerNorm's backward pass leaves for the feed-forward layer below it."""
    rng = np.random.default_rng(d)
    p = make_block_params(rng, d, 2 * d)
    batch, seq = 2, rows // 2
    x, seed = (rng.standard_normal((batch, seq, d)).astype(np.float32) for _ in range(2))
    g = og.Graph(oracle64)
    cx, cp = og.Node(x), {k: og.Node(v) for k, v in p.items()}
    cout = g.transformer_block(cx, cp, d // 32, 1e-5, "gelu", causal=True)
    cout.grad = seed.copy()
    og.backward_graph(cout)
    gx = on_gpu(x)
    block, gp = gpu_block(p, d // 32, "gelu", True)
    for total in (1, 2):
        out = block.forward(gx)
        gpu.set_grad(out, seed)
        backward_graph(out)
        for k in gp:
            assert rel_l2(gpu.read_grad(gp[k]), total * cp[k].grad) <= 2e-5, (k, total)   # (the bound of the block's other tests)


@pytest.mark.parametrize("rows,cols", [(1, 33), (255, 32), (256, 40), (1000, 257), (4100, 64), (70000, 8)])
@pytest.mark.parametrize("add", [0, 1])
def test_column_and_channel_sums(gpu_ctx, rows, cols, add):
    """Splits folded by the last block to arrive: of columns, and of channels (rows as images of 5 and of 8 pixels)."""
    rng = np.random.default_rng(rows + cols)
    a, old = rng.standard_normal((rows, cols)).astype(np.float32), rng.standard_normal(cols).astype(np.float32)
    out = Dev(gpu_ctx, old)
    call(gpu_ctx, "nrs_sum_axis0", Dev(gpu_ctx, a), out, rows, cols, add)
    ref = a.astype(np.float64).sum(0) + add * old
    # at most 14 additions in a row in any of the three stages below 4096 rows, rows / 2048 more above
    bound = (16 + rows / 1024) * 2.0**-23 * (np.abs(a).astype(np.float64).sum(0) + np.abs(old))
    assert (np.abs(out.get() - ref) <= bound).all()
    for px in (5, 8):
        if rows * px > 20000:
            continue
        img = rng.standard_normal((rows, cols, px)).astype(np.float32)
        out = Dev(gpu_ctx, old)
        call(gpu_ctx, "nrs_channel_sum", Dev(gpu_ctx, img), out, rows, cols, px, add)
        ref = img.astype(np.float64).sum((0, 2)) + add * old
        assert (np.abs(out.get() - ref) <= (24 + rows / 64) * 2.0**-23 * (np.abs(img).astype(np.float64).sum((0, 2)) + np.abs(old))).all()


@pytest.mark.parametrize("tokens,vocab,dim", [(1, 3, 5), (255, 7, 64), (1024, 2, 260), (1025, 50, 256), (5000, 3, 40), (600, 40, 1030)])
def test_embedding_gradient_in_token_order(gpu_ctx, tokens, vocab, dim):
    """The additions of a serial walk over the tokens, bit for bit, and rows that no token names."""
    rng = np.random.default_rng(tokens)
    g = rng.standard_normal((tokens, dim)).astype(np.float32)
    idx = rng.integers(0, max(1, vocab - 1), tokens).astype(np.int32)
    ref = np.zeros((vocab, dim), np.float32)
    for t in range(tokens):
        ref[idx[t]] += g[t]
    out = Dev(gpu_ctx, shape=(vocab, dim))
    call(gpu_ctx, "nrs_embedding_bwd", Dev(gpu_ctx, g), Dev(gpu_ctx, idx), out, tokens, dim, vocab, 0)
    assert np.array_equal(out.get(), ref)


def test_collected_chains_in_tf32(gpu_ctx):
    """Sixteen weight gradients over 2^17 rows in one launch: no accumulation chain becomes longer than 4096 rows for it.  All
    values are positive and exact in TF32, so what is lost is what the tensor core cuts: at most 2^-23 of the partial sum at each
    step of 8 rows, half of that over a chain whose sum grows evenly; the chains' sums are added up in f32."""
    rows, d, n = 1 << 17, 64, 16
    rng = np.random.default_rng(9)
    x, seed = ((1.0 + rng.integers(0, 1024, (rows, d)) / 1024.0).astype(np.float32) for _ in range(2))
    ref = x.astype(np.float64).T @ seed.astype(np.float64)
    gpu_ctx.set_math_mode(_lib.MATH_TF32)
    try:
        gx = on_gpu(x)   # (its gradient is wanted: the planes of the incoming one serve both products, and the second may wait)
        gw = [on_gpu((0.1 * rng.standard_normal((d, d))).astype(np.float32)) for _ in range(n)]
        out = graph.matmul(gx, gw[0])
        for w in gw[1:]:
            out = graph.add(out, graph.matmul(gx, w))
        gpu.set_grad(out, seed)
        backward_graph(out)
        for w in gw:
            assert rel_l2(gpu.read_grad(w), ref) <= (4096 / 8 / 2 + rows / 4096 + 8) * 2.0**-23
    finally:
        gpu_ctx.set_math_mode(_lib.MATH_3XTF32)


def test_ranges_of_a_captured_graph(gpu_ctx):
    """A graph of convolutions, replayed between eager work: its ranges start from nothing each time, and the tensors that were
    staged after its capture keep theirs."""
    n, ci, h, co, layers = 2, 32, 6, 32, 150
    args = (n, ci, h, h, co, 3, 3, 1, 1, 0)
    rng = np.random.default_rng(12)
    x = rng.standard_normal((n, ci, h, h)).astype(np.float32)
    wt = (rng.standard_normal((co, ci, 3, 3)) / 17).astype(np.float32)
    cu, ctx = ctypes.CDLL("libcuda.so.1"), cuda.Context(0)
    try:
        wd, bd = Dev(ctx, wt), Dev(ctx, np.zeros(co, np.float32))
        xd, ys = Dev(ctx, x), [Dev(ctx, shape=(n, co, h, h)) for _ in range(layers)]
        eager = Dev(ctx, shape=(n, co, h, h))

        def expect(values):
            call(ctx, "nrs_h2d", xd, _lib.VP(values.ctypes.data), values.nbytes)
            call(ctx, "nrs_conv2d_fwd", xd, wd, bd, eager, *args)
            return eager.get()

        want = {s: expect(np.ascontiguousarray(x * np.float32(s))) for s in (1.0, 1e6, 1e-6)}
        stream, graph_h, exec_h = ctypes.c_void_p(ctx._l.nrs_get_stream(ctx.h)), ctypes.c_void_p(), ctypes.c_void_p()
        assert cu.cuStreamBeginCapture_v2(stream, 2) == 0      # relaxed
        for y in ys:
            call(ctx, "nrs_conv2d_fwd", xd, wd, bd, y, *args)
        assert cu.cuStreamEndCapture(stream, ctypes.byref(graph_h)) == 0
        assert cu.cuGraphInstantiateWithFlags(ctypes.byref(exec_h), graph_h, ctypes.c_ulonglong(0)) == 0
        scaled = [(2.0**i, Dev(ctx, (x * np.float32(2.0**i)).astype(np.float32))) for i in range(-20, 20)]
        scaled += [(1.0, Dev(ctx, x)) for _ in range(260)]      # (more than a page of ranges)
        for _, t in scaled:
            call(ctx, "nrs_planes_cache", t, n, ci, h, h)
        for s, ref in list(want.items()) * 2:
            v = np.ascontiguousarray(x * np.float32(s))
            call(ctx, "nrs_h2d", xd, _lib.VP(v.ctypes.data), v.nbytes)
            assert cu.cuGraphLaunch(exec_h, stream) == 0
            ctx.sync()
            assert all(np.array_equal(ys[i].get(), ref) for i in (0, 1, layers // 2, layers - 1)), s
        for f, t in scaled:
            call(ctx, "nrs_conv2d_fwd", t, wd, bd, eager, *args)
            assert np.array_equal(eager.get(), want[1.0] * np.float32(f)), f
        assert cu.cuGraphExecDestroy(exec_h) == 0 and cu.cuGraphDestroy(graph_h) == 0
    finally:
        ctx.close()


def test_profiling_brackets_what_a_step_launches(gpu_ctx):
    """The launches of a step are the same with brackets around them, and a family's work is its layers'."""
    shape, layers = NETS["deep"]
    n = 13
    rng = np.random.default_rng(1)
    x, t = rng.standard_normal((n, *shape)).astype(np.float32), np.eye(10, dtype=np.float32)[rng.integers(0, 10, n)]
    tr = cuda.Trainer(layers, shape, 10, ctx=gpu_ctx)
    tr.set_params([p.ravel() for p in workloads.he_init(layers, 7)])
    tr.step(x, t)
    launches, ms, work, calls = [], ctypes.c_double(), ctypes.c_double(), ctypes.c_uint64()
    try:
        for on in (0, 1):
            call(gpu_ctx, "nrs_profile_enable", on)
            before = gpu_ctx.launch_count()
            tr.step(x, t)
            launches.append(gpu_ctx.launch_count() - before)
        call(gpu_ctx, "nrs_profile_get", 2, ctypes.byref(ms), ctypes.byref(work), ctypes.byref(calls))   # weight gradients of convolutions
    finally:
        call(gpu_ctx, "nrs_profile_enable", 0)
        call(gpu_ctx, "nrs_profile_reset")
    assert launches[0] == launches[1] and calls.value < 15 and ms.value > 0
    assert np.isclose(work.value, sum(18.0 * n * 64 * ly[1] * ly[2] for ly in layers if ly[0] == "conv"))


def test_rows_far_below_the_largest_through_two_products(gpu_ctx):
    """A hidden layer whose pairs take their exponent from K * max * max, with rows down to 2^-44 of the largest: what is lost of
    a row is its own rounding and 2^-50 of the bounds, no more; rows within 2^-16 keep their bits."""
    m, k, hid, n = 64, 256, 1024, 128
    rng = np.random.default_rng(13)
    x = (rng.standard_normal((m, k)) * 2.0 ** -(np.arange(m) % 45)[:, None]).astype(np.float32)
    w1, w2 = ((rng.standard_normal(s) / np.sqrt(s[0])).astype(np.float32) for s in ((k, hid), (hid, n)))
    h = nn.linear_act(on_gpu(x), on_gpu(w1), on_gpu(np.zeros(hid, np.float32)), _lib.ACT_GELU)
    got = gpu.to_host(nn.Linear(on_gpu(w2), on_gpu(np.zeros(n, np.float32))).forward(h)).reshape(m, n)
    pre = x.astype(np.float64) @ w1.astype(np.float64)
    hr = 0.5 * pre * (1.0 + np.tanh(np.sqrt(2.0 / np.pi) * (pre + 0.044715 * pre**3)))
    bound_h = 1.001 * k * np.abs(x).max() * np.abs(w1).max()
    # (GELU: its slope, a few roundings, and its exponential's error, which is relative to the argument's size)
    err_h = 1.13 * entry_bound(x, w1, k) + 2.0**-20 * (np.abs(hr) + np.abs(pre) * 2.0**-2) + 2.0**-50 * bound_h
    a2 = np.abs(w2).astype(np.float64)
    rel = 3 * 2.0**-22 + (2 * hid / 16 + 4) * 2.0**-23
    most = rel * (np.abs(hr) @ a2) + err_h @ a2 + 2.0**-50 * (bound_h * a2.sum(0)[None, :] + np.abs(hr).sum(1)[:, None] * a2.max())
    ref = hr @ w2.astype(np.float64)
    err = np.abs(got - ref)
    assert (err <= most).all(), float((err / most).max())
    kept = np.arange(m) % 45 <= 16
    assert (np.linalg.norm(err[kept], axis=1) <= (chain_tolerance(k) + chain_tolerance(hid) + 2.0**-20) * np.linalg.norm(ref[kept], axis=1)).all()
