"""Convolutions off the aligned path on the tensor cores: ragged channel counts, strides, few-channel layers through
patch planes, rows wider than a tile, wide inputs; forward, data gradient, weight gradient and bias gradient against
the CPU oracle, in overwrite and accumulate mode."""
import numpy as np
import pytest

from neuralrs_b200 import _lib
from .conftest import rel_l2
from .gpu_util import Dev, call

pytestmark = pytest.mark.gpu
TOL = {_lib.MATH_3XTF32: 1e-4, _lib.MATH_TF32: 1e-2}

CASES = [
    # n, ci, h, w, co, kh, kw, stride, pad
    (3, 48, 13, 11, 80, 3, 3, 2, 1),     # stride 2, both channel counts ragged, odd image
    (2, 16, 9, 9, 16, 3, 3, 1, 1),       # less than one channel block
    (2, 10, 9, 7, 6, 3, 3, 1, 1),        # no multiple of four: padded pixel rows
    (2, 33, 8, 8, 130, 3, 3, 1, 1),      # one channel into the second block, two into the second row tile
    (2, 40, 7, 29, 36, 5, 5, 1, 2),      # 29-pixel rows
    (1, 32, 6, 150, 32, 3, 3, 1, 1),     # rows wider than a pixel tile
    (2, 24, 12, 10, 40, 2, 2, 3, 0),     # stride larger than the kernel: pixels without a gradient
    (2, 32, 11, 12, 48, 1, 1, 2, 0),     # 1x1 with stride
    (2, 64, 15, 15, 32, 3, 5, 4, 2),     # stride 4, rectangular kernel
    (2, 260, 6, 6, 40, 3, 3, 1, 1),      # more input channels than one column block
    (6, 3, 24, 20, 20, 5, 5, 1, 2),      # 75-value patches
    (6, 2, 33, 31, 24, 3, 3, 2, 1),      # strided patches
    (5, 1, 28, 28, 16, 3, 3, 1, 1),      # 16 output channels on patches
    (2, 32, 10, 10, 32, 3, 3, 1, 0),     # no padding: the gradient's image is larger than dy's
    (1, 5, 6, 6, 7, 3, 3, 1, 1),         # few pixels, few channels
]


@pytest.mark.parametrize("mode", [_lib.MATH_3XTF32, _lib.MATH_TF32], ids=["3xtf32", "tf32"])
@pytest.mark.parametrize("cfg", CASES)
def test_conv_general_shapes(gpu_ctx, oracle64, mode, cfg):
    n, ci, h, w, co, kh, kw, s, p = cfg
    rng = np.random.default_rng(sum(cfg))
    x = rng.normal(size=(n, ci, h, w)).astype(np.float32)
    wt = (rng.normal(size=(co, ci, kh, kw)) * np.sqrt(2.0 / (ci * kh * kw))).astype(np.float32)
    b = rng.normal(size=co).astype(np.float32) * 0.1
    yref = oracle64.conv2d_fwd(x, wt, b, s, p)
    dy = rng.normal(size=yref.shape).astype(np.float32)
    refs = oracle64.conv2d_bwd(x, wt, dy, s, p)
    gpu_ctx.set_math_mode(mode)
    try:
        xd, wd, bd, dyd = (Dev(gpu_ctx, a) for a in (x, wt, b, dy))
        y = Dev(gpu_ctx, shape=yref.shape)
        grads = [Dev(gpu_ctx, shape=a.shape) for a in (x, wt, b)]
        for cached in (False, True):
            if cached:
                call(gpu_ctx, "nrs_planes_cache", xd, n, ci, h, w)
                call(gpu_ctx, "nrs_planes_cache", dyd, n, co, *yref.shape[2:])
            call(gpu_ctx, "nrs_conv2d_fwd", xd, wd, bd, y, *cfg, 1)
            assert rel_l2(y.get(), np.maximum(yref, 0)) <= TOL[mode]
            for k in (1, 2):
                call(gpu_ctx, "nrs_conv2d_bwd", xd, wd, dyd, *grads, *cfg, k - 1)
                for g, ref in zip(grads, refs):
                    assert rel_l2(g.get(), k * ref) <= TOL[mode]
        call(gpu_ctx, "nrs_planes_drop", xd)
        call(gpu_ctx, "nrs_planes_drop", dyd)
    finally:
        gpu_ctx.set_math_mode(_lib.MATH_3XTF32)
