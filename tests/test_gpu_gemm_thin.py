"""GEMMs with few rows: one row to fifteen (weights streamed once, K-splits folded by the last block), sixteen and more
on padded tensor-core tiles with short K-splits, ragged columns and reductions; A^T B on MN-major slices for an output
beyond the weight-gradient kernel's; against the f64 oracle."""
import ctypes as C

import numpy as np
import pytest

from neuralrs_b200 import _lib
from .conftest import rel_l2
from .gpu_util import Dev, call

pytestmark = pytest.mark.gpu
F = C.c_float
TOL = {_lib.MATH_3XTF32: 1e-4, _lib.MATH_FP32: 1e-4, _lib.MATH_TF32: 1e-2}
SHAPES = [(1, 128, 3136), (1, 10, 128), (2, 33, 64), (5, 1000, 515), (9, 40, 1030), (15, 257, 700), (16, 128, 3136), (33, 70, 600), (63, 96, 40)]


@pytest.mark.parametrize("mode", list(TOL), ids=["3xtf32", "fp32", "tf32"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_gemm_few_rows(gpu_ctx, oracle64, mode, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.normal(size=(m, k)).astype(np.float32), rng.normal(size=(k, n)).astype(np.float32)
    bias, c0 = rng.normal(size=n).astype(np.float32), rng.normal(size=(m, n)).astype(np.float32)
    ref = oracle64.matmul_fwd(a, b)
    gpu_ctx.set_math_mode(mode)
    try:
        for ta in (0, 1):
            for tb in (0, 1):
                da, db, dc = Dev(gpu_ctx, a.T if ta else a), Dev(gpu_ctx, b.T if tb else b), Dev(gpu_ctx, c0)
                call(gpu_ctx, "nrs_gemm", ta, tb, m, n, k, da, db, dc, None, 0, F(1))
                assert rel_l2(dc.get(), ref + c0) <= TOL[mode]
        call(gpu_ctx, "nrs_gemm", 0, 0, m, n, k, Dev(gpu_ctx, a), Dev(gpu_ctx, b), dc, Dev(gpu_ctx, bias), 1, F(0))
        assert rel_l2(dc.get(), np.maximum(ref + bias, 0)) <= TOL[mode]
    finally:
        gpu_ctx.set_math_mode(_lib.MATH_3XTF32)


@pytest.mark.parametrize("mode", [_lib.MATH_3XTF32, _lib.MATH_TF32], ids=["3xtf32", "tf32"])
def test_gemm_tn_large_output(gpu_ctx, mode):
    m, n, k = 2080, 2144, 200      # above the weight-gradient kernel's output size, ragged tiles, ragged last K-slice
    rng = np.random.default_rng(3)
    a, b = rng.normal(size=(k, m)).astype(np.float32), rng.normal(size=(k, n)).astype(np.float32)
    ref = a.astype(np.float64).T @ b.astype(np.float64)
    gpu_ctx.set_math_mode(mode)
    try:
        dc = Dev(gpu_ctx, shape=(m, n))
        for i in (1, 2):
            call(gpu_ctx, "nrs_gemm", 1, 0, m, n, k, Dev(gpu_ctx, a), Dev(gpu_ctx, b), dc, None, 0, F(i - 1))
            assert rel_l2(dc.get(), i * ref) <= TOL[mode]
    finally:
        gpu_ctx.set_math_mode(_lib.MATH_3XTF32)


@pytest.mark.parametrize("m,n,k", [(1300, 1000, 8300), (2500, 130, 4100), (1408, 1024, 12288)])
def test_gemm_long_reduction_in_chunks(gpu_ctx, oracle64, m, n, k):
    """Reductions beyond one accumulation chain with enough tiles to fill the GPU; every operand order, added to C."""
    rng = np.random.default_rng(k)
    a, b = rng.normal(size=(m, k)).astype(np.float32), rng.normal(size=(k, n)).astype(np.float32)
    bias, c0 = rng.normal(size=n).astype(np.float32), rng.normal(size=(m, n)).astype(np.float32)
    rows = np.r_[0:3, 127:130, m - 2:m]
    ref = oracle64.matmul_fwd(a[rows], b)
    for ta, tb in ((0, 0), (0, 1), (1, 0)):
        da, db, dc = Dev(gpu_ctx, a.T if ta else a), Dev(gpu_ctx, b.T if tb else b), Dev(gpu_ctx, c0)
        call(gpu_ctx, "nrs_gemm", ta, tb, m, n, k, da, db, dc, None, 0, F(1))
        assert rel_l2(dc.get()[rows], ref + c0[rows]) <= 5e-5
    call(gpu_ctx, "nrs_gemm", 1, 0, m, n, k, da, db, dc, Dev(gpu_ctx, bias), 1, F(0))
    assert rel_l2(dc.get()[rows], np.maximum(ref + bias, 0)) <= 5e-5


def test_conv_long_reduction_in_chunks(gpu_ctx, oracle64):
    rng = np.random.default_rng(9)
    n, ci, h, co = 16, 4100, 10, 330
    x, w = rng.normal(size=(n, ci, h, h)).astype(np.float32), rng.normal(size=(co, ci, 1, 1)).astype(np.float32)
    y = Dev(gpu_ctx, shape=(n, co, h, h))
    call(gpu_ctx, "nrs_conv2d_fwd", Dev(gpu_ctx, x), Dev(gpu_ctx, w), None, y, n, ci, h, h, co, 1, 1, 1, 0, 0)
    got = y.get()
    for i in (0, n - 1):
        assert rel_l2(got[i], oracle64.matmul_fwd(w[:, :, 0, 0], x[i].reshape(ci, h * h))) <= 5e-5
