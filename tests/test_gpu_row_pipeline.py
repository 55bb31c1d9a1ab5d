"""The shared-memory row pipeline of the row-wise operators: sizes where it takes over, odd widths, groups of rows with
a ragged last copy, rows spread over several warps, one row, and the widest row it takes; against the f64 oracle."""
import ctypes as C

import numpy as np
import pytest

from .conftest import rel_l2
from .gpu_util import Dev, call

pytestmark = pytest.mark.gpu
F = C.c_float
SHAPES = [(3, 17), (9001, 17), (1031, 515), (4100, 256), (1060, 1000), (257, 2050), (130, 4097), (17, 8192), (17, 8193), (70001, 2), (8400, 1000), (4400, 1406), (8401, 1001),
          (33601, 250)]


@pytest.mark.parametrize("rows,f", SHAPES)
def test_row_pipeline(gpu_ctx, oracle64, rows, f):
    rng = np.random.default_rng(rows + f)
    a, b, g = (rng.normal(size=(rows, f)).astype(np.float32) for _ in range(3))
    gamma, beta = rng.normal(size=f).astype(np.float32), rng.normal(size=f).astype(np.float32)
    labels = rng.integers(0, f, rows).astype(np.int32)
    t = np.zeros((rows, f), np.float32)
    t[np.arange(rows), labels] = 1.0
    x = (a + b).astype(np.float32)
    ad, bd, gd, gm, bt, td, lb = (Dev(gpu_ctx, v) for v in (a, b, g, gamma, beta, t, labels))
    y, xh, o1 = (Dev(gpu_ctx, shape=(rows, f)) for _ in range(3))
    ist, dg, db, loss = Dev(gpu_ctx, shape=(rows,)), Dev(gpu_ctx, shape=(f,)), Dev(gpu_ctx, shape=(f,)), Dev(gpu_ctx, shape=(1,))
    if f > 1:   # one feature has no variance
        yr, xhr, isr = oracle64.layernorm_fwd(x, gamma, beta, 1e-5)
        call(gpu_ctx, "nrs_layernorm_residual_fwd", ad, bd, gm, bt, y, xh, ist, rows, f, F(1e-5))
        assert np.abs(y.get() - yr).max() <= 2e-4 and np.abs(xh.get() - xhr).max() <= 2e-4
        dxr, dgr, dbr = oracle64.layernorm_bwd(g, xhr, isr, gamma)
        o2 = Dev(gpu_ctx, np.ones_like(a))
        call(gpu_ctx, "nrs_layernorm_residual_bwd", gd, xh, ist, gm, o1, o2, dg, db, rows, f, 0, 1, 0)
        assert rel_l2(o1.get(), dxr) <= 2e-5 and rel_l2(o2.get() - 1.0, dxr) <= 4e-5
        assert rel_l2(dg.get(), dgr) <= 1e-5 and rel_l2(db.get(), dbr) <= 1e-5
    xd = Dev(gpu_ctx, x)
    pr = oracle64.softmax_fwd(x)
    call(gpu_ctx, "nrs_softmax_fwd", xd, y, rows, f)
    assert rel_l2(y.get(), pr) <= 1e-6
    sr = pr * (g - (pr * g).sum(1, keepdims=True))
    for k in (1, 2):
        call(gpu_ctx, "nrs_softmax_bwd", y, gd, o1, rows, f, k - 1)
        assert np.linalg.norm(o1.get() - k * sr) <= 1e-5 * np.linalg.norm(pr * g)
    ref_loss = -np.log(pr[np.arange(rows), labels]).mean()
    for name, target in (("nrs_ce_fwd_bwd", td), ("nrs_ce_fwd_bwd_indexed", lb)):
        call(gpu_ctx, name, xd, target, loss, o1, rows, f, rows)
        assert abs(loss.get()[0] - ref_loss) <= 1e-5 * max(1.0, abs(ref_loss))
        assert np.linalg.norm(o1.get() - (pr - t) / rows) <= 2e-6 * np.linalg.norm(t) / rows


# Both sides of the lines between the pipeline and the kernels it stands beside (rows, columns).
LINES = [(16500, 256), (33000, 260), (32900, 384), (11000, 400), (6100, 1000), (1024, 255), (1029, 255), (200, 1025), (127, 1028),
         (16800, 501), (1050, 4004), (2100, 4004), (95000, 90), (140000, 90), (1600, 90), (17000, 250), (210000, 40),
         (5400, 777), (10900, 777), (17000, 511), (4300, 1402), (4300, 1403), (149, 1401), (1125, 1401)]


@pytest.mark.parametrize("rows,f", LINES)
def test_layernorm_beside_its_lines(gpu_ctx, oracle64, rows, f):
    rng = np.random.default_rng(rows * 3 + f)
    x, g = (rng.normal(size=(rows, f)).astype(np.float32) for _ in range(2))
    gamma, beta = rng.normal(size=f).astype(np.float32), rng.normal(size=f).astype(np.float32)
    xd, gd, gm, bt = (Dev(gpu_ctx, v) for v in (x, g, gamma, beta))
    y, xh, dx = (Dev(gpu_ctx, shape=(rows, f)) for _ in range(3))
    ist, dg, db = Dev(gpu_ctx, shape=(rows,)), Dev(gpu_ctx, np.ones(f, np.float32)), Dev(gpu_ctx, np.ones(f, np.float32))
    yr, xhr, isr = oracle64.layernorm_fwd(x, gamma, beta, 1e-5)
    call(gpu_ctx, "nrs_layernorm_fwd", xd, gm, bt, y, xh, ist, rows, f, F(1e-5))
    assert np.abs(y.get() - yr).max() <= 2e-4 and np.abs(xh.get() - xhr).max() <= 2e-4 and rel_l2(ist.get(), isr) <= 1e-6
    dxr, dgr, dbr = oracle64.layernorm_bwd(g, xhr, isr, gamma)
    call(gpu_ctx, "nrs_layernorm_bwd", gd, xh, ist, gm, dx, None, None, rows, f, 0, 0)
    assert rel_l2(dx.get(), dxr) <= 2e-5
    for k in (1, 2):   # parameters alone, added to what is there
        call(gpu_ctx, "nrs_layernorm_bwd", gd, xh, ist, gm, None, dg, db, rows, f, 0, 1)
        assert rel_l2(dg.get() - 1.0, k * dgr) <= 2e-5 and rel_l2(db.get() - 1.0, k * dbr) <= 2e-5
    call(gpu_ctx, "nrs_layernorm_bwd", gd, xh, ist, gm, dx, dg, db, rows, f, 1, 0)
    assert rel_l2(dx.get(), 2.0 * dxr) <= 2e-5 and rel_l2(dg.get(), dgr) <= 1e-5 and rel_l2(db.get(), dbr) <= 1e-5


SOFTMAX_LINES = [(150, 1281), (3300, 1281), (9900, 1281), (4300, 1401), (4000, 1502), (2950, 2050), (2050, 3000), (17000, 1502), (1500, 4096)]


@pytest.mark.parametrize("rows,f", SOFTMAX_LINES)
def test_softmax_beside_its_lines(gpu_ctx, oracle64, rows, f):
    rng = np.random.default_rng(rows + 5 * f)
    x = (4.0 * rng.normal(size=(rows, f))).astype(np.float32)
    x[1, ::2] = np.finfo(np.float32).min   # a masked row, and one with a single live column
    x[2, 1:] = -np.inf
    g = rng.normal(size=(rows, f)).astype(np.float32)
    xd, gd, y, dx = Dev(gpu_ctx, x), Dev(gpu_ctx, g), Dev(gpu_ctx, shape=(rows, f)), Dev(gpu_ctx, shape=(rows, f))
    call(gpu_ctx, "nrs_softmax_fwd", xd, y, rows, f)
    got = y.get()
    assert rel_l2(got, oracle64.softmax_fwd(x)) <= 1e-6
    assert (got[1, ::2] == 0).all() and got[2, 0] == 1.0 and (got[2, 1:] == 0).all()
    yg = got.astype(np.float64) * g
    want = yg - got * yg.sum(1, keepdims=True)
    for k in (1, 2):
        call(gpu_ctx, "nrs_softmax_bwd", y, gd, dx, rows, f, k - 1)
        assert np.linalg.norm(dx.get() - k * want) <= 1e-5 * np.linalg.norm(yg)


# Both sides of the lines against the pipeline; the scalar kernel with its own mean and with a second launch for it.
CE_LINES = [(8400, 1000), (16400, 512), (33000, 256), (33000, 255), (21900, 385), (32800, 385), (6600, 1281), (5600, 1502), (5600, 1501),
            (1, 7), (2048, 63), (2100, 63), (4096, 31), (4097, 31), (2048, 127), (300, 1001), (70, 1801), (65535, 7), (65536, 7), (262144, 3)]


@pytest.mark.parametrize("rows,f", CE_LINES)
def test_cross_entropy_beside_its_lines(gpu_ctx, oracle64, rows, f):
    rng = np.random.default_rng(rows + 7 * f)
    x = (3.0 * rng.normal(size=(rows, f))).astype(np.float32)
    labels = rng.integers(0, f, rows).astype(np.int32)
    t = np.zeros((rows, f), np.float32)
    t[np.arange(rows), labels] = 1.0
    xd, td, lb = (Dev(gpu_ctx, v) for v in (x, t, labels))
    g, loss, rl = Dev(gpu_ctx, shape=(rows, f)), Dev(gpu_ctx, shape=(1,)), Dev(gpu_ctx, shape=(rows,))
    p = oracle64.softmax_fwd(x)
    each = -np.log(p[np.arange(rows), labels].astype(np.float64))
    for name, target in (("nrs_ce_fwd_bwd", td), ("nrs_ce_fwd_bwd_indexed", lb)):
        call(gpu_ctx, name, xd, target, loss, g, rows, f, rows)
        assert abs(loss.get()[0] - each.mean()) <= 1e-5 * each.mean()
        assert np.linalg.norm(g.get() - (p - t) / rows) <= 2e-6 * np.linalg.norm(t) / rows
    call(gpu_ctx, "nrs_ce_fwd", xd, td, None, rl, rows, f, rows)
    assert rel_l2(rl.get(), each) <= 1e-6
    call(gpu_ctx, "nrs_ce_fwd", xd, td, loss, rl, rows, f, 2 * rows)
    assert abs(loss.get()[0] - each.mean() / 2) <= 1e-5 * each.mean() and rel_l2(rl.get(), each) <= 1e-6
