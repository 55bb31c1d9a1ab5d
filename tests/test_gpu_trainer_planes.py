"""A trainer's operand planes at ragged sizes: weights of both forms (taps beyond one tile, channels that are no multiple
of a tile, linear layers with odd rows), batch-normalised tensors whose planes come out of the normalise and dx kernels,
images smaller than a tile; gradients in every math mode against the f64 oracle."""
import numpy as np
import pytest

from neuralrs_b200 import _lib, cuda, workloads
from oracle import models
from .conftest import rel_l2

pytestmark = pytest.mark.gpu
NETS = {
    "bn": ((3, 10, 10), [("conv", 3, 40, 5, 1, 2), ("batchnorm", 40), ("relu",), ("conv", 40, 72, 3, 1, 1), ("batchnorm", 72), ("relu",),
                         ("conv", 72, 48, 5, 1, 2), ("batchnorm", 48), ("maxpool", 2, 2), ("flatten",), ("linear", 1200, 70), ("relu",),
                         ("linear", 70, 10)]),
    "odd": ((4, 9, 7), [("conv", 4, 33, 3, 1, 1), ("relu",), ("conv", 33, 65, 4, 1, 2), ("relu",), ("conv", 65, 17, 7, 1, 3), ("relu",), ("flatten",),
                        ("linear", 1360, 131), ("relu",), ("linear", 131, 10)]),
    # classifier heads over fused activations, more rows than one block takes
    "head": ((2, 6, 9), [("flatten",), ("linear", 108, 136), ("relu",), ("linear", 136, 10)]),
    "head_gelu": ((2, 6, 9), [("flatten",), ("linear", 108, 72), ("gelu",), ("linear", 72, 10)]),
}


def gradients(ctx, mode, shape, layers, x, t, params):
    ctx.set_math_mode(mode)
    try:
        tr = cuda.Trainer(layers, shape, 10, ctx=ctx)
        if params is None:
            rng = np.random.default_rng(3)
            params = [(rng.standard_normal(tr.param_len(i)) * 0.08).astype(np.float32) for i in range(tr.n_params)]
        tr.set_params(params)
        loss = tr.forward_backward(x, t)
        return loss, params, [tr.get_grad(i) for i in range(tr.n_params)]
    finally:
        ctx.set_math_mode(_lib.MATH_3XTF32)


# Relative error (2-norm) of a tensor's gradient.  FP32 and 3xTF32: a chain of K elements errs by some 7e-9 K in 3xTF32, K
# up to 1800 here, and the layers' errors add (4.7e-6 is the most seen).  TF32 operands carry 11 bits, 1.4e-4 rms each, so a
# product errs by 2e-4 and a network of smooth layers by a few times that.  A ReLU turns a pre-activation that such an error d
# moves across zero into a whole unit of gradient: with unit variance a share of 0.8 d of them, which is an error of
# sqrt(0.8 d) = 2e-2 for d = 5e-4 (3.4e-2 is the most seen, under batch normalisation).
TOL = {_lib.MATH_FP32: 3e-6, _lib.MATH_3XTF32: 2e-5, _lib.MATH_TF32: 6e-2}
TOL_SMOOTH_TF32 = 1.5e-3


@pytest.mark.parametrize("net", list(NETS))
@pytest.mark.parametrize("mode", list(TOL), ids=["fp32", "3xtf32", "tf32"])
def test_trainer_planes_ragged(gpu_ctx, oracle64, net, mode):
    shape, layers = NETS[net]
    rng = np.random.default_rng(5)
    batch = 150 if net.startswith("head") else 24
    x = rng.standard_normal((batch, *shape)).astype(np.float32)
    t = np.eye(10, dtype=np.float32)[rng.integers(0, 10, batch)]
    loss, params, got = gradients(gpu_ctx, mode, shape, layers, x, t, None)
    shaped = [p.reshape(like.shape) for p, like in zip(params, workloads.he_init(layers, 1))]
    ref_loss, ref, _ = models.forward_backward(oracle64, layers, shaped, x, t, buffers=workloads.bn_buffers(layers))
    tol = TOL_SMOOTH_TF32 if mode == _lib.MATH_TF32 and net == "head_gelu" else TOL[mode]
    assert np.isclose(loss, ref_loss, rtol=min(tol, 5e-4))
    scale = max(np.abs(b).max() for b in ref)
    for i, (a, b) in enumerate(zip(got, ref)):
        if np.abs(b).max() < 1e-5 * scale:   # a bias under a batch normalisation: rounding noise
            assert np.abs(a).max() < 1e-6 * scale, i
        else:
            assert rel_l2(a, b) <= tol, i
