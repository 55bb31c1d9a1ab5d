"""A trainer's operand planes at ragged sizes: weights of both forms (taps beyond one tile, channels that are no multiple
of a tile, linear layers with odd rows), batch-normalised tensors whose planes come out of the normalise and dx kernels,
images smaller than a tile; gradients against the same trainer in FP32 mode, which reads no
planes."""
import numpy as np
import pytest

from neuralrs_b200 import _lib, cuda
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


@pytest.mark.parametrize("net", list(NETS))
@pytest.mark.parametrize("mode,tol", [(_lib.MATH_3XTF32, 2e-4), (_lib.MATH_TF32, 2e-2)], ids=["3xtf32", "tf32"])
def test_trainer_planes_ragged(gpu_ctx, net, mode, tol):
    shape, layers = NETS[net]
    rng = np.random.default_rng(5)
    batch = 150 if net.startswith("head") else 24
    x = rng.standard_normal((batch, *shape)).astype(np.float32)
    t = np.eye(10, dtype=np.float32)[rng.integers(0, 10, batch)]
    ref_loss, params, ref = gradients(gpu_ctx, _lib.MATH_FP32, shape, layers, x, t, None)
    loss, _, got = gradients(gpu_ctx, mode, shape, layers, x, t, params)
    assert np.isclose(loss, ref_loss, rtol=tol)
    scale = max(np.abs(b).max() for b in ref)
    for i, (a, b) in enumerate(zip(got, ref)):
        if np.abs(b).max() < 1e-5 * scale:   # a bias under a batch normalisation: rounding noise
            assert np.abs(a).max() < tol * scale, i
        else:
            assert rel_l2(a, b) <= 10 * tol, i
