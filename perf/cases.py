"""Workloads that the performance of this framework is judged on, and how to run one.

A case is a plain dict.  Its "kind" says which program of a user it stands for:

    infer    one forward pass of a small CNN through the node API: image from the host, logits back to it
    loop     the reference's own training loop through the node API (to_cuda, zero_grad, forward, cross_entropy,
             cross_entropy_backward, backward_graph, AdamW.step)
    epoch    the native trainer over a few staged batches (losses read one step behind), weights read back at the end
    conv     one convolution layer, forward and all three gradients, through the operator-level C ABI
    rows     the row-wise operators (LayerNorm with residual, softmax, cross-entropy), forward and backward,
             through the operator-level C ABI

Everything runs on one CUDA stream owned by the caller, as inside a host framework.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from neuralrs_b200 import _lib, cuda, workloads
from neuralrs_b200._lib import VP, check

MODES = {"3xtf32": _lib.MATH_3XTF32, "tf32": _lib.MATH_TF32, "fp32": _lib.MATH_FP32}

# The three-convolution digit classifier of the reference's README (16 -> 32 -> 64 channels).
DIGITS_CNN = dict(
    in_shape=(1, 28, 28), classes=10,
    layers=[("conv", 1, 16, 3, 1, 1), ("relu",), ("maxpool", 2, 2), ("conv", 16, 32, 3, 1, 1), ("relu",), ("maxpool", 2, 2),
            ("conv", 32, 64, 3, 1, 1), ("relu",), ("flatten",), ("linear", 3136, 128), ("relu",), ("linear", 128, 10)])


def listed():
    return [
        # One image classified on request: latency and launches are all there is.
        {"name": "infer_b1", "kind": "infer", "batch": 1, "mode": "3xtf32"},
        # The README's training run: define-by-run loop, batch 32, operators not fused.
        {"name": "loop_digits_b32", "kind": "loop", "model": "digits", "batch": 32, "mode": "3xtf32"},
        # The small CNN configuration at its batch of 64.
        {"name": "small_cnn_b64", "kind": "epoch", "model": "small_cnn", "batch": 64, "steps": 16, "mode": "3xtf32"},
        # The CIFAR-shaped CNN at about one rank's share of its global batch on eight GPUs, a ragged one.
        {"name": "vgg_b100", "kind": "epoch", "model": "vgg", "batch": 100, "steps": 12, "mode": "3xtf32"},
        # The headline configuration: the CIFAR-shaped CNN at batch 1024.
        {"name": "vgg_b1024", "kind": "epoch", "model": "vgg", "batch": 1024, "steps": 6, "mode": "3xtf32"},
        # The reference example's BatchNorm + Dropout model with its augmentation, in the faster opt-in precision.
        {"name": "vgg_bn_b256_tf32", "kind": "epoch", "model": "vgg_bn", "batch": 256, "steps": 8, "mode": "tf32"},
        # The language-model configuration: 32 sequences of 128 tokens.
        {"name": "lm_b32_s128", "kind": "epoch", "model": "lm", "batch": 32, "seq": 128, "d_model": 256, "heads": 8,
         "steps": 12, "mode": "3xtf32"},
        # A wider language model on longer sequences of an odd length.
        {"name": "lm_b6_s500", "kind": "epoch", "model": "lm", "batch": 6, "seq": 500, "d_model": 512, "heads": 8,
         "steps": 8, "mode": "3xtf32"},
        # The wide MLP at its global batch, inputs resident on the device: the largest contractions.
        {"name": "loop_mlp_b16384", "kind": "loop", "model": "mlp", "width": 4096, "depth": 4, "batch": 16384, "mode": "3xtf32"},
        # The convolution micro-benchmark layer.
        {"name": "conv_64to128", "kind": "conv", "n": 256, "ci": 64, "h": 32, "w": 32, "co": 128, "k": 3, "stride": 1, "pad": 1,
         "mode": "3xtf32"},
        # A strided layer with channel counts that are no multiples of 32 and an odd image.
        {"name": "conv_strided_ragged", "kind": "conv", "n": 64, "ci": 48, "h": 57, "w": 57, "co": 80, "k": 3, "stride": 2, "pad": 1,
         "mode": "3xtf32"},
        # Row-wise operators on a vocabulary-sized activation, beyond the L2 cache.
        {"name": "rows_16384x1000", "kind": "rows", "rows": 16384, "width": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any of the programs above at any size of its range."""
    kind = rng.choice(["infer", "loop", "mlp", "epoch", "epoch", "bn", "lm", "lm", "conv", "conv", "rows"])
    mode = rng.choice(["3xtf32", "3xtf32", "3xtf32", "tf32"])
    if kind == "infer":
        return {"kind": "infer", "batch": _log_int(rng, 1, 64), "mode": mode}
    if kind == "loop":
        return {"kind": "loop", "model": "digits", "batch": _log_int(rng, 8, 256), "mode": rng.choice([mode, "fp32"])}
    if kind == "mlp":
        return {"kind": "loop", "model": "mlp", "width": rng.choice([512, 1000, 1536, 2048, 3072]), "depth": rng.choice([2, 3, 4]),
                "batch": _log_int(rng, 256, 16384), "mode": mode}
    if kind == "epoch":
        if rng.random() < 0.4:
            return {"kind": "epoch", "model": "small_cnn", "batch": _log_int(rng, 16, 512), "steps": 16, "mode": mode}
        b = _log_int(rng, 32, 1024)
        return {"kind": "epoch", "model": "vgg", "batch": b, "steps": 12 if b < 256 else 6, "mode": mode}
    if kind == "bn":
        return {"kind": "epoch", "model": "vgg_bn", "batch": _log_int(rng, 32, 512), "steps": 6, "mode": mode}
    if kind == "lm":
        d, dh = rng.choice([128, 256, 512]), rng.choice([16, 32, 64])
        seq = _log_int(rng, 16, 512)
        return {"kind": "epoch", "model": "lm", "batch": max(1, _log_int(rng, 512, 8192) // seq), "seq": seq, "d_model": d,
                "heads": d // dh, "steps": 8, "mode": mode}
    if kind == "conv":
        k = rng.choice([1, 3, 3, 3, 5])
        ci, co = rng.choice([3, 16, 32, 48, 64, 96, 128, 200, 256]), rng.choice([16, 32, 64, 80, 96, 128, 200, 256])
        hw = _log_int(rng, 7, 64)
        most = 4.0e10 / (2.0 * ci * co * k * k * hw * hw)          # at most about the micro-benchmark layer's work
        return {"kind": "conv", "n": max(1, min(256, int(most * rng.uniform(0.2, 1.0)))), "ci": ci, "h": hw,
                "w": max(7, hw - rng.choice([0, 0, 1, 3])), "co": co, "k": k, "stride": rng.choice([1, 1, 1, 2]), "pad": k // 2,
                "mode": rng.choice([mode, mode, mode, "fp32"])}
    width = _log_int(rng, 17, 4096)
    return {"kind": "rows", "rows": min(131072, max(1, _log_int(rng, 1 << 14, 1 << 24) // width)), "width": width}


# ------------------------------------------------------------------------------------------------ models

def _model(case):
    if case["model"] == "digits":
        return DIGITS_CNN
    if case["model"] == "small_cnn":
        return workloads.SMALL_CNN
    if case["model"] == "vgg":
        return workloads.VGG_CIFAR
    if case["model"] == "vgg_bn":
        return workloads.VGG_CIFAR_BN
    if case["model"] == "lm":
        d, s = case["d_model"], case["seq"]
        block = ("transformer_block", d, case["heads"], 4 * d, workloads.ACT_GELU, 1)
        return dict(in_shape=(s,), classes=1000, vocab=1000, layers=[("embedding", 1000, d, s), block, block, ("linear", d, 1000)])
    width, layers = case["width"], []
    for _ in range(case["depth"]):
        layers += [("linear", width, width), ("gelu",)]
    return dict(in_shape=(width,), classes=1000, layers=layers + [("linear", width, 1000)])


def _init(layers, gen):
    """The parameters of workloads.he_init drawn on the device (same order, shapes and spreads; biases small, not zero,
    and of order one in front of a batchnorm layer, which takes them out again)."""
    def randn(shape, std):
        return (torch.randn(shape, device="cuda", generator=gen) * std).cpu().numpy()
    out = []
    for i, ly in enumerate(layers):
        bias = 0.5 if i + 1 < len(layers) and layers[i + 1][0] == "batchnorm" else 0.05
        if ly[0] == "conv":
            out += [randn((ly[2], ly[1], ly[3], ly[3]), math.sqrt(2.0 / (ly[1] * ly[3] * ly[3]))), randn((ly[2],), bias)]
        elif ly[0] == "linear":
            out += [randn((ly[1], ly[2]), math.sqrt(2.0 / ly[1])), randn((ly[2],), bias)]
        elif ly[0] == "batchnorm":
            out += [1.0 + randn((ly[1],), 0.05), randn((ly[1],), 0.05)]
        elif ly[0] == "embedding":
            out.append(randn((ly[1], ly[2]), 0.5))
        elif ly[0] == "transformer_block":
            d, ff = ly[1], ly[3]
            out += [randn((d, d), 1 / math.sqrt(d)) for _ in range(4)]
            out += [1.0 + randn((d,), 0.05), randn((d,), 0.05), 1.0 + randn((d,), 0.05), randn((d,), 0.05)]
            out += [randn((d, ff), 1 / math.sqrt(d)), randn((ff,), 0.05), randn((ff, d), 1 / math.sqrt(ff)), randn((d,), 0.05)]
    return out


def _layer_work(case):
    """(flops of a forward pass, flops of a training step, parameter count) of a model at the case's batch."""
    m = _model(case)
    b, shp, fwd, step, params, first = case["batch"], list(m["in_shape"]), 0.0, 0.0, 0, True
    for ly in m["layers"]:
        f = 0.0
        if ly[0] == "conv":
            _, ci, co, k, s, p = ly
            shp = [co, (shp[1] + 2 * p - k) // s + 1, (shp[2] + 2 * p - k) // s + 1]
            f = 2.0 * b * shp[1] * shp[2] * co * ci * k * k
            params += co * ci * k * k + co
        elif ly[0] == "maxpool":
            shp = [shp[0], (shp[1] - ly[1]) // ly[2] + 1, (shp[2] - ly[1]) // ly[2] + 1]
        elif ly[0] == "flatten":
            shp = [int(np.prod(shp))]
        elif ly[0] == "linear":
            f = 2.0 * b * ly[1] * ly[2] * (shp[0] if len(shp) == 2 else 1)
            shp = shp[:-1] + [ly[2]]
            params += ly[1] * ly[2] + ly[2]
        elif ly[0] == "batchnorm":
            params += 2 * ly[1]
        elif ly[0] == "embedding":
            shp, params, first = [shp[0], ly[2]], params + ly[1] * ly[2], False
        elif ly[0] == "transformer_block":
            d, ff, t = ly[1], ly[3], b * shp[0]
            f = 2.0 * t * (4 * d * d + 2 * d * ff) + 2.0 * t * shp[0] * d      # the causal half of the two S x S products
            params += 4 * d * d + 2 * d * ff + ff + 5 * d
        fwd += f
        step += f * (2 if first and f else 3)
        first = first and not f
    return fwd, step, params


# ------------------------------------------------------------------------------------------------ plumbing

class _Context(cuda.Context):
    """A context on the caller's stream, closed when the last thing made in it is gone."""
    _stream = None

    def __init__(self, mode):
        super().__init__(torch.cuda.current_device())
        if _Context._stream is None:
            _Context._stream = torch.cuda.Stream()
        self.set_stream(_Context._stream.cuda_stream)
        self.set_math_mode(MODES[mode])

    def __del__(self):
        self.close()


class _Buffer:
    """A node's device memory as something torch can wrap; keeps the node alive."""

    def __init__(self, node, ptr):
        self.node = node
        self.__cuda_array_interface__ = {"shape": tuple(node.shape), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _view(node, ptr):
    return torch.as_tensor(_Buffer(node, ptr), device="cuda")


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def _inputs(case, m, gen, batch):
    """Samples as the data sets give them: pixels in [0, 1) for digits, normalised (N(0, 1)) otherwise."""
    shape = (batch,) + tuple(m["in_shape"])
    make = torch.rand if m["in_shape"][0] == 1 and len(m["in_shape"]) == 3 else torch.randn
    return make(shape, device="cuda", generator=gen)


def _labels(gen, count, classes):
    return torch.randint(0, classes, (count,), device="cuda", generator=gen)


def _one_hot(labels, classes):
    return torch.nn.functional.one_hot(labels, classes).float()


def _forward(m, params, x):
    """The model through the node API, operator by operator as the reference's programs call it; GELU layers through
    the fused linear operator."""
    h, i, layers = x, 0, m["layers"]
    for k, ly in enumerate(layers):
        if ly[0] == "conv":
            h = cuda.nn.conv2d(h, params[i], params[i + 1], ly[4], ly[5])
            i += 2
        elif ly[0] == "linear":
            if k + 1 < len(layers) and layers[k + 1][0] == "gelu":
                h = cuda.nn.linear_act(h, params[i], params[i + 1], _lib.ACT_GELU)
            else:
                h = cuda.nn.Linear(params[i], params[i + 1]).forward(h)
            i += 2
        elif ly[0] == "relu":
            h = cuda.graph.relu(h)
        elif ly[0] == "maxpool":
            h = cuda.nn.maxpool2d(h, ly[1], ly[2])
        elif ly[0] == "flatten":
            h = cuda.nn.flatten(h)
    return h


# ------------------------------------------------------------------------------------------------ prepare

def prepare(case, seed):
    gen = _gen(seed)
    state = {"infer": _prepare_nodes, "loop": _prepare_nodes, "epoch": _prepare_epoch, "conv": _prepare_conv,
             "rows": _prepare_rows}[case["kind"]](case, gen)
    torch.cuda.synchronize()          # inputs are made on torch's own stream
    state["case"] = case
    return state


def _prepare_nodes(case, gen):
    m = workloads.SMALL_CNN if case["kind"] == "infer" else _model(case)
    ctx = _Context(case["mode"])
    params = [cuda.Node.new(p, p.shape, ctx=ctx) for p in _init(m["layers"], gen)]
    for p in params:
        cuda.runtime.to_cuda(p)
    x = _inputs(case, m, gen, case["batch"]).cpu().numpy()
    gx = cuda.Node.new(x, x.shape, ctx=ctx)
    gx.requires_grad = False
    cuda.runtime.to_cuda(gx)
    state = {"ctx": ctx, "model": m, "params": params, "x": x, "gx": gx}
    if case["kind"] == "infer":
        for p in params:
            p.requires_grad = False
        return state
    t = _one_hot(_labels(gen, case["batch"], m["classes"]), m["classes"]).cpu().numpy()
    gt = cuda.Node.new(t, t.shape, ctx=ctx)
    cuda.runtime.to_cuda(gt)
    cuda.runtime.flatten_params(params)          # one optimizer launch; the pointers below stay put
    ctx.sync()
    hp = workloads.ADAMW_HP
    state.update(t=t, gt=gt, resident=case["model"] == "mlp",
                 opt=cuda.optim.AdamW(1e-4, hp["beta1"], hp["beta2"], hp["eps"], hp["wd"], ctx=ctx),
                 views=[(_view(p, p.data_ptr()), _view(p, p.grad_ptr())) for p in params])
    return state


def _prepare_epoch(case, gen):
    m, batch = _model(case), case["batch"]
    ctx = _Context(case["mode"])
    hp = workloads.ADAMW_HP
    tr = cuda.Trainer(m["layers"], m["in_shape"], m["classes"], 1e-4, hp["beta1"], hp["beta2"], hp["eps"], hp["wd"], fuse=True, ctx=ctx)
    tr.set_params(_init(m["layers"], gen))
    batches = []
    for _ in range(min(4, case["steps"])):       # the epoch walks over four different host batches
        if case["model"] == "lm":
            ids = torch.randint(0, m["vocab"], (batch, case["seq"]), device="cuda", generator=gen, dtype=torch.int32)
            batches.append((_pinned(ids), _pinned(ids.roll(-1, 1).reshape(-1))))
        elif case["model"] == "vgg_bn":          # class indices and augmentation on the device
            batches.append((_pinned(_inputs(case, m, gen, batch)), _pinned(_labels(gen, batch, m["classes"]).int())))
        else:
            batches.append((_pinned(_inputs(case, m, gen, batch)), _pinned(_one_hot(_labels(gen, batch, m["classes"]), m["classes"]))))
    if case["model"] == "vgg_bn":
        tr.set_augment(4, True)
    return {"ctx": ctx, "trainer": tr, "batches": batches}


def _prepare_conv(case, gen):
    n, ci, h, w, co, k, s, p = (case[key] for key in ("n", "ci", "h", "w", "co", "k", "stride", "pad"))
    oh, ow = (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1
    randn = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)  # noqa: E731
    x, dy = randn(n, ci, h, w), randn(n, co, oh, ow)
    wt, b = randn(co, ci, k, k) * math.sqrt(2.0 / (ci * k * k)), randn(co) * 0.05
    return {"ctx": _Context(case["mode"]), "x": x, "dy": dy, "w": wt, "b": b, "y": torch.empty_like(dy), "dx": torch.empty_like(x),
            "dw": torch.empty_like(wt), "db": torch.empty_like(b), "dims": (n, ci, h, w, co, k, k, s, p)}


def _prepare_rows(case, gen):
    r, f = case["rows"], case["width"]
    randn = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)  # noqa: E731
    s = {"ctx": _Context("3xtf32"), "a": randn(r, f), "b": randn(r, f), "g": randn(r, f), "gamma": 1 + 0.1 * randn(f), "beta": 0.1 * randn(f),
         "target": _one_hot(_labels(gen, r, f), f)}
    for key in ("y", "xhat", "da", "db", "p", "dp", "dlogits"):
        s[key] = torch.empty(r, f, device="cuda")
    s["istd"], s["loss"] = torch.empty(r, device="cuda"), torch.empty(1, device="cuda")
    s["dgamma"], s["dbeta"] = torch.empty(f, device="cuda"), torch.empty(f, device="cuda")
    return s


# ------------------------------------------------------------------------------------------------ run

def run(state):
    return {"infer": _run_infer, "loop": _run_loop, "epoch": _run_epoch, "conv": _run_conv, "rows": _run_rows}[state["case"]["kind"]](state)


def _run_infer(s):
    s["gx"].set_data(s["x"])                     # a new request's pixels
    cuda.runtime.to_cuda(s["gx"])
    return cuda.runtime.to_host(_forward(s["model"], s["params"], s["gx"]))


def _run_loop(s):
    params, gx, gt = s["params"], s["gx"], s["gt"]
    if not s["resident"]:                        # the data set's next batch comes from the host
        gx.set_data(s["x"])
        cuda.runtime.to_cuda(gx)
        gt.set_data(s["t"])
        cuda.runtime.to_cuda(gt)
    cuda.runtime.zero_grad(params)
    logits = _forward(s["model"], params, gx)
    loss = cuda.loss.cross_entropy(logits, gt)
    cuda.loss.cross_entropy_backward(logits, gt)
    cuda.backward_graph(logits)
    s["opt"].step(params)
    return {"loss": loss, "params": [v[0] for v in s["views"]], "grads": [v[1] for v in s["views"]]}


def _stage(s, i):
    tr, (x, t) = s["trainer"], s["batches"][i % len(s["batches"])]
    model = s["case"]["model"]
    if model == "lm":
        tr.stage_next_tokens_ptr(x.ctypes.data, t.ctypes.data, s["case"]["batch"])
    elif model == "vgg_bn":
        tr.stage_next_indexed(x, t)
    else:
        tr.stage_next(x, t)


def _run_epoch(s):
    tr, steps, losses = s["trainer"], s["case"]["steps"], []
    _stage(s, 0)
    for i in range(steps):
        if i + 1 < steps:
            _stage(s, i + 1)                     # its copy overlaps this step
        loss = tr.step_staged_lagged()
        if i > 0:
            losses.append(loss)
    losses.append(tr.last_loss())
    return {"losses": np.array(losses, np.float32), "params": [tr.get_param(i) for i in range(tr.n_params)],
            "buffers": [tr.get_buffer(i) for i in range(tr.n_buffers)]}


def _p(t):
    return VP(t.data_ptr())


def _run_conv(s):
    ctx, d = s["ctx"], s["dims"]
    lib, x, w, dy = ctx._l, _p(s["x"]), _p(s["w"]), _p(s["dy"])
    # x is read by the forward pass and by the weight gradient
    check(ctx.h, lib.nrs_planes_cache(ctx.h, x, *d[:4]))
    check(ctx.h, lib.nrs_conv2d_fwd(ctx.h, x, w, _p(s["b"]), _p(s["y"]), *d, _lib.ACT_NONE))
    check(ctx.h, lib.nrs_conv2d_bwd(ctx.h, x, w, dy, _p(s["dx"]), _p(s["dw"]), _p(s["db"]), *d, 0))
    check(ctx.h, lib.nrs_planes_drop(ctx.h, x))
    return [s["y"], s["dx"], s["dw"], s["db"]]


def _run_rows(s):
    ctx, r, f = s["ctx"], s["case"]["rows"], s["case"]["width"]
    lib, h = ctx._l, ctx.h
    a, b, g, gamma = _p(s["a"]), _p(s["b"]), _p(s["g"]), _p(s["gamma"])
    y, xhat, istd, p = _p(s["y"]), _p(s["xhat"]), _p(s["istd"]), _p(s["p"])
    check(h, lib.nrs_layernorm_residual_fwd(h, a, b, gamma, _p(s["beta"]), y, xhat, istd, r, f, C.c_float(1e-5)))
    check(h, lib.nrs_softmax_fwd(h, y, p, r, f))
    check(h, lib.nrs_ce_fwd_bwd(h, y, _p(s["target"]), _p(s["loss"]), _p(s["dlogits"]), r, f, r))
    check(h, lib.nrs_softmax_bwd(h, p, g, _p(s["dp"]), r, f, 0))
    check(h, lib.nrs_layernorm_residual_bwd(h, g, xhat, istd, gamma, _p(s["da"]), _p(s["db"]), _p(s["dgamma"]), _p(s["dbeta"]),
                                            r, f, 0, 0, 0))
    return [s[key] for key in ("y", "xhat", "istd", "p", "loss", "dlogits", "dp", "da", "db", "dgamma", "dbeta")]


# ------------------------------------------------------------------------------------------------ work and tolerance

def work(case):
    """Bytes and flops of one pass that no implementation can do without."""
    if case["kind"] == "infer":
        m = dict(case, model="small_cnn")
        fwd, _, params = _layer_work(m)
        return {"bytes": 4.0 * (params + case["batch"] * 784 + case["batch"] * 10), "flops": fwd}
    if case["kind"] in ("loop", "epoch"):
        m = _model(case)
        _, step, params = _layer_work(case)
        rows = case["batch"] * (case["seq"] if case["model"] == "lm" else 1)
        targets = rows * (1 if case["model"] in ("lm", "vgg_bn") else m["classes"])
        # inputs and targets once; parameters and both moments read and written, gradients written and read
        per_step = 4.0 * (case["batch"] * int(np.prod(m["in_shape"])) + targets) + 32.0 * params
        n = case.get("steps", 1)
        return {"bytes": n * per_step + (4.0 * params if case["kind"] == "epoch" else 0.0), "flops": n * step}
    if case["kind"] == "conv":
        n, ci, h, w, co, k, s, p = (case[key] for key in ("n", "ci", "h", "w", "co", "k", "stride", "pad"))
        pix = n * ((h + 2 * p - k) // s + 1) * ((w + 2 * p - k) // s + 1)
        return {"bytes": 4.0 * (2 * n * ci * h * w + 2 * pix * co + 2 * co * ci * k * k + 2 * co), "flops": 6.0 * pix * co * ci * k * k}
    r, f = case["rows"], case["width"]
    return {"bytes": 4.0 * (11 * r * f + r + 4 * f + 1), "flops": 40.0 * r * f}


def tolerance(case):
    if case["kind"] == "rows":
        # f32 arithmetic and sums over a row or a column
        return {"rel": 2e-5, "max": 1e-3}
    tf32 = case["mode"] == "tf32"
    if case["kind"] in ("infer", "conv"):
        # One chain of contractions.  3xTF32 and f32 sums: some 1e-5 on the longest reductions.  TF32 inputs carry 11 bits.
        return {"rel": 2e-3, "max": 5e-2} if tf32 else {"rel": 5e-5, "max": 2e-3}
    # Training steps.  Where a pre-activation within rounding error of zero falls on the other side of its ReLU, or of its
    # pooling winner, a gradient moves by far more than the arithmetic's own error, and AdamW then moves a weight whose
    # gradient is about zero by a different fraction of the learning rate (the biases in front of a batchnorm layer, whose
    # gradient is zero up to rounding, among them).  Measured between f32 and 3xTF32 contractions over two passes:
    # 8e-6 for the language models, 2e-4 for the MLP and the small CNN, 2e-3 for the deep CNN, 7e-3 with batchnorm.
    if tf32 or case["model"] == "vgg_bn":
        return {"rel": 1.5e-2, "max": 0.5}
    if case["model"] == "vgg":
        return {"rel": 5e-3, "max": 0.3}
    return {"rel": 1e-4, "max": 2e-2} if case["model"] == "lm" else {"rel": 1e-3, "max": 5e-2}
