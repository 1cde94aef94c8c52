"""Performance cases of the DenseBlock / FeedForwardNetwork path: training steps and forward passes through the
public API (`GpuContext`, `DenseBlock`, `FeedForwardNetwork`), over the sizes, precisions and options it is used at.

A case is a dict:
  kind      "train" (forward, backward and optimiser step) or "infer" (forward of an inference-mode network)
  dims      layer widths, "784-128-64-10"
  batch     rows per pass
  dtype     f32, f16, bf16, or f32tc (f32 with the tensor-core option of the context switched on)
  norm, act normalisation (none / rms / layer / batch) and activation of the hidden blocks
  loss      ce (softmax + cross-entropy), mse, mse_sigmoid, bce (sigmoid + binary cross-entropy)
  optim     adam, sgd, nesterov
  dropout   probability in the hidden blocks
  graph     the step is bracketed by `ctx.step_graph()`, as launch-bound programs do

Networks are drawn as they look in the middle of a training run: nonzero biases, moments of the size of the
gradients, a step counter of 1000. (At step 1 Adam moves a weight by lr * sign(gradient), which no two correct
implementations agree on where the gradient is rounding noise.)
"""
from __future__ import annotations

import math

import torch

from soklyn_b200 import core, device, ffn, function, mlp
from soklyn_b200.context import LayerInitConfig, LossConfig, MultiLayerTrainContext

_PREC = {"f32": function.Precision.FP32, "f32tc": function.Precision.FP32, "f16": function.Precision.FP16,
         "bf16": function.Precision.BF16}
_NORM = {"none": function.Normalisation.Disabled, "rms": function.Normalisation.RMSNorm,
         "layer": function.Normalisation.LayerNorm, "batch": function.Normalisation.BatchNorm}
_ACT = {"relu": function.Activation.ReLU, "leaky": function.Activation.LeakyReLU(0.1), "tanh": function.Activation.Tanh,
        "silu": function.Activation.SiLU, "mish": function.Activation.Mish, "sigmoid": function.Activation.Sigmoid}
_LOSS = {"ce": (function.LossFunc.CrossEntropyLoss, function.Activation.Softmax),
         "mse": (function.LossFunc.MeanSquareLoss, function.Activation.Identity),
         "mse_sigmoid": (function.LossFunc.MeanSquareLoss, function.Activation.Sigmoid),
         "bce": (function.LossFunc.BinaryCrossEntropy, function.Activation.Sigmoid)}
_OPTIM = {"adam": function.Optimiser.Adam(0.9, 0.999, 1e-8), "sgd": function.Optimiser.SGD(0.0, False),
          "nesterov": function.Optimiser.SGD(0.9, True)}
_STEP, _ID_STEP, _LOSS_SCALE = 1000, 1000, 512.0   # steps taken before the first pass; tensor ids between blocks; scale of the deltas


def _case(kind, dims, batch, dtype, norm, act, loss="mse", optim="adam", lr=1e-4, dropout=0.0, graph=False, **name):
    return dict(name, kind=kind, dims=dims, batch=batch, dtype=dtype, norm=norm, act=act, loss=loss, optim=optim, lr=lr,
                dropout=dropout, graph=graph)


def listed():
    return [
        # the smallest training step: an f32 digit classifier, a dozen kernels of microseconds, launches and latency
        _case("train", "784-128-64-10", 64, "f32", "none", "relu", "ce", "sgd", 1e-2, graph=True, name="mlp_f32_b64"),
        # autoencoder on images in mixed precision, few tiles per product
        _case("train", "784-256-64-256-784", 256, "f16", "none", "silu", "mse_sigmoid", "adam", 1e-3, graph=True,
              name="autoencoder_f16_b256"),
        # image classifier: LayerNorm + Mish + dropout, long products with few output tiles and a 10-wide head
        _case("train", "3072-1024-512-10", 512, "f16", "layer", "mish", "ce", "adam", 1e-3, dropout=0.1, graph=True,
              name="classifier_f16_b512"),
        # widths and batch that fit no tile and no 16-byte row pitch, stepped kernel by kernel
        _case("train", "777-1001-333-10", 300, "bf16", "none", "silu", "ce", "nesterov", 1e-3, name="ragged_bf16_b300"),
        # batch normalisation (column statistics), many rows
        _case("train", "3072-1024-1024-10", 4096, "f16", "batch", "tanh", "ce", "nesterov", 1e-3, name="batchnorm_f16_b4096"),
        # tall and narrow: the weight gradient sums over 65536 rows into few tiles, epilogues dominate the rest
        _case("train", "1024-1024-1024", 65536, "f16", "none", "tanh", "mse", "adam", 1e-4, name="tall_f16_b65536"),
        # the wide network at one GPU's share of an eight-way batch split
        _case("train", "4096-16384-4096-16384-4096", 1024, "bf16", "rms", "silu", "mse", "adam", 1e-4, name="wide_bf16_b1024"),
        # the wide network at the full batch: the flagship training step
        _case("train", "4096-16384-4096-16384-4096", 8192, "f16", "rms", "silu", "mse", "adam", 1e-4, name="wide_f16_b8192"),
        # f32 training on the FFMA kernels
        _case("train", "1024-4096-1024", 4096, "f32", "rms", "silu", "mse", "adam", 1e-4, name="blocks_f32_b4096"),
        # the same precision class through the tensor-core option
        _case("train", "4096-4096-4096", 4096, "f32tc", "rms", "silu", "mse", "adam", 1e-4, name="blocks_f32tc_b4096"),
        # serving a handful of requests: the weights are read once for 16 rows
        _case("infer", "4096-16384-4096-16384-4096", 16, "f16", "rms", "silu", name="serve_wide_f16_b16"),
        # evaluation of a classifier over a large batch
        _case("infer", "3072-1024-512-10", 8192, "f16", "layer", "mish", name="evaluate_f16_b8192"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    w = _log(rng, lo, hi)
    return max(lo, w - w % 8) if rng.random() < 0.6 else w   # most widths are whole 16-byte rows, some are odd


def draw(rng):
    while True:
        kind = "infer" if rng.random() < 0.25 else "train"
        dtype = rng.choice(["f16", "f16", "bf16", "f32", "f32tc"])
        loss = rng.choice(["ce", "mse", "mse", "mse_sigmoid", "bce"])
        dims = [_width(rng, 64, 8192)] + [_width(rng, 64, 16384) for _ in range(rng.choice([1, 1, 2, 3]))]
        dims.append(rng.choice([10, 10, 100]) if loss == "ce" else _width(rng, 32, 4096))
        batch = _log(rng, 1 if kind == "infer" else 16, 65536)
        norm = rng.choice(["none", "rms", "layer", "batch"])
        if norm == "batch" and batch < 2:
            continue
        optim = rng.choice(["adam", "adam", "sgd", "nesterov"])
        dropout = 0.1 if kind == "train" and rng.random() < 0.3 else 0.0
        acts = ["tanh", "silu", "silu", "mish", "sigmoid"]
        if kind == "infer" or (dtype == "f32" and sum(dims) * batch <= 100000):
            acts += ["relu", "leaky"]   # not where rounding moves some inputs across the kink and flips their derivative
        act = rng.choice(acts)
        graph = kind == "train" and dtype != "f32tc" and rng.random() < 0.4
        case = _case(kind, "-".join(map(str, dims)), batch, dtype, norm, act, loss, optim, 1e-4, dropout, graph)
        need = work(case)
        # no larger than the largest listed case of its precision; odd 16-bit widths may run off the tensor cores
        odd = any(d % 8 for d in dims)
        most = 1e12 if dtype == "f32tc" else 2e11 if dtype == "f32" or odd else 6e12
        if need["flops"] <= most and need["bytes"] <= 8e9 and sum(dims) * batch <= 2.5e8:
            return case


def _dims(case):
    return [int(d) for d in case["dims"].split("-")]


def _inputs(case, seed):
    """What a program has in hand, as plain tensors: the parameters and moments of each block, the input and the target."""
    dims, batch, train = _dims(case), case["batch"], case["kind"] == "train"
    dev, dtype = torch.device("cuda", 0), core.TORCH_DTYPE[_PREC[case["dtype"]]]
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)

    def randn(*shape):
        return torch.randn(shape, generator=gen, device=dev)

    def params(w, b, scale):
        """w, b and, for training, dv_w, dv_b, dm_w, dm_b of the size of the gradients."""
        first = lambda t: randn(*t.shape).mul_(0.1 * scale)
        second = lambda t: torch.rand(t.shape, generator=gen, device=dev).add_(0.5).mul_(scale * scale)
        dv = second if case["optim"] == "adam" else first
        w, b = w.to(dtype), b.to(dtype)
        return [w, b, dv(w), dv(b), first(w), first(b)] if train else [w, b, None, None, None, None]

    blocks = []
    for k, n in zip(dims[:-1], dims[1:]):
        linear = params(randn(k, n).mul_(math.sqrt(1.5 / k)), randn(1, n).mul_(0.05), 0.5 / math.sqrt(batch))
        norm = params(randn(1, n).mul_(0.1).add_(1.0), randn(1, n).mul_(0.05), 0.5 / math.sqrt(batch))
        blocks.append((linear, norm))

    if case["loss"] in ("ce", "bce", "mse_sigmoid") and case["norm"] == "none":   # pixels
        x = torch.randint(0, 256, (batch, dims[0]), generator=gen, device=dev).float().div_(255.0)
    else:
        x = randn(batch, dims[0])
    if case["loss"] == "ce":
        t = torch.nn.functional.one_hot(torch.randint(0, dims[-1], (batch,), generator=gen, device=dev), dims[-1]).float()
    elif case["loss"] == "mse":
        t = randn(batch, dims[-1])
    else:
        t = torch.rand(batch, dims[-1], generator=gen, device=dev)
    return blocks, x.to(dtype), t.to(dtype)


def prepare(case, seed):
    dims, batch, prec, train = _dims(case), case["batch"], _PREC[case["dtype"]], case["kind"] == "train"
    blocks, x, t = _inputs(case, seed)
    ctx = device.GpuContext(16, 0)
    f32 = function.Precision.FP32

    def state(w, b, *moments):
        params = [core.Tensor(w, prec), core.Tensor(b, prec)]
        masters = [core.Tensor(p.float(), f32) if prec != f32 else None for p in (w, b)]
        return mlp.ParamState(*params, *masters, *(core.Tensor(m, f32) if train else None for m in moments))

    layers = []
    for i, (linear, norm) in enumerate(blocks):
        hidden = i + 2 < len(dims)
        core.reset_tensor_ids(_ID_STEP * i)   # a block's first id, its weights', seeds its dropout masks
        config = LayerInitConfig(_NORM[case["norm"]] if hidden else function.Normalisation.Disabled,
                                 _ACT[case["act"]] if hidden else function.Activation.Identity,
                                 function.Regularisation.none(), case["dropout"] if hidden else 0.0)
        layers.append(mlp.DenseBlock.from_tensors(ctx, train, state(*linear), state(*norm), batch, config, prec))
    net = ffn.FeedForwardNetwork(layers, dims[0])
    data = [core.Tensor(d, prec, take_id=False) for d in (x, t)]

    if case["dtype"] == "f32tc":
        # three bf16 parts per operand of the largest product
        ctx.reserve(6 * max(batch * k + k * n + batch * n for k, n in zip(dims[:-1], dims[1:])) + (1 << 20))
        ctx.set_f32_tensor_cores(True)
    optims = [_OPTIM[case["optim"]]] * len(layers)
    return {"ctx": ctx, "net": net, "x": data[0], "t": data[1], "case": case, "step": _STEP,
            "loss": LossConfig(*_LOSS[case["loss"]]), "train": MultiLayerTrainContext(optims, optims, batch, case["lr"])}


def _step(s):
    case, ctx, net = s["case"], s["ctx"], s["net"]
    outs = net.forward(ctx, s["x"], case["batch"], case["dropout"] > 0, s["step"])
    net.backward(ctx, outs, s["t"], s["x"], s["loss"], s["train"], s["step"])


def run(state):
    case, ctx, net = state["case"], state["ctx"], state["net"]
    if case["kind"] == "infer":
        net.forward(ctx, state["x"], case["batch"], False, 0)
        return [[t.data for t in (l.get_outputs(), l.get_predrop_outputs(), l.get_preact_outputs()) +
                 ((l.get_prenorm_outputs(), l.get_centered_outputs()) if l.get_normalisation().ordinal() else ())]
                for l in net.get_layers()]
    state["step"] += 1
    if case["graph"]:
        with ctx.step_graph():
            _step(state)
    else:
        _step(state)
    got = []
    for l in net.get_layers():
        of = [l.get_outputs(), l.get_preact_outputs(), l.get_grads(), l.get_delta_prenorm_out(), l.get_weights(), l.get_biases(),
              l.get_dv_weights(), l.get_dv_biases()]
        if case["optim"] == "adam":
            of += [l.get_dm_weights(), l.get_dm_biases()]
        if l.get_master_weights() is not None:
            of += [l.get_master_weights()]
        if l.get_normalisation().ordinal():
            of += [l.get_norm_weights(), l.get_dv_norm_weights(), l.get_norm_weights_grad()]
        if l.get_mask_coeff() > 0:
            of += [l.get_masks()]
        got.append([t.data for t in of])
    return got


def _f32(v):
    return float(torch.tensor(v, dtype=torch.float32))


def _activation(name, x):
    return {"relu": lambda: x.clamp_min(0.0), "leaky": lambda: torch.where(x > 0, x, _f32(0.1) * x), "tanh": lambda: x.tanh(),
            "silu": lambda: x * x.sigmoid(), "mish": lambda: x * torch.nn.functional.softplus(x).tanh(),
            "sigmoid": lambda: x.sigmoid(), "identity": lambda: x}[name]()


def _slope(name, x):
    """Derivative of the activation at its input x."""
    if name in ("relu", "leaky"):
        return torch.where(x > 0, 1.0, 0.0 if name == "relu" else _f32(0.1)).double()
    sg = x.sigmoid()
    if name == "tanh":
        return 1.0 - x.tanh() ** 2
    if name == "silu":
        return sg * (1.0 + x * (1.0 - sg))
    if name == "mish":
        th = torch.nn.functional.softplus(x).tanh()
        return th + x * sg * (1.0 - th * th)
    return sg * (1.0 - sg) if name == "sigmoid" else torch.ones_like(x)


def _mask(case, block, shape, dev):
    """Inverted-dropout mask of the step from the integer hash of row, column, step and tensor id."""
    u = 0xFFFFFFFF
    h = ((_STEP + 1) * 1103515245 + _ID_STEP * block) & u
    h = ((h ^ (h >> 16)) * 1103515245) & u
    row = torch.arange(shape[0], dtype=torch.int64, device=dev)[:, None]
    col = torch.arange(shape[1], dtype=torch.int64, device=dev)[None, :]
    s = ((row * 1103515245) & u) ^ ((col * 0x4C957F2D) & u) ^ (((h ^ (h >> 15)) + row * 7) & u)
    s = ((s ^ (s >> 17)) * 1103515245 + 12345) & u
    keep = (s ^ (s >> 15)).float() * 2.0 ** -32 >= case["dropout"]
    return keep.double() / (1.0 - _f32(case["dropout"]))


def exact(case, seed):
    """The same pass in 64 bits, from the same parameters, moments and data, in plain torch."""
    need = work(case)
    if need["bytes"] > 5e9:   # 64-bit tensors of the wide networks would not fit beside the pass
        return None
    dims, m, train = _dims(case), case["batch"], case["kind"] == "train"
    blocks, x, t = _inputs(case, seed)
    blocks = [[[p if p is None else p.double() for p in of] for of in pair] for pair in blocks]
    x, t = x.double(), t.double()
    kept = []   # per block: input, centred or raw values before the normalisation, rstd, preact, predrop, mask, out
    for i, (linear, norm) in enumerate(blocks):
        w, b, nw, nb = linear[0], linear[1], norm[0], norm[1]
        hidden = i + 2 < len(dims)
        kind = case["norm"] if hidden else "none"
        z = x @ w + (0.0 if kind == "batch" else b)
        pre, cen, rstd = z, z, None
        if kind == "rms":
            rstd = (z.square().mean(1, keepdim=True) + 1e-6).rsqrt()
            pre = z * rstd * nw
        elif kind != "none":
            over = 1 if kind == "layer" else 0
            cen = z - z.mean(over, keepdim=True)
            rstd = (cen.square().mean(over, keepdim=True) + 1e-6).rsqrt()
            pre = cen * rstd * nw + nb
        drop = _activation(case["act"] if hidden else "identity", pre)
        mask = _mask(case, i, z.shape, z.device) if train and hidden and case["dropout"] else torch.ones((), dtype=z.dtype, device=z.device)
        out = drop * mask
        kept.append((x, z, cen, rstd, pre, drop, mask, out, kind, hidden))
        x = out
    if not train:
        return [[k[7], k[5], k[4]] + ([k[1], k[2]] if k[8] != "none" else []) for k in kept]

    lr, step = _f32(case["lr"]), _STEP + 1
    b1, b2, eps = (_f32(0.9), _f32(0.999), _f32(1e-8))

    def update(p, v, mo, g):
        """(parameter, dv, dm) after the optimiser step on the mean gradient g."""
        if case["optim"] == "adam":
            mo, v = b1 * mo + (1.0 - b1) * g, b2 * v + (1.0 - b2) * g * g
            return p - lr * (mo / (1.0 - b1 ** step)) / ((v / (1.0 - b2 ** step)).sqrt() + eps), v, mo
        mom = b1 if case["optim"] == "nesterov" else 0.0
        v = mom * v + g
        return p - lr * (g + mom * v if case["optim"] == "nesterov" else v), v, mo

    got = [None] * len(blocks)
    back = None   # gradient at the block's output, times the loss scale
    for i in reversed(range(len(blocks))):
        (w, b, vw, vb, mw, mb), (nw, nb, vnw, _, mnw, _) = blocks[i]
        x, z, cen, rstd, pre, drop, mask, out, kind, hidden = kept[i]
        if back is None:
            final = {"ce": "softmax", "mse": "identity", "mse_sigmoid": "sigmoid", "bce": "sigmoid"}[case["loss"]]
            o = out.softmax(1) if final == "softmax" else _activation(final, out)
            delta = o - t
            if case["loss"] == "mse_sigmoid":
                delta = delta * o * (1.0 - o)
            out = o if final == "softmax" else out
            dp = delta * _LOSS_SCALE
        else:
            delta = back * _slope(case["act"], pre) * mask
            dp = delta
        gnw = torch.zeros_like(z)
        if kind != "none":
            gnw = delta * cen * rstd
            over = dims[i + 1] if kind != "batch" else m
            # the element-wise form this path uses, not the full derivative of the normalisation
            dp = nw * rstd * (delta - (rstd * cen) ** 2 / over if kind == "rms"
                              else delta * (1.0 - 1.0 / over - (rstd * cen) ** 2 / over))
        scale = 1.0 / (_LOSS_SCALE * m)
        w, vw, mw = update(w, vw, mw, (x.T @ dp) * scale)
        if kind != "batch":
            b, vb, mb = update(b, vb, mb, dp.sum(0, keepdim=True) * scale)
        of = [out, pre, delta, dp, w, b, vw, vb]
        if case["optim"] == "adam":
            of += [mw, mb]
        if not case["dtype"].startswith("f32"):
            of += [w]
        if kind != "none":
            nw, vnw, mnw = update(nw, vnw, mnw, gnw.sum(0, keepdim=True) * scale)
            of += [nw, vnw, gnw]
        if hidden and case["dropout"]:
            of += [mask]
        got[i] = of
        back = dp @ w.T
    return got


def work(case):
    """Operations of the products; bytes of what a pass is given (inputs, targets, parameters and their optimiser
    state) and of what it leaves (the updated state and the cache and gradient tensors of the API)."""
    dims, m, train = _dims(case), case["batch"], case["kind"] == "train"
    s = 4 if case["dtype"].startswith("f32") else 2
    flops, nbytes = 0.0, float(m * dims[0] * s + (m * dims[-1] * s if train else 0))
    for i, (k, n) in enumerate(zip(dims[:-1], dims[1:])):
        hidden = i + 2 < len(dims)
        flops += 2.0 * m * k * n * (1 if not train else 2 if i == 0 else 3)
        normed = hidden and case["norm"] != "none"
        nbytes += m * n * s * (5 if normed else 3)
        nbytes += k * n * s
        if train:
            moments = 4 if case["optim"] == "adam" else 2
            nbytes += k * n * (4 * moments + (s + 8 if s == 2 else s))
            nbytes += m * n * (16 + (s if hidden and case["dropout"] else 0))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the path differs by from itself with the sums of its products in another order (FFMA
    against tensor cores): rel 2.5e-6 / 7e-4 / 3.8e-3 and max 3e-5 / 0.02 / 0.11 in f32 / f16 / bf16 at worst."""
    return {"f32": {"rel": 1e-5, "max": 2e-4}, "f32tc": {"rel": 1e-5, "max": 2e-4}, "f16": {"rel": 4e-3, "max": 0.1},
            "bf16": {"rel": 1.6e-2, "max": 0.5}}[case["dtype"]]
