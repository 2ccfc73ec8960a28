"""What the speed of this framework is measured on: calls that a user's program makes, over the range in which it makes them.

Every case is one pass through a public entry point: `Trainer.step`, `Trainer.replay` and `Trainer.fit_stream`
(ml_framework_b200/train.py), `Sequential.fit` and `Sequential.predict` and the hand-written training loop
(ml_framework_b200/seera.py), the tensor operators (ml_framework_b200/cuTen.py) and the operator entries of the binding.
Models and their sizes are the package's own training configurations (ml_framework_b200/workloads.py): a small CNN on
1x28x28 images, an MLP 784-1024-1024-10, a VGG-style CNN on 3x32x32 images, a convolutional autoencoder on 1x64x64 images.

A case holds the kind of call, the model or operator sizes, and the batch.  The precision follows the use: captured steps run the
policy of `train.policy_for` (the one a benchmark or a long training run picks), eager loops, `fit` and `predict` run the
engine's default, the convolution operator runs either one bf16 pass or the default.
"""
import math
import random

import numpy as np
import torch

from ml_framework_b200 import seera as S
from ml_framework_b200 import seera_cuda as sc
from ml_framework_b200 import train
from ml_framework_b200 import workloads as wl
from ml_framework_b200.cuTen import cuten

DEFAULT_PRECISION = 3
#: Step size of the Adam configurations here, one of fine-tuning: one step's rounding does not grow over the next few.
ADAM_LR = 1e-5


def listed():
    return [
        # one image classified as it arrives: the smallest call, all latency
        {"name": "predict_cnn_1", "kind": "predict", "model": "c1", "batch": 1},
        # a test set classified in large batches, the last of them ragged
        {"name": "predict_vgg_777", "kind": "predict", "model": "c3", "batch": 777},
        # the training loop most scripts call: one epoch over host arrays, last batch ragged
        {"name": "fit_cnn_500_by_64", "kind": "fit", "model": "c1", "samples": 500, "batch": 64},
        # the step written out by hand, every launch enqueued from Python
        {"name": "step_vgg_100", "kind": "step", "model": "c3", "batch": 100},
        # the same with batch normalisation between the layers
        {"name": "step_batchnorm_128", "kind": "step_bn", "batch": 128},
        # long runs: the step recorded once and replayed, each configuration at its own batch
        {"name": "replay_cnn_64", "kind": "replay", "model": "c1", "batch": 64},
        {"name": "replay_mlp_4096", "kind": "replay", "model": "c2", "batch": 4096},
        {"name": "replay_vgg_512", "kind": "replay", "model": "c3", "batch": 512},
        {"name": "replay_autoencoder_256", "kind": "replay", "model": "c4", "batch": 256},
        # the same fed from page-locked host batches, the loss of every step read back
        {"name": "stream_mlp_1000", "kind": "stream", "model": "c2", "batch": 1000, "batches": 4},
        # the backward call of one convolution through the binding (dX and dW), one bf16 pass
        {"name": "conv_bwd_256x14_256", "kind": "conv_bwd", "batch": 256, "channels": 256, "filters": 256, "size": 14, "stride": 1,
         "precision": 1},
        # a dense layer composed from tensor operators, as scripts on the tensor class do
        {"name": "operators_1000x784x1024", "kind": "operators", "rows": 1000, "inner": 784, "cols": 1024},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


#: Batches in use for each model: from a handful of samples to the configuration's own batch, or above it where that is small.
_BATCHES = {"c1": (8, 1024), "c2": (32, 4096), "c3": (8, 512), "c4": (8, 256)}


def draw(rng: random.Random):
    kind = rng.choice(["predict", "fit", "step", "step_bn", "replay", "replay", "stream", "conv_bwd", "operators"])
    model = rng.choice(["c1", "c2", "c3", "c4"])
    lo, hi = _BATCHES[model]
    if kind == "predict":
        return {"kind": kind, "model": model, "batch": _log(rng, 1, 2 * hi)}
    if kind == "fit":
        return {"kind": kind, "model": "c1", "samples": rng.randint(200, 500), "batch": rng.randint(48, 128)}
    if kind == "step":
        return {"kind": kind, "model": model, "batch": _log(rng, lo, hi // 2)}
    if kind == "step_bn":
        return {"kind": kind, "batch": _log(rng, 16, 256)}
    if kind == "replay":
        return {"kind": kind, "model": model, "batch": _log(rng, lo, hi)}
    if kind == "stream":
        return {"kind": kind, "model": model, "batch": _log(rng, lo, hi // 4), "batches": rng.randint(2, 6)}
    if kind == "operators":
        return {"kind": kind, "rows": _log(rng, 16, 4096), "inner": _log(rng, 16, 2048), "cols": _log(rng, 17, 2048)}
    while True:
        case = {"kind": kind, "batch": _log(rng, 1, 256), "channels": _log(rng, 8, 512), "filters": _log(rng, 8, 512),
                "size": rng.randint(7, 56), "stride": rng.choice([1, 1, 1, 2]), "precision": rng.choice([1, 1, DEFAULT_PRECISION])}
        n_elems = case["batch"] * max(case["channels"], case["filters"]) * case["size"] ** 2
        if n_elems <= 256 * 64 * 56 * 56 and work(case)["flops"] <= (1.2e11 if case["precision"] == 1 else 2e10):
            return case


# ---- states -------------------------------------------------------------------------------------------------------------------
class _Block:
    """A device tensor of the engine, for torch: shares the memory and keeps its owner alive."""

    def __init__(self, t):
        self.owner = t
        self.__cuda_array_interface__ = {"shape": tuple(t.shape), "typestr": "<i4" if t.dtype == "int32" else "<f4",
                                         "data": (int(t.main_ptr), False), "version": 3, "strides": None, "stream": None}


def _view(t):
    return torch.as_tensor(_Block(t), device="cuda")


class _State:
    """What the program keeps between calls; gives recorded steps and page-locked buffers back at its end."""
    trainer, pinned = None, ()

    def __del__(self):
        if self.trainer is not None:
            self.trainer.release_graph()
        for buffers in self.pinned:
            for p in buffers:
                sc.host_free_pinned(p)


def _workload(model):
    work = wl.WORKLOADS[model]()
    if work.opt["kind"] == "adam":
        work.opt = {"kind": "adam", "lr": ADAM_LR}
    return work


def _kept(model, opt):
    """The buffers that a step leaves updated: every gradient, the weights, the optimizer's moments."""
    out = {"grad_%02d" % i: _view(t._grad_slot) for i, t in enumerate(model.parameters())}
    out["weights"] = _view(model.params)
    if isinstance(opt, S.Adam):
        out["m"], out["v"] = _view(opt.m), _view(opt.v)
    else:
        out["velocity"] = _view(opt.velocity)
    return out


def _trainer(s, case, seed, precision):
    work = _workload(case["model"])
    s.trainer = train.Trainer(work, seed=seed, precision=precision)
    X, Y = work.batch(case["batch"], seed)
    s.x, s.y = S.Tensor(X, is_leaf=True), S.Tensor(Y, is_leaf=True)
    s.kept = _kept(s.trainer.model, s.trainer.opt)
    return work


def _captured(s, case, seed):
    """A step recorded after two eager ones, the model then set back to its initial weights."""
    work = _trainer(s, case, seed, train.policy_for(_workload(case["model"])))
    tr = s.trainer
    for _ in range(2):
        tr.step(s.x, s.y)
    tr.capture(s.x, s.y)
    for layer, p in zip(tr.model.model[1:], work.params(seed)):
        if p is not None:
            layer.set_weights(p[0], p[1])
    for name in ("m", "v", "velocity"):
        if hasattr(tr.opt, name):
            sc.cuda_memset(getattr(tr.opt, name).main_ptr, 0, 4 * tr.model.n_arena)
    if isinstance(tr.opt, S.Adam):
        tr.opt.t = 1
    return work


def _batchnorm_model():
    return S.Sequential([S.Input((3, 32, 32)), S.Conv2D(32, 3, (3, 3), "relu", stride=1, zero_padding=1), S.BatchNorm2d(32),
                         S.MaxPool2D((2, 2), stride=2), S.Conv2D(64, 32, (3, 3), "relu", stride=1, zero_padding=1),
                         S.BatchNorm2d(64), S.MaxPool2D((2, 2), stride=2), S.Flatten(), S.Dense(4096, 128, activation="relu"),
                         S.BatchNorm1d(128), S.Dense(128, 10, activation="softmax")])


def _onehot(rs, n):
    return np.eye(10, dtype=np.float32)[rs.randint(0, 10, n)]


def prepare(case, seed):
    s = _State()
    s.kind = kind = case["kind"]
    sc.set_precision(case.get("precision", DEFAULT_PRECISION))
    rs = np.random.RandomState(seed % (1 << 32))
    if kind == "predict":
        work = _workload(case["model"])
        s.model = train.build_model(work, work.params(seed % 100000))
        s.x = S.Tensor(work.batch(case["batch"], seed % (1 << 32))[0], is_leaf=True)
    elif kind == "fit":
        work = _workload(case["model"])
        s.model = train.build_model(work, work.params(seed % 100000))
        s.opt, s.seed, s.batch = S.Adam(s.model, lr=ADAM_LR), seed % (1 << 32), case["batch"]
        s.host = work.batch(case["samples"], seed % (1 << 32))
        s.kept = _kept(s.model, s.opt)
    elif kind == "step":
        _trainer(s, case, seed % 100000, None)
    elif kind == "step_bn":
        np.random.seed(seed % (1 << 32))           # the layers draw their initial weights from NumPy's generator
        s.model = _batchnorm_model()
        s.opt, s.loss = S.SGD(s.model, lr=0.01, momentum=0.9), S.Loss().categorical_cross_entropy
        s.x = S.Tensor(rs.standard_normal((case["batch"], 3, 32, 32)).astype(np.float32), is_leaf=True)
        s.y = S.Tensor(_onehot(rs, case["batch"]), is_leaf=True)
        s.kept = _kept(s.model, s.opt)
        for i, layer in enumerate(s.model.model):
            if isinstance(layer, (S.BatchNorm1d, S.BatchNorm2d)):
                s.kept["mean_%d" % i], s.kept["var_%d" % i] = _view(layer._rm), _view(layer._rv)
    elif kind == "replay":
        _captured(s, case, seed % 100000)
    elif kind == "stream":
        work = _captured(s, case, seed % 100000)
        s.pinned = []
        for i in range(case["batches"]):
            buffers = []
            for a in work.batch(case["batch"], (seed + 1 + i) % (1 << 32)):
                p = sc.host_alloc_pinned(a.nbytes)
                sc.host_view(p, a.nbytes).view(np.float32)[:] = a.ravel()
                buffers.append(p)
            s.pinned.append(tuple(buffers))
    elif kind == "conv_bwd":
        n, c, f, h = case["batch"], case["channels"], case["filters"], case["size"]
        oh = (h - 1) // case["stride"] + 1
        g = torch.Generator(device="cuda").manual_seed(seed)
        normal = lambda *shape: torch.randn(shape, generator=g, device="cuda")          # noqa: E731
        s.x, s.dy = normal(n, c, h, h).relu_(), normal(n, f, oh, oh) * 1e-3
        s.w = normal(f, c, 3, 3) * math.sqrt(2.0 / (9 * c))
        s.dx, s.dw = torch.empty_like(s.x), torch.empty_like(s.w)
        s.sizes = (n, c, h, h, f, 3, 3, case["stride"], case["stride"], 1, 1)
    elif kind == "operators":
        m, k, n = case["rows"], case["inner"], case["cols"]
        s.x = cuten(rs.standard_normal((m, k)).astype(np.float32))
        s.w = cuten((rs.standard_normal((k, n)) * math.sqrt(2.0 / k)).astype(np.float32))
        s.b = cuten((rs.standard_normal((1, n)) * 0.1).astype(np.float32))
        s.head = cuten((rs.standard_normal((n, 10)) * math.sqrt(1.0 / n)).astype(np.float32))
    else:
        raise ValueError(kind)
    return s


def run(s):
    kind = s.kind
    if kind == "predict":
        return _view(s.model.predict(s.x).value)
    if kind == "fit":
        np.random.seed(s.seed)                     # the order of the samples
        history = s.model.fit(s.host[0], s.host[1], s.opt, S.Loss().categorical_cross_entropy, 1, batch_size=s.batch)
        return {"history": history, **s.kept}
    if kind == "step":
        loss = s.trainer.step(s.x, s.y)
        return {"loss": _view(loss.value), "prediction": _view(s.trainer.pred.value), **s.kept}
    if kind == "step_bn":
        pred = s.model.forward(s.x)
        loss = s.loss(pred, s.y)
        s.model.zero_grad()
        S.autograd4nn(loss)
        s.opt.step()
        return {"loss": _view(loss.value), "prediction": _view(pred.value), **s.kept}
    if kind == "replay":
        loss = s.trainer.replay()
        return {"loss": _view(loss.value), "prediction": _view(s.trainer.pred.value), **s.kept}
    if kind == "stream":
        return {"losses": s.trainer.fit_stream(s.pinned), **s.kept}
    if kind == "conv_bwd":
        sc.cuda_conv2d_bwd(s.w.data_ptr(), s.x.data_ptr(), s.dy.data_ptr(), s.dx.data_ptr(), s.dw.data_ptr(), *s.sizes)
        return {"dx": s.dx, "dw": s.dw}
    hidden = (s.x @ s.w + s.b).relu()
    prob = (hidden @ s.head).softmax()
    return {"hidden": _view(hidden), "prob": _view(prob), "class": _view(prob.argmax(1)), "top": _view(prob.max(1)),
            "mean": _view(hidden.mean(0))}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------------
def _n_params(layers):
    n = 0
    for L in layers:
        if L["type"] in ("conv", "convT"):
            n += L["in"] * L["out"] * L["k"][0] * L["k"][1] + L["out"]
        elif L["type"] == "dense":
            n += L["in"] * L["out"] + L["out"]
    return n


def _step_work(work, n):
    """One training step: the three products of every layer but the first one's data gradient; the batch read, the prediction
    written, the weights and moments read and written, the gradients written."""
    flops_first = wl._fwd_flops(work.layers[:1], work.in_shape)
    p = _n_params(work.layers)
    per_weight = 28 if work.opt["kind"] == "adam" else 20
    x = int(np.prod(work.in_shape))
    out = x if work.loss == "mse" else 10
    return {"bytes": 4.0 * n * (x + 2 * out) + per_weight * p, "flops": float(n) * (3 * work.flops_fwd - flops_first)}


def work(case):
    kind = case["kind"]
    if kind in ("predict", "fit", "step", "replay", "stream"):
        w = _workload(case["model"])
        if kind == "predict":
            x = int(np.prod(w.in_shape))
            return {"bytes": 4.0 * (case["batch"] * (x + (x if w.loss == "mse" else 10)) + _n_params(w.layers)),
                    "flops": float(case["batch"]) * w.flops_fwd}
        if kind == "fit":
            steps = -(-case["samples"] // case["batch"])
            one = _step_work(w, case["samples"])
            return {"bytes": one["bytes"] + (steps - 1) * 28.0 * _n_params(w.layers), "flops": one["flops"]}
        one = _step_work(w, case["batch"])
        times = case.get("batches", 1)
        return {k: v * times for k, v in one.items()}
    if kind == "step_bn":
        layers = [wl.conv(32, 3, 3, "relu", 1, 1), wl.maxpool(2, 2), wl.conv(64, 32, 3, "relu", 1, 1), wl.maxpool(2, 2), wl.flatten(),
                  wl.dense(4096, 128), wl.dense(128, 10, "softmax")]
        fwd = wl._fwd_flops(layers, (3, 32, 32))
        p = _n_params(layers) + 2 * (32 + 64 + 128)
        return {"bytes": 4.0 * case["batch"] * (3072 + 20) + 20.0 * p,
                "flops": float(case["batch"]) * (3 * fwd - wl._fwd_flops(layers[:1], (3, 32, 32)))}
    if kind == "conv_bwd":
        n, c, f, h = case["batch"], case["channels"], case["filters"], case["size"]
        oh = (h - 1) // case["stride"] + 1
        return {"bytes": 4.0 * (2 * n * c * h * h + n * f * oh * oh + 2 * f * c * 9), "flops": 2 * 2.0 * n * f * oh * oh * c * 9}
    m, k, n = case["rows"], case["inner"], case["cols"]
    return {"bytes": 4.0 * (m * k + k * n + m * n + n * 10 + m * 10 + 2 * m + 2 * n), "flops": 2.0 * m * n * (k + 10)}


def tolerance(case):
    """Between two correct implementations at the same precision."""
    kind = case["kind"]
    if kind == "conv_bwd":                  # one bf16 pass, or split products with 32-bit sums over up to 800 k terms
        return {"rel": 5e-3, "max": 0.1} if case["precision"] == 1 else {"rel": 3e-5, "max": 1e-3}
    if kind == "operators":
        return {"rel": 1e-5, "max": 1e-3, "differ": 1e-3}
    if kind == "predict":
        return {"rel": 2e-5, "max": 1e-3}
    # A step: where another order of the sums moves a value by its last bits across a ReLU's or a max-pool's tie, one
    # contribution to a gradient is there or not.  That is rare, but in a deep model on noise images, whose first-layer gradients
    # are sums that nearly cancel, a few such decisions are 1e-3 to 1e-2 of a gradient (the framework's own bound against exact
    # arithmetic is 2e-3 for one step of its full batch), and the steps of a stream add up.
    model = case.get("model")
    if model == "c3":
        return {"rel": 3e-2, "max": 0.8} if kind == "stream" else {"rel": 1.5e-2, "max": 0.4}
    if model == "c2":                       # its backward products are one pass on 16-bit operands
        return {"rel": 5e-3, "max": 0.5}
    return {"rel": 1e-3, "max": 0.05}
