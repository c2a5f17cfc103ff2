"""What this framework is timed on: one training step of a GPU rank, and whole training sessions.

A framework whose only job is training has two things a user waits for. A long run is its steps, so most cases are ONE
optimizer step of a rank on one GPU: the batch crosses PCIe out of pinned host memory one step ahead, forward, loss,
backward, optimizer, and the loss of an earlier step is read, in the order in which the runtime's own loop issues them
(``GpuRank``, ``BatchFeeder.stage``, ``gpu_loop.run_batch``). A short run is ``orchestrate(...).wait()`` from start to end,
planning, initialisation, first steps and the trained model's way back to the host included, so three cases are whole sessions.

``kind`` "step" / "session"; ``arch``: the layers, comma separated: ``conv:F:K:stride:padding:act``, ``pool:K``,
``dense:width:act`` (an activation may be empty); ``x``: features of a sample, or ``CxHxW``; ``y``: outputs of the last layer.
"""
import json
import threading

import numpy as np
import torch

import orchestra
from orchestra import _orchestra as core
from orchestra import orchestrate
from orchestra import activations as A
from orchestra.arch import Conv2d, Dense, MaxPooling
from orchestra.datasets import InlineDataset
from orchestra.initialization import Kaiming, Xavier, XavierUniform
from orchestra.loss_fns import CrossEntropy, Mse
from orchestra.optimizers import Adam, GradientDescent, GradientDescentWithMomentum
from orchestra.serializer import BaseSerializer, SparseSerializer
from orchestra.store import BlockingStore
from orchestra.sync import BarrierSync

LENET5 = "conv:6:5:1:2:tanh,pool:2,conv:16:5:1:0:tanh,pool:2,dense:120:tanh,dense:84:tanh"
NIELSEN = "conv:20:5:1:0:,pool:2,dense:100:sigmoid"
CNN = "conv:32:3:1:1:relu,conv:64:3:2:1:relu,conv:64:3:2:1:relu,dense:128:relu"


def _case(name, kind, arch, x, y, *, tile, opt, batch, loss="cross_entropy", data="uniform", **more):
    return dict(name=name, kind=kind, arch=arch, x=str(x), y=y, tile=tile, opt=opt, batch=batch, loss=loss, data=data, **more)


def listed():
    return [
        # the smallest network of the benchmark (784-128-10, batch 32): a step is launches and latency
        _case("step_mlp_b32", "step", "dense:128:relu", 784, 10, tile="tf32", opt="sgd", batch=32),
        # the two small convolutional networks of the examples and the published benchmark rows, at their two batch sizes
        _case("step_lenet5_b64", "step", LENET5, "1x28x28", 10, tile="tf32", opt="sgd", batch=64, data="digits"),
        _case("step_nielsen_b256", "step", NIELSEN, "1x28x28", 10, tile="tf32", opt="momentum", batch=256, data="digits"),
        # regression on widths that are no multiple of anything, a batch that fills no tile: every row is unaligned
        _case("step_ragged_mse_b200", "step", "dense:1001:tanh,dense:333:sigmoid", 517, 6, tile="tf32", opt="adam", batch=200,
              loss="mse"),
        # an ordinary GELU network with bf16 tiles
        _case("step_bf16_2048x4_b256", "step", "dense:2048:gelu," * 3 + "dense:2048:gelu", 1024, 100, tile="bf16", opt="adam",
              batch=256, data="normal"),
        # the benchmark's CNN: a global batch of 2048 over 6 workers; and the whole of it on one GPU with bf16 tiles
        _case("step_cnn_b342", "step", CNN, "1x28x28", 10, tile="tf32", opt="adam", batch=342, strategy="ps"),
        _case("step_cnn_bf16_b2048", "step", CNN, "1x28x28", 10, tile="bf16", opt="adam", batch=2048, strategy="ps"),
        # the benchmark's wide network (784-4096x3-10)
        _case("step_wide_b1024", "step", "dense:4096:relu,dense:4096:relu,dense:4096:relu", 784, 10, tile="tf32", opt="adam",
              batch=1024),
        # the headline benchmark: 8 layers of 8192, 545 M parameters
        _case("step_deep_b512", "step", ",".join(["dense:8192:gelu"] * 8), 8192, 1000, tile="bf16", opt="momentum", batch=512,
              data="normal", strategy="ps"),
        # a whole run of the smallest network: one epoch over 60000 samples, 1875 steps
        _case("session_mlp_1epoch", "session", "dense:128:relu", 784, 10, tile="tf32", opt="sgd", batch=32, rows=60000, epochs=1,
              cadence="step"),
        # the example program as it stands: LeNet-5, 4096 samples, 4 epochs, one exchange per epoch (the default cadence)
        _case("session_lenet5_4epochs", "session", LENET5, "1x28x28", 10, tile="tf32", opt="sgd", batch=64, data="digits",
              rows=4096, epochs=4, cadence="round"),
        # the same cadence with the sparse gradient wire on a network of a few million parameters
        _case("session_sparse_4epochs", "session", "dense:1024:relu,dense:1024:relu", 784, 10, tile="tf32", opt="adam", batch=256,
              rows=4096, epochs=4, cadence="round", sparse=0.1),
    ]


def _log(rng, lo, hi):
    """A size spread over its logarithm; one in three rounded to a multiple of 16, as widths and batches mostly are."""
    v = int(round(lo * (hi / lo) ** rng.random()))
    return max(lo, min(hi, (v + 8) // 16 * 16)) if rng.random() < 1 / 3 and hi >= 64 else v


MOST_FLOPS = 1.6e12          # the largest listed step
MOST_COLS = 3.0e8            # elements of the largest layer's unfolded input that a drawn convolution may have


def draw(rng):
    while True:
        c = _draw(rng)
        w = work(c)
        if w["flops"] <= MOST_FLOPS and w["bytes"] <= 8.7e9 and max(_cols(c), default=0) <= MOST_COLS:
            return c


def _draw(rng):
    what = rng.choice(["small", "tf32", "tf32", "bf16", "bf16", "conv", "conv", "session"])
    opt = rng.choice(["sgd", "momentum", "adam"])
    loss = rng.choice(["cross_entropy", "cross_entropy", "mse"])
    y = _log(rng, 2, 1000) if what in ("tf32", "bf16") else 10
    if what == "conv":
        k = rng.choice([3, 5])
        side = rng.choice([28, 28, 32, 20])
        f1, f2 = _log(rng, 4, 64), _log(rng, 8, 96)
        act = rng.choice(["relu", "tanh"])
        if rng.random() < 0.5:
            arch = "conv:%d:%d:1:%d:%s,pool:2,conv:%d:%d:1:0:%s,pool:2,dense:%d:%s" % (f1, k, k // 2, act, f2, k, act, _log(rng, 32, 512), act)
        else:
            arch = "conv:%d:3:1:1:%s,conv:%d:3:2:1:%s,dense:%d:%s" % (f1, act, f2, act, _log(rng, 32, 512), act)
        return dict(kind="step", arch=arch, x="%dx%dx%d" % (rng.choice([1, 1, 3]), side, side), y=y, tile=rng.choice(["tf32", "bf16"]),
                    opt=opt, batch=_log(rng, 16, 2048), loss="cross_entropy", data="digits")
    if what == "session":
        arch = rng.choice([LENET5, NIELSEN, "dense:%d:relu" % _log(rng, 32, 512), "dense:%d:relu,dense:%d:tanh" % (_log(rng, 64, 1024), _log(rng, 32, 512))])
        batch, epochs = _log(rng, 32, 256), rng.choice([1, 2, 4])
        rows = min(_log(rng, 1024, 60000), (600 if arch.startswith("conv") else 1800) * batch // epochs)
        return dict(kind="session", arch=arch, x="1x28x28" if arch.startswith("conv") else "784", y=10, tile="tf32", opt="sgd", batch=batch,
                    loss="cross_entropy", data="digits", rows=rows, epochs=epochs, cadence=rng.choice(["step", "round"]))
    lo, hi, deep, bmax = {"small": (16, 256, 2, 256), "tf32": (64, 4096, 4, 2048), "bf16": (128, 8192, 8, 1024)}[what]
    acts = ["relu", "tanh", "sigmoid", "gelu"]
    widths = [_log(rng, lo, hi)] * rng.randint(1, deep) if rng.random() < 0.5 else [_log(rng, lo, hi) for _ in range(rng.randint(1, deep))]
    act = rng.choice(acts)
    return dict(kind="step", arch=",".join("dense:%d:%s" % (w, act) for w in widths), x=str(_log(rng, 8 if what == "small" else 64, min(4096, 4 * hi))), y=y,
                tile="bf16" if what == "bf16" else "tf32", opt=opt, batch=_log(rng, 8, bmax), loss=loss, data=rng.choice(["uniform", "normal"]))


# ------------------------------------------------------------------------------------------------------------------
def _dims(c):
    return [int(v) for v in c["x"].split("x")]


def _layers(c):
    """(kind, in, out, multiply-adds of a sample, parameters, unfolded elements of a sample) of every layer, the output layer last."""
    shape, out = _dims(c), []
    for spec in c["arch"].split(","):
        f = spec.split(":")
        if f[0] == "dense":
            i, o = int(np.prod(shape)), int(f[1])
            out.append(("dense", i, o, i * o, (i + 1) * o, 0))
            shape = [o]
            continue
        ch, h, w = shape
        k, s, p, fo = (int(f[2]), int(f[3]), int(f[4]), int(f[1])) if f[0] == "conv" else (int(f[1]), int(f[1]), 0, ch)
        oh, ow = (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1
        if f[0] == "conv":
            out.append(("conv", ch * h * w, fo * oh * ow, oh * ow * fo * ch * k * k, fo * (ch * k * k + 1), oh * ow * ch * k * k))
        else:
            out.append(("pool", ch * h * w, fo * oh * ow, 0, 0, 0))
        shape = [fo, oh, ow]
    i = int(np.prod(shape))
    return out + [("dense", i, c["y"], i * c["y"], (i + 1) * c["y"], 0)]


def _cols(c):
    return [l[5] * c["batch"] for l in _layers(c)]


def work(case):
    """A step: the batch read, parameters and optimizer state read and written once, the three products of every layer
    (no input gradient below the first). A session: the same steps, its parameters moved once and its samples once an epoch."""
    ls = _layers(case)
    params = sum(l[4] for l in ls)
    macs = sum(l[3] for l in ls)
    per_sample = 2.0 * (3 * macs - ls[0][3])
    row = 4.0 * (ls[0][1] + case["y"])
    state = {"sgd": 2, "momentum": 4, "adam": 6}[case["opt"]] * 4.0 * params
    if case["kind"] == "step":
        return {"bytes": case["batch"] * row + state, "flops": case["batch"] * per_sample}
    n = case["rows"] * case["epochs"]
    return {"bytes": n * row + state, "flops": n * per_sample}


def tolerance(case):
    """About four times what gradients and moments were off by against the same step in 64 bits: 0.1 to 0.5 % for smooth
    activations with tf32 tiles; 1 to 5 % with bf16 tiles or a ReLU, whose gradient jumps where a pre-activation is within
    rounding of zero (single entries then differ by as much as their own size). A session's weights have moved little."""
    if case["kind"] == "session":
        return {"rel": 1e-2 if case.get("sparse") else 1e-3}
    if case["tile"] == "bf16" or "relu" in case["arch"]:
        return {"rel": 3e-2, "max": 0.99}
    return {"rel": 2e-2, "max": 0.6}


# ------------------------------------------------------------------------------------------------------------------
def _act(name):
    return {"": lambda: None, "relu": lambda: A.ReLU(0.0), "tanh": A.Tanh, "sigmoid": A.Sigmoid, "gelu": A.GELU}[name]()


def _model(c):
    shape, out = _dims(c), []
    init = XavierUniform if "conv" not in c["arch"] and c["tile"] == "tf32" else Xavier if "tanh" in c["arch"] else Kaiming
    for spec in c["arch"].split(","):
        f = spec.split(":")
        if f[0] == "dense":
            out.append(Dense(int(f[1]), init(), _act(f[2])))
            continue
        ch, h, w = shape
        if f[0] == "conv":
            fo, k, s, p = (int(v) for v in f[1:5])
            out.append(Conv2d((ch, h, w), (fo, ch, k), s, p, init(), _act(f[5])))
        else:
            fo, k, s, p = ch, int(f[1]), int(f[1]), 0
            out.append(MaxPooling((ch, h, w), k, s, p))
        shape = [fo, (h + 2 * p - k) // s + 1, (w + 2 * p - k) // s + 1]
    return orchestra.Sequential(out + [Dense(c["y"], init(), A.Softmax() if c["loss"] == "cross_entropy" else None)])


def _data(c, rows, seed):
    """Samples and labels of a seed: pixels or features ~U[0,1] or ~N(0,1) with labels drawn uniformly, or blurry class prototypes."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x_size, y = int(np.prod(_dims(c))), c["y"]
    label = torch.randint(0, y, (rows,), device="cuda", generator=g)
    if c["data"] == "normal":
        xs = torch.randn(rows, x_size, device="cuda", generator=g)
    else:
        xs = torch.rand(rows, x_size, device="cuda", generator=g)
        if c["data"] == "digits":
            proto = torch.rand(y, x_size, device="cuda", generator=g)
            xs = (proto[label] + 0.35 * torch.randn(rows, x_size, device="cuda", generator=g)).clamp_(0, 1)
    if c["loss"] == "mse":
        ys = torch.rand(rows, y, device="cuda", generator=g)
    else:
        ys = torch.zeros(rows, y, device="cuda").scatter_(1, label[:, None], 1.0)
    return InlineDataset(xs.cpu().numpy(), ys.cpu().numpy(), x_size, y)


def _training(c, ds, epochs, seed, cadence):
    opt = {"sgd": lambda: GradientDescent(0.01), "momentum": lambda: GradientDescentWithMomentum(0.01, 0.9), "adam": lambda: Adam(1e-3)}[c["opt"]]()
    loss = CrossEntropy() if c["loss"] == "cross_entropy" else Mse()
    b200 = {"tile_dtype": c["tile"], "sync_every": cadence}
    kw = dict(max_epochs=epochs, batch_size=c["batch"], seed=seed, serializer=SparseSerializer(c["sparse"]) if c.get("sparse") else BaseSerializer())
    if c.get("strategy") == "ps":
        return orchestra.parameter_server(["gpu:0"], 1, ds, opt, loss, BarrierSync(), BlockingStore(), b200=dict(b200, sharding="even", colocate=True), **kw)
    return orchestra.all_reduce(["gpu:0"], ds, opt, loss, b200=b200, **kw)


class _Loop:
    """A rank in the middle of its training loop: the next batch is on its way, one step may still be running."""

    def __init__(self, case, seed):
        from oxidized_neural_orchestra_b200.runtime.gpu_worker import GpuRank

        ds = _data(case, 4 * case["batch"], seed)
        cfg = _training(case, ds, 1, seed, "step")
        plan = json.loads(core.adapt_configs(json.dumps(_model(case).to_config()), json.dumps(cfg.to_config(with_data=False))))
        self.rank = GpuRank(plan, 0, 1, torch.device("cuda", 0), ds.samples, ds.labels, lambda ev: None, threading.Event())
        self.steps = self.rank.feeder.steps_per_epoch()
        self.rows, self.it, self.loss = [0, 0], 0, 0.0
        self.rows[0] = self.rank.feeder.stage(0, 0, 0)

    def step(self):
        from oxidized_neural_orchestra_b200.runtime.gpu_loop import run_batch

        r, slot = self.rank, self.it % 2
        here = torch.cuda.current_stream()
        r.stream.wait_stream(here)
        if self.it >= 2:                        # the loop reads every loss, two steps late
            r.loss_evt[slot].synchronize()
            self.loss = float(r.loss_pin[slot].item())
        run_batch(r, slot, self.rows[slot])
        self.it += 1
        self.rows[slot ^ 1] = r.feeder.stage(slot ^ 1, self.it // self.steps, self.it % self.steps)
        here.wait_stream(r.stream)
        out = {"params": r.C, "loss": r.engine.loss_sum}
        if r.sync_opt.kind == "sgd":
            out["grads"] = r.G
        else:
            out["m"] = r.m_loc                  # momentum: the gradients' own sum
        if r.sync_opt.kind == "adam":
            out["v"] = r.v_loc
        return out


class _Session:
    def __init__(self, case, seed):
        ds = _data(case, case["rows"], seed)
        self.model, self.training = _model(case), _training(case, ds, case["epochs"], seed, case["cadence"])

    def step(self):
        trained = orchestrate(self.model, self.training).wait(quiet=True)
        return {"params": trained.weights_array(), "losses": np.asarray(trained.loss_history())}


def prepare(case, seed):
    return (_Loop if case["kind"] == "step" else _Session)(case, seed)


def run(state):
    return state.step()
