"""Performance cases: the work a training program has this framework do, through its public entry points.

A case is a dict of plain sizes.  `prepare` builds what the program holds before the call (layers with bound parameters,
a parameter-server module, a batch), `run` makes one pass, `exact` gives the same results in 64 bits from plain torch.
Layer cases run forward and backward, since nothing here is used for inference alone, and as a training program runs its
layers: recorded once and replayed as a graph (PSModule(use_graph=True) does the same with a whole step).  The training
step and the table clocks go through their calls one by one.  Sizes come from the networks in geeps_b200/models and from
the push / pull sweep (geeps_b200/utils/pushpull_bench.py).
"""
from __future__ import annotations

import math
import socket

import torch
import torch.nn.functional as TF

from geeps_b200.models.alexnet import alexnet
from geeps_b200.models.net import Concat
from geeps_b200.ops import _lib as L
from geeps_b200.ops.layers import LRN, BatchNorm, Conv2d, Input, Linear, LRNMaxPool, Pool, SoftmaxLoss
from geeps_b200.parallel.ps import GeePs
from geeps_b200.parallel.ps_module import PSModule
from geeps_b200.utils.config import DEVICE_CUDA, TABLE_SGD_MOMENTUM, TRANSPORT_NVLINK, GeePsConfig

BF = torch.bfloat16
LR, MOMENTUM, DECAY = 0.01, 0.9, 5e-4
MEAN, SCALE, SRC = (104.0, 117.0, 123.0), 1.0 / 58.0, 256      # pixels of 256 x 256 source images, Caffe's mean values


def listed():
    return [
        # one training step of the flagship network (images/s is the headline metric): input layer, forward, backward,
        # parameter push, as the trainer runs it
        dict(name="alexnet_step_b256", kind="step", batch=256),
        # single layers and blocks of that step
        dict(name="conv_5x5_27_b256", kind="conv", batch=256, hw=27, cin=96, cout=256, k=5, stride=1, pad=2, groups=2),
        dict(name="conv_3x3_13_b256", kind="conv", batch=256, hw=13, cin=256, cout=384, k=3, stride=1, pad=1, groups=1),
        dict(name="lrn_pool_55_b256", kind="lrn_pool", batch=256, hw=55, c=96),
        dict(name="fc_9216_4096_b256", kind="fc", batch=256, n_in=9216, n_out=4096),
        # a batch of 8-bit source images cropped, mirrored, mean-subtracted and scaled into the network's input layout
        dict(name="input_u8_b256", kind="input", batch=256, crop=227),
        # layers and blocks of the Inception networks: a down-sampling convolution of the 32 x 32 network at its batch
        # of 100, then the 22K-class network at its batch of 32: its widest BatchNorm, one of its modules (some 50
        # small kernels on four streams) and its classifier with the loss
        dict(name="conv_3x3s2_32_b100", kind="conv", batch=100, hw=32, cin=80, cout=80, k=3, stride=2, pad=1, groups=1),
        dict(name="bn_relu_56_b32", kind="bn", batch=32, hw=56, c=192),
        dict(name="inception_14_b32", kind="inception", batch=32, hw=14, cin=576, c1=160, c3r=128, c3=160, cd3r=128,
             cd3=160, cproj=128),
        dict(name="head_21841_b32", kind="head", batch=32, n_in=1024, classes=21841),
        # a clock of the raw table interface (read all rows, write an update, push): 1 MiB, where latency counts, and
        # 256 MiB
        dict(name="clock_1mb", kind="clock", rows=2048),
        dict(name="clock_256mb", kind="clock", rows=524288),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "conv", "conv", "conv", "lrn_pool", "fc", "fc", "input", "bn", "inception", "head", "clock",
                       "clock"])
    if kind == "step":
        return dict(kind=kind, batch=_log(rng, 8, 255))
    if kind == "conv":
        k = rng.choice([3, 3, 5])
        stride = rng.choice([1, 1, 2]) if k == 3 else 1
        groups = rng.choice([1, 1, 2])
        hw = _log(rng, 7, 56)
        cin, cout = (groups * 8 * rng.randint(4, 48 // groups) for _ in range(2))
        batch = _log(rng, 1, 256)
        batch = max(1, min(batch, 40_000_000 // (hw * hw * max(cin, cout))))
        return dict(kind=kind, batch=batch, hw=hw, cin=cin, cout=cout, k=k, stride=stride, pad=k // 2, groups=groups)
    if kind == "lrn_pool":
        return dict(kind=kind, batch=_log(rng, 1, 255), hw=rng.randint(13, 55), c=8 * rng.randint(4, 12))
    if kind == "fc":
        return dict(kind=kind, batch=_log(rng, 1, 256), n_in=8 * _log(rng, 32, 1152), n_out=_log(rng, 10, 4096))
    if kind == "input":
        return dict(kind=kind, batch=_log(rng, 1, 255), crop=rng.randint(200, 240))
    if kind == "bn":
        return dict(kind=kind, batch=_log(rng, 1, 100), hw=rng.randint(7, 56), c=8 * rng.randint(4, 24))
    if kind == "inception":
        c = lambda lo, hi: 32 * rng.randint(lo, hi)     # noqa: E731
        return dict(kind=kind, batch=_log(rng, 4, 32), hw=rng.choice([7, 14, 28]), cin=c(6, 18), c1=c(2, 6), c3r=c(2, 4),
                    c3=c(2, 6), cd3r=c(2, 4), cd3=c(2, 6), cproj=c(1, 4))
    if kind == "head":
        return dict(kind=kind, batch=_log(rng, 4, 64), n_in=1024, classes=_log(rng, 100, 21841))
    return dict(kind="clock", rows=_log(rng, 1000, 524288))


# ---- what a program holds before the call ----

_stream = None


def _on_stream():
    """Everything runs on one side stream, as in a trainer (captures are not possible on the default stream)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream(priority=-1)
    return torch.cuda.stream(_stream)


class _Open:
    """Closes a parameter-server client when nothing holds it any more: neither the state nor a result, since rows and
    gradients are views of memory that the client owns."""

    def __init__(self, ps):
        self.ps = ps

    def lend(self, views):
        for v in views:
            v.client = self
        return views

    def __del__(self):
        torch.cuda.synchronize()
        self.ps.close()


_next_port = 11000


def _port() -> int:
    global _next_port
    while True:
        _next_port = 11000 + (_next_port - 11000 + 20) % 20000
        with socket.socket() as s:
            try:
                s.bind(("127.0.0.1", _next_port))
                return _next_port
            except OSError:
                pass


def _config():
    return GeePsConfig(device=DEVICE_CUDA, cuda_device=torch.cuda.current_device(), transport=TRANSPORT_NVLINK,
                       table_mode=TABLE_SGD_MOMENTUM, port_list=[_port()], learning_rate=LR, momentum=MOMENTUM,
                       weight_decay=DECAY, bf16_compute_cache=1)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(gen, *shape):
    return torch.randn(shape, device="cuda", generator=gen)


def _bind(layer, gen):
    """Parameters as the parameter server hands them to a layer: fp32 and bf16 rows, and rows for the gradients."""
    for l in _sublayers(layer):
        for sp in l.param_specs():
            if sp.name == "weight":
                w = _randn(gen, *sp.shape) * math.sqrt(2.0 / (sp.valid_cols or sp.shape[1]))
                w[:, sp.valid_cols or sp.shape[1]:] = 0
            elif sp.name == "gamma":
                w = 1 + 0.1 * _randn(gen, *sp.shape)
            else:
                w = 0.1 * _randn(gen, *sp.shape)
            l.p32[sp.name], l.p16[sp.name], l.g32[sp.name] = w, w.to(BF), torch.zeros_like(w)


def _module(c):
    """1x1 | 1x1 - 3x3 | 1x1 - 3x3 - 3x3 | average pooling - 1x1, each convolution with BatchNorm and ReLU."""
    def conv(cout, k):
        return [Conv2d("conv", cout, k, pad=k // 2, bias=False, std=0.0), BatchNorm("bn", relu=True)]
    return Concat("in", [conv(c["c1"], 1), conv(c["c3r"], 1) + conv(c["c3"], 3),
                         conv(c["cd3r"], 1) + conv(c["cd3"], 3) + conv(c["cd3"], 3),
                         [Pool("avg", 3, 1, pad=1, ceil_mode=False)] + conv(c["cproj"], 1)])


def _layer(c):
    k = c["kind"]
    if k == "conv":
        return Conv2d("conv", c["cout"], c["k"], stride=c["stride"], pad=c["pad"], groups=c["groups"], relu=True)
    if k == "fc":
        return Linear("fc", c["n_out"], relu=True)
    if k == "head":
        return Linear("fc", c["classes"], fp32_out=True)
    if k == "bn":
        return BatchNorm("bn", relu=True)
    if k == "inception":
        return _module(c)
    lrn, pool = LRN(5, 1e-4, 0.75, 1.0), Pool("max", 3, 2)
    assert LRNMaxPool.fusable(lrn, pool, _in_shape(c))
    return LRNMaxPool(lrn, pool)


def _in_shape(c):
    if c["kind"] in ("fc", "head"):
        return (c["batch"], c["n_in"])
    return (c["batch"], c["hw"], c["hw"], c.get("cin", c.get("c")))


def _batch(c, seed):
    """Images and labels, or the activations and output gradients that reach a layer."""
    gen = _gen(seed)
    k = c["kind"]
    if k == "step":
        return dict(x=_randn(gen, c["batch"], 3, 227, 227).to(BF),
                    labels=torch.randint(0, 1000, (c["batch"],), device="cuda", generator=gen))
    if k == "input":
        B, room = c["batch"], SRC - c["crop"] + 1
        return dict(x=torch.randint(0, 256, (B, 3, SRC, SRC), device="cuda", generator=gen, dtype=torch.uint8),
                    aug=torch.stack([torch.randint(0, n, (B,), device="cuda", generator=gen) for n in (room, room, 2)], 1))
    if k == "clock":
        return dict(w0=_randn(gen, c["rows"], 128) * 0.05, update=_randn(gen, c["rows"], 128) * 0.01)
    x = _randn(gen, *_in_shape(c))
    if k == "bn":
        x = 2 * x + 0.5                                  # a convolution's output
    elif k == "lrn_pool":
        x = torch.relu(3 * x)                            # behind a convolution with ReLU
    else:
        x = torch.relu(x)
    out = dict(x=x.to(BF))
    if k == "head":
        out["labels"] = torch.randint(0, c["classes"], (c["batch"],), device="cuda", generator=gen)
    return out


def prepare(case, seed):
    c = case
    s = dict(c, **_batch(c, seed))
    dev = torch.device("cuda", torch.cuda.current_device())
    if c["kind"] in ("step", "clock"):
        torch.cuda.synchronize()
        with _on_stream():
            if c["kind"] == "step":
                s["mod"] = PSModule(alexnet(), (c["batch"], 3, 227, 227), _config(), device=dev, seed=seed,
                                    bf16_weights_only=True, use_graph=True)
                s["open"] = _Open(s["mod"])
            else:
                s["ps"] = ps = GeePs(0, _config())
                s["open"] = _Open(ps)
                ids = range(c["rows"])
                s["read"], s["pre"] = ps.virtual_read(0, ids, 0), ps.virtual_pre_update(0, ids)
                s["post"], s["upd"] = ps.virtual_post_read(s["read"]), ps.virtual_update(s["pre"])
                ps.virtual_clock()
                ps.finish_virtual_iteration()
                ps.pre_update(s["pre"]).copy_(s.pop("w0"))          # the first update carries the initial values
                ps.update(s["upd"])
                ps.clock()
                ps.start_iterations()
        return s
    if c["kind"] == "input":
        s["layer"] = Input(s2d=4, s2d_k=11, cpad=64, mean=MEAN, scale=SCALE)
        s["layer"].setup((c["batch"], 3, c["crop"], c["crop"]), dev)
        s["layer"].set_augmentation(s["aug"])
        return _capture(s)
    gen = _gen(seed + 1_000_003)
    s["layer"] = layer = _layer(c)
    shape = layer.setup(_in_shape(c), dev)
    _bind(layer, gen)
    if c["kind"] == "head":
        s["loss"] = SoftmaxLoss()
        s["loss"].setup(shape, dev)
        return _capture(s)
    s["dy"] = (_randn(gen, *shape) * 0.01).to(BF)
    if c["kind"] in ("fc", "bn", "conv", "inception"):
        s["dy"] = s["dy"].view(-1, shape[-1])
    if c["kind"] == "lrn_pool":                # behind a convolution, as the network container sets the pair up
        layer.mask_relu_input, layer.bias_grad = True, torch.zeros(c["c"], device="cuda")
    return _capture(s)


def _capture(s):
    """Record one pass over the layers and capture it as a graph; the pass leaves no trace in the layers' state."""
    torch.cuda.synchronize()
    with _on_stream():
        L.start_recording()
        try:
            s["out"] = _pass(s)
        finally:
            tape = L.stop_recording()
        s["graph"] = L.StepGraph(tape, _stream)
        for l in _sublayers(s["layer"]):
            if isinstance(l, BatchNorm):
                l.running_mean.zero_()
                l.running_var.fill_(1.0)
    return s


# ---- one pass ----

def _sublayers(layer):
    return list(layer.sublayers()) if hasattr(layer, "sublayers") else [layer]


def _grads(layer):
    return [l.g32[sp.name] for l in _sublayers(layer) for sp in l.param_specs()]


def run(state):
    s = state
    k = s["kind"]
    if k == "step":
        with _on_stream():
            loss = s["mod"].step(s["x"], s["labels"])
        layers = s["mod"].net.param_layers()
        return [loss, layers[-1].y] + s["open"].lend([g for l in layers for g in _grads(l)])
    if k == "clock":
        ps = s["ps"]
        with _on_stream():
            rows = ps.read(s["read"])
            buf = ps.pre_update(s["pre"])
            ps.post_read(s["post"])
            buf.copy_(s["update"])             # the worker writes its update in place
            ps.update(s["upd"])
            ps.clock()
        return s["open"].lend([rows])
    s["graph"].launch()
    return s["out"]


def _pass(s):
    """Forward and backward of a layer case; returns the buffers that hold its results."""
    k, layer = s["kind"], s["layer"]
    if k == "input":
        return layer.forward(s["x"])
    if k == "head":
        logits = layer.forward(s["x"])
        loss = s["loss"].forward(logits, s["labels"])
        return [logits, loss, layer.backward(s["loss"].backward())] + _grads(layer)
    y = layer.forward(s["x"])
    dx = layer.backward(s["dy"])
    if k == "lrn_pool":
        return [y, layer.argmax, dx, layer.bias_grad]
    if k == "bn":
        return [y, dx] + _grads(layer) + [layer.running_mean, layer.running_var]
    return [y, dx] + _grads(layer)


# ---- what a pass cannot do without ----

def _conv_work(B, hw_in, hw_out, cin, cout, k, groups):
    m, n = B * hw_out * hw_out, cout * k * k * (cin // groups)
    x, y = 2 * B * hw_in * hw_in * cin, 2 * m * cout
    return 2 * x + 2 * y + (2 + 4) * n, 3 * 2 * m * n          # x, dy, w in; y, dx, dw out: three products


def work(case):
    c = case
    k, B = c["kind"], c.get("batch", 0)
    if k == "step":
        # per image 2.27 GFLOP in the three products of every layer but conv1 (no data gradient); per step the 61 M
        # parameters: fp32 gradient out, and for the optimizer fp32 gradient, weight and momentum in, weight, momentum
        # and bf16 copy out
        conv1 = 2 * 55 * 55 * 96 * 363
        rest = 2 * (27 * 27 * 256 * 1200 + 13 * 13 * (384 * 2304 + 384 * 1728 + 256 * 1728) + 9216 * 4096 + 4096 * 4096
                    + 4096 * 1000)
        acts = 290400 + 186624 + 64896 * 2 + 43264             # convolution outputs of one image
        return {"bytes": 60_965_224 * (4 * 6 + 2) + B * (2 * 154587 + 4 * 2 * acts), "flops": B * (2 * conv1 + 3 * rest)}
    if k == "clock":
        return {"bytes": c["rows"] * 512 * 8 + c["rows"] * 256, "flops": c["rows"] * 128 * 5}
    if k == "input":
        n = ((c["crop"] - 11) // 4 + 3) ** 2 * 64
        return {"bytes": B * (3 * c["crop"] ** 2 + 2 * n), "flops": B * 3 * c["crop"] ** 2 * 2}
    if k in ("fc", "head"):
        n = c.get("n_out") or c["classes"]
        w = c["n_in"] * n
        return {"bytes": 6 * w + 2 * B * (2 * c["n_in"] + (4 if k == "head" else 2) * n), "flops": 6 * B * w}
    if k == "lrn_pool":
        out = math.ceil((c["hw"] - 3) / 2) + 1
        n = B * c["c"]
        return {"bytes": n * (4 * c["hw"] ** 2 + 5 * out ** 2), "flops": n * c["hw"] ** 2 * 30}
    if k == "bn":
        n = B * c["hw"] ** 2 * c["c"]
        return {"bytes": 8 * n, "flops": 16 * n}
    if k == "conv":
        out = (c["hw"] + 2 * c["pad"] - c["k"]) // c["stride"] + 1
        b, f = _conv_work(B, c["hw"], out, c["cin"], c["cout"], c["k"], c["groups"])
        return {"bytes": b, "flops": f}
    hw, cin = c["hw"], c["cin"]
    flops = sum(_conv_work(B, hw, hw, i, o, kk, 1)[1] for i, o, kk in _convs(c))
    weights = sum(i * o * kk * kk for i, o, kk in _convs(c))
    outs = c["c1"] + c["c3"] + c["cd3"] + c["cproj"]
    return {"bytes": 2 * 2 * B * hw * hw * (cin + outs) + 6 * weights, "flops": flops}


def _convs(c):
    return [(c["cin"], c["c1"], 1), (c["cin"], c["c3r"], 1), (c["c3r"], c["c3"], 3), (c["cin"], c["cd3r"], 1),
            (c["cd3r"], c["cd3"], 3), (c["cd3"], c["cd3"], 3), (c["cin"], c["cproj"], 1)]


def tolerance(case):
    return {
        # the whole network: bf16 roundings travel through eight layers, and a rounding that moves the maximum of a
        # pooling window or the sign in front of a ReLU moves a gradient
        "step": {"rel": 0.03, "max": 0.9},
        # single layers: bf16 results of fp32 sums
        "conv": {"rel": 4e-3, "max": 0.1}, "fc": {"rel": 4e-3, "max": 0.1}, "head": {"rel": 4e-3, "max": 0.1},
        "bn": {"rel": 4e-3, "max": 0.9}, "lrn_pool": {"rel": 1e-2, "max": 0.9, "differ": 1e-3},
        # a block: bf16 between its layers, sums over ReLU masks in its gradients
        "inception": {"rel": 2e-2, "max": 0.9},
        "input": {"rel": 1e-4, "max": 8e-3},
        "clock": {"rel": 1e-6, "max": 1e-5},
    }[case["kind"]]


# ---- the same results in 64 bits ----

def _conv64(x, w, stride, pad, groups=1):
    """Convolution of NHWC x with w [cout, k, k, cin / groups] as one matrix product per tap (a 64-bit convolution of the
    library is far slower)."""
    k, xp = w.shape[1], TF.pad(x, (0, 0, pad, pad, pad, pad))
    n = (x.shape[1] + 2 * pad - k) // stride + 1
    ci, co = w.shape[3], w.shape[0] // groups
    out = []
    for g in range(groups):
        acc = 0
        for t in range(k * k):
            h, v = t // k, t % k
            tap = xp[:, h:h + (n - 1) * stride + 1:stride, v:v + (n - 1) * stride + 1:stride, g * ci:(g + 1) * ci]
            acc = acc + tap.reshape(-1, ci) @ w[g * co:(g + 1) * co, h, v].t()
        out.append(acc)
    return torch.cat(out, 1).view(x.shape[0], n, n, -1)


def _weight(l, cin):
    """The convolution weight of a layer as [cout, k, k, cin], from its rows."""
    k = l.k
    return l.p16["weight"].double()[:, :k * k * cin].reshape(-1, k, k, cin).clone().requires_grad_(True)


def _weight_grad(l, w):
    g = torch.zeros(l.p16["weight"].shape, dtype=torch.float64, device=w.device)
    g[:, :w[0].numel()] = w.grad.reshape(w.shape[0], -1)
    return g


def exact(case, seed):
    c = case
    k = c["kind"]
    if k == "step":
        return None               # random dropout masks, and roundings between eight layers
    if k == "clock":
        b = _batch(c, seed)
        w0, g = b["w0"].double(), b["update"].double()
        return [w0 - LR * (g + DECAY * w0)]
    if k == "input":
        b = _batch(c, seed)
        n, hw = c["crop"], (c["crop"] - 11) // 4 + 3
        y = torch.zeros(c["batch"], 3, 4 * hw, 4 * hw, dtype=torch.float64, device="cuda")
        mean = torch.tensor(MEAN, dtype=torch.float64, device="cuda").view(3, 1, 1)
        m = min(n, 4 * hw)
        for i, (h, w, mirror) in enumerate(b["aug"].tolist()):
            win = (b["x"][i, :, h:h + n, w:w + n].double() - mean) * SCALE
            y[i, :, :m, :m] = (win.flip(-1) if mirror else win)[:, :m, :m]
        y = y.view(-1, 3, hw, 4, hw, 4).permute(0, 2, 4, 3, 5, 1).reshape(-1, hw, hw, 48)
        return TF.pad(y, (0, 16))
    s = prepare(case, seed)
    layer, x = s["layer"], s["x"].double().requires_grad_(True)
    if k in ("fc", "head"):
        w, b = (layer.p16["weight"].double().requires_grad_(True), layer.p32["bias"].double().requires_grad_(True))
        y = TF.linear(x, w, b)
        if k == "head":
            loss = TF.cross_entropy(y, s["labels"])
            loss.backward()
            return [y.detach(), loss.detach().view(1), x.grad, w.grad, b.grad]
        y = torch.relu(y)
        y.backward(s["dy"].double())
        return [y.detach(), x.grad, w.grad, b.grad]
    to, back = (lambda t: t.permute(0, 3, 1, 2)), (lambda t: t.permute(0, 2, 3, 1))     # noqa: E731
    if k == "conv":
        w, b = _weight(layer, c["cin"] // c["groups"]), layer.p32["bias"].double().requires_grad_(True)
        y = torch.relu(_conv64(x, w, c["stride"], c["pad"], c["groups"]) + b)
        y.backward(s["dy"].double().view(y.shape))
        return [y.detach().reshape(-1, c["cout"]), x.grad, _weight_grad(layer, w), b.grad]

    def norm(l, t):
        g, b = (l.p32[n].double().requires_grad_(True) for n in ("gamma", "beta"))
        return torch.relu(TF.batch_norm(t, None, None, g, b, training=True, eps=l.eps)), g, b

    if k == "bn":
        y, g, b = norm(layer, to(x))
        y.backward(to(s["dy"].double().view(x.shape)))
        flat = x.detach().view(-1, c["c"])
        mean, var = flat.mean(0), flat.var(0, unbiased=False)
        return [back(y.detach()).reshape(-1, c["c"]), x.grad.view(-1, c["c"]), g.grad, b.grad, 0.1 * mean, 0.9 + 0.1 * var]
    if k == "inception":
        outs, grads = [], []
        for branch in layer.branches:
            h = to(x)
            for l in branch:
                if isinstance(l, Pool):
                    hw, p = c["hw"], TF.pad(h, (1, 1, 1, 1))        # 3 x 3 average, stride 1, zeros counted
                    h = sum(p[..., t // 3:t // 3 + hw, t % 3:t % 3 + hw] for t in range(9)) / 9
                elif isinstance(l, Conv2d):
                    w = _weight(l, h.shape[1])
                    h = to(_conv64(back(h), w, 1, l.pad))
                    grads.append((l, w))
                else:
                    h, g, b = norm(l, h)
                    grads += [(None, g), (None, b)]
            outs.append(h)
        y = torch.cat(outs, 1)
        y.backward(to(s["dy"].double().view(back(y).shape)))
        return ([back(y.detach()).reshape(-1, y.shape[1]), x.grad.view(-1, c["cin"])]
                + [g.grad if l is None else _weight_grad(l, g) for l, g in grads])
    # LRN + pooling: the maximum is taken over the bf16 values that the layer stores between the two
    y = TF.local_response_norm(to(x), 5, alpha=1e-4, beta=0.75, k=1.0)
    hw, out = c["hw"], s["dy"].shape[1]
    pad = (out - 1) * 2 + 3 - hw
    q = TF.pad(y.detach().to(BF).double(), (0, pad, 0, pad), value=-math.inf)
    best, code, pick = torch.full_like(q[:, :, :out, :out], -math.inf), None, 0
    full = TF.pad(y, (0, pad, 0, pad))
    for t in range(9):
        sl = (..., slice(t // 3, t // 3 + 2 * out - 1, 2), slice(t % 3, t % 3 + 2 * out - 1, 2))
        gt = q[sl] > best
        best = torch.where(gt, q[sl], best)
        code = torch.where(gt, t, code) if code is not None else torch.zeros_like(gt, dtype=torch.uint8)
        pick = torch.where(gt, full[sl], pick) if t else full[sl]
    pick.backward(to(s["dy"].double()))
    dx = torch.where(x > 0, x.grad, torch.zeros_like(x.grad)).detach()
    return [back(pick.detach()), None, dx, dx.sum((0, 1, 2))]
