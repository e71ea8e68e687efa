"""The work whose time is tracked, each case one call a user's program makes again and again.

Four kinds, all through the public entry points:

* ``train``: one training step of a network, ``Model.train_batch`` (forward, loss, backward, SGD update);
* ``infer``: one batch through a network in evaluation, ``Model.evaluate_batch`` with the fused inference layers;
* ``conv``:  one Conv2D layer's forward pass, weight + bias gradient and input gradient through the C ABI;
* ``fc``:    one FC layer's forward and backward pass through the C ABI.

Networks and sizes are those of the benchmark (``bench.py``), of the shape sweep (batch 32, images of 7 to 112, 64 to
512 channels, filters of 1 to 7, stride 1 and 2, both layouts, float32 and float64) and of the model tests, plus the
small images and channel counts that are not multiples of the tile sizes which users bring along.
"""
import ctypes
import math

import numpy as np
import torch

from pydtnn_b200 import _lib, nets
from pydtnn_b200.layers import FC, Conv2D, Flatten, Input, MaxPool2D
from pydtnn_b200.model import Model
from pydtnn_b200.optimizers import SGD

_TORCH = {"float32": torch.float32, "float64": torch.float64}


def _conv(name, n, h, w, ci, co, k, stride, dtype, layout):
    return dict(name=name, kind="conv", n=n, h=h, w=w, ci=ci, co=co, k=k, stride=stride, dtype=dtype, layout=layout)


def _net(name, kind, net, n, hw, layout, dtype="float32", width=0):
    return dict(name=name, kind=kind, net=net, n=n, hw=hw, layout=layout, dtype=dtype, width=width)


def listed():
    return [
        # training jobs: ImageNet classification (the benchmark's configuration), the same network in the layout the
        # reference's GPU back end defaults to, a 32x32-image classifier, a digit classifier, and a double-precision
        # run of the kind used to check a model's gradients
        _net("train_resnet50_b64", "train", "resnet50", 64, 224, "NHWC"),
        _net("train_resnet50_nchw_b32", "train", "resnet50", 32, 224, "NCHW"),
        _net("train_vgg16bn_32px_b64", "train", "vgg16bn", 64, 32, "NHWC"),
        _net("train_digits_b64", "train", "digits", 64, 28, "NCHW"),
        _net("train_resnet_f64_b32", "train", "resnet_small", 32, 32, "NHWC", "float64", 16),
        # serving: single images (latency), and full batches of the benchmark's inference configuration
        _net("infer_resnet50_b1", "infer", "resnet50", 1, 224, "NHWC"),
        _net("infer_alexnet_nchw_b64", "infer", "alexnet", 64, 227, "NCHW"),
        # single layers: the benchmark's single-layer configuration, two points of the shape sweep, and a detection
        # style feature map with channel counts that fit no tile
        _conv("conv_32px_64_64_k3", 64, 32, 32, 64, 64, 3, 1, "float32", "NHWC"),
        _conv("conv_f64_28px_256_256_k3", 32, 28, 28, 256, 256, 3, 1, "float64", "NHWC"),
        _conv("conv_nchw_56px_128_256_k5_s2", 32, 56, 56, 128, 256, 5, 2, "float32", "NCHW"),
        _conv("conv_ragged_75x43_40_72_k3", 9, 75, 43, 40, 72, 3, 1, "float32", "NHWC"),
        # the classifier head of the ImageNet networks (1000 classes fit no tile either)
        dict(name="fc_b64_4096_1000", kind="fc", n=64, n_in=4096, n_out=1000, dtype="float32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("conv", "fc", "train", "infer"), (5, 2, 3, 3))[0]
    if kind == "conv":
        while True:
            dtype = rng.choices(("float32", "float64"), (3, 1))[0]
            h = _log_int(rng, 7, 112)
            w = h if rng.random() < 0.6 else _log_int(rng, 7, 112)
            # half of the channel counts are the sweep's powers of two, the other half any number
            ci, co = (rng.choice((64, 128, 256, 512)) if rng.random() < 0.5 else _log_int(rng, 3, 512) for _ in "io")
            c = dict(kind="conv", n=_log_int(rng, 1, 64), h=h, w=w, ci=ci, co=co, k=rng.choice((1, 3, 3, 5, 7)),
                     stride=rng.choice((1, 1, 2)), dtype=dtype, layout=rng.choice(("NHWC", "NCHW")))
            if 1e7 < work(c)["flops"] < (3e11 if dtype == "float32" else 5e10):
                return c
    if kind == "fc":
        dtype = rng.choices(("float32", "float64"), (3, 1))[0]
        return dict(kind="fc", n=_log_int(rng, 1, 256), n_in=_log_int(rng, 64, 9216), n_out=_log_int(rng, 10, 4096), dtype=dtype)
    layout = rng.choice(("NHWC", "NCHW"))
    net = rng.choice(("resnet50", "resnet_small", "vgg16bn", "digits") + (("alexnet",) if kind == "infer" else ()))
    n = _log_int(rng, 1 if kind == "infer" else 8, 64)
    if net == "resnet50":
        # images of 64 to 224, and no more of them than the listed cases have
        hw = 32 * rng.randint(2, 7)
        return dict(kind=kind, net=net, n=min(n, 48) if layout == "NHWC" else min(n, 32), hw=hw, layout=layout, dtype="float32", width=0)
    if net == "resnet_small":
        dtype = rng.choice(("float32", "float64"))
        return dict(kind=kind, net=net, n=n, hw=4 * rng.randint(8, 16), layout=layout, dtype=dtype, width=rng.choice((8, 16, 20, 32, 64 if dtype == "float32" else 24)))
    hw = {"vgg16bn": 32 * rng.randint(1, 2), "digits": rng.randint(20, 40), "alexnet": 227}[net]
    return dict(kind=kind, net=net, n=n, hw=hw, layout=layout, dtype="float32", width=0)


# ---- what a pass cannot do without -----------------------------------------------------------------------------

def _out(size, k, stride, pad):
    return (size + 2 * pad - k) // stride + 1


def _net_gemms(c):
    """[(output rows, multiplications per output value, output channels, has batch norm)] of the network's Conv2D and
    FC layers, in order."""
    n, hw, out = c["n"], c["hw"], []

    def conv(s, ci, co, k, stride, pad, bn=True):
        s = _out(s, k, stride, pad)
        out.append((n * s * s, ci * k * k, co, bn))
        return s

    def fc(i, o):
        out.append((n, i, o, False))

    if c["net"] in ("resnet50", "resnet_small"):
        stages = [[64, 3, 1], [128, 4, 2], [256, 6, 2], [512, 3, 2]] if c["net"] == "resnet50" else [[c["width"], 2, 1], [2 * c["width"], 2, 2]]
        s = _out(conv(hw, 3, 64, 7, 2, 3, False), 3, 2, 1)
        ci = 64
        for f, blocks, stride in stages:
            for b in range(blocks):
                st = stride if b == 0 else 1
                conv(s, ci, f, 1, 1, 0)
                s2 = conv(s, f, f, 3, st, 1)
                conv(s2, f, 4 * f, 1, 1, 0)
                if b == 0:
                    conv(s, ci, 4 * f, 1, st, 0)
                s, ci = s2, 4 * f
        fc(ci, _classes(c))
    elif c["net"] == "vgg16bn":
        s, ci = hw, 3
        for f, convs in ((64, 2), (128, 2), (256, 3), (512, 3), (512, 3)):
            for _ in range(convs):
                s = conv(s, ci, f, 3, 1, 1)
                ci = f
            s //= 2
        fc(s * s * ci, 4096), fc(4096, 4096), fc(4096, _classes(c))
    elif c["net"] == "alexnet":
        s = _out(conv(hw, 3, 96, 11, 4, 0, False), 3, 2, 0)
        s = _out(conv(s, 96, 256, 5, 1, 2, False), 3, 2, 0)
        for ci, co in ((256, 384), (384, 384), (384, 256)):
            s = conv(s, ci, co, 3, 1, 1, False)
        fc(_out(s, 3, 2, 0) ** 2 * 256, 4096), fc(4096, 4096), fc(4096, _classes(c))
    else:
        s = conv(hw, 1, 16, 3, 1, 1, False) // 2
        s = conv(s, 16, 32, 3, 1, 1, False) // 2
        fc(s * s * 32, 128), fc(128, 10)
    return out


def work(case):
    size = 4 if case["dtype"] == "float32" else 8
    if case["kind"] == "conv":
        n, h, w, ci, co, k, st = (case[x] for x in ("n", "h", "w", "ci", "co", "k", "stride"))
        rows = n * _out(h, k, st, k // 2) * _out(w, k, st, k // 2)
        x, y, f = n * h * w * ci, rows * co, ci * k * k * co
        return {"bytes": size * (2 * x + 2 * y + 2 * f + 2 * co), "flops": 3 * 2 * rows * ci * k * k * co}
    if case["kind"] == "fc":
        n, i, o = case["n"], case["n_in"], case["n_out"]
        return {"bytes": size * (2 * n * i + 2 * n * o + 2 * i * o + 2 * o), "flops": 3 * 2 * n * i * o}
    gemms = _net_gemms(case)
    channels = 1 if case["net"] == "digits" else 3
    x = case["n"] * case["hw"] ** 2 * channels
    params = sum(k * co + co * (3 if bn else 1) for _, k, co, bn in gemms)
    fwd = sum(2 * m * k * co for m, k, co, _ in gemms)
    if case["kind"] == "infer":
        return {"bytes": size * (x + params + case["n"] * gemms[-1][2]), "flops": fwd}
    # training: the layers' outputs are more than the chip holds, so each is written once and read once in backward;
    # parameters and velocities are read and written, gradients written; no input gradient for the first layer
    kept = sum(m * co for m, _, co, _ in gemms)
    first = 2 * gemms[0][0] * gemms[0][1] * gemms[0][2]
    return {"bytes": size * (x + 2 * kept + 5 * params), "flops": 3 * fwd - first}


def tolerance(case):
    f64 = case["dtype"] == "float64"
    if case["kind"] in ("conv", "fc"):
        # the bars of the parity tests: one dot product per value
        return {"rel": 1e-12, "max": 1e-10} if f64 else {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "infer":
        return {"rel": 1e-11, "max": 1e-9} if f64 else {"rel": 2e-4, "max": 1e-2}
    # A training step chains every layer's rounding through batch norms and ReLU masks and back: a value within rounding
    # of zero takes the other side of its mask and moves whole gradient entries.  Measured between two float32 engines,
    # and for a change of 1e-7 in the input: 2e-3 to 1e-2 of a gradient's norm, single entries by up to half of it.
    return {"rel": 1e-8, "max": 1e-4} if f64 else {"rel": 2e-2, "max": 0.9}


# ---- inputs and passes -----------------------------------------------------------------------------------------

def _classes(c):
    return 1000 if c["net"] in ("resnet50", "alexnet") else 10


def _build(c, seed, **flags):
    np.random.seed(seed % (1 << 32))
    model = Model(batch_size=c["n"], tensor_format=c["layout"], dtype=np.dtype(c["dtype"]).type, **flags)
    if c["net"] == "resnet50":
        nets.create_resnet50_imagenet(model, input_hw=c["hw"])
    elif c["net"] == "resnet_small":
        nets.create_resnet50_imagenet(model, input_hw=c["hw"], nclasses=10, layout=[[c["width"], 2, 1], [2 * c["width"], 2, 2]])
    elif c["net"] == "vgg16bn":
        nets.create_vgg16bn_imagenet(model, input_hw=c["hw"], nclasses=10)
    elif c["net"] == "alexnet":
        nets.create_alexnet_imagenet(model)
    else:
        model.add(Input(shape=(c["hw"], c["hw"], 1)))
        for co in (16, 32):
            model.add(Conv2D(nfilters=co, filter_shape=(3, 3), padding=1, activation="relu", weights_initializer="he_uniform"))
            model.add(MaxPool2D(pool_shape=(2, 2), stride=2))
        model.add(Flatten())
        model.add(FC(shape=(128,), activation="relu", weights_initializer="he_uniform"))
        model.add(FC(shape=(10,), activation="softmax", weights_initializer="he_uniform"))
    return model


def _randn(gen, shape, dtype, scale=1.0):
    return torch.randn(shape, generator=gen, dtype=_TORCH[dtype], device="cuda") * scale


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if c["kind"] == "conv":
        return _prepare_conv(c, gen)
    if c["kind"] == "fc":
        return _prepare_fc(c, gen)
    training = c["kind"] == "train"
    flags = dict(enable_fused_bn_relu=True) if training else dict(enable_fused_conv_relu=True, enable_fused_conv_bn=True, enable_fused_conv_bn_relu=True)
    model = _build(c, seed, **flags)
    shape = (c["n"], *model.layers[0].shape)
    if c["net"] in ("alexnet", "digits"):                      # pixels in [0, 1]
        x = torch.randint(0, 256, shape, generator=gen, device="cuda").to(_TORCH[c["dtype"]]) / 255
    else:                                                      # normalised images
        x = _randn(gen, shape, c["dtype"])
    labels = torch.randint(0, _classes(c), (c["n"],), generator=gen, dtype=torch.int32, device="cuda")
    norms = [l for l in model.get_all_layers() if l.canonical_name == "BatchNormalization"]
    state = dict(c, model=model, x=x, labels=labels, norms=norms, optimizer=SGD(learning_rate=1e-5, momentum=0.9))
    for l in model.get_all_layers():
        # residual branches start small, as is usual for networks of this depth
        if l.canonical_name == "AdditionBlock":
            l.paths[0][-1].gamma.ary.t.fill_(0.2)
    if not training and norms:
        # a trained network's running statistics: those of its own activations, not the initial zeros
        momentum = [l.momentum for l in norms]
        for l in norms:
            l.momentum = 0.0
        model.train_batch(x, labels, SGD(learning_rate=0.0, momentum=0.0))
        for l, m in zip(norms, momentum):
            l.momentum = m
            l.running_var.ary.t.clamp_(min=0.1)
    return state


def _prepare_conv(c, gen):
    nhwc = c["layout"] == "NHWC"
    k, st, dt = c["k"], c["stride"], c["dtype"]
    ho, wo = _out(c["h"], k, st, k // 2), _out(c["w"], k, st, k // 2)
    act = (lambda h, w, ch: (c["n"], h, w, ch) if nhwc else (c["n"], ch, h, w))
    filt = (c["co"], k, k, c["ci"]) if nhwc else (c["co"], c["ci"], k, k)
    desc = _lib.ConvDesc(_lib.LAYOUT_NHWC if nhwc else _lib.LAYOUT_NCHW, _lib.dtype_code(dt), _lib.W_KRSC if nhwc else _lib.W_KCRS,
                         _lib.ENGINE_AUTO, c["n"], c["h"], c["w"], c["ci"], c["co"], k, k, k // 2, k // 2, st, st, 1, 1)
    s = dict(c, desc=desc, x=_randn(gen, act(c["h"], c["w"], c["ci"]), dt), dy=_randn(gen, act(ho, wo, c["co"]), dt),
             w=_randn(gen, filt, dt, math.sqrt(2.0 / (c["ci"] * k * k))), b=_randn(gen, (c["co"],), dt))
    s.update(y=torch.empty_like(s["dy"]), dx=torch.empty_like(s["x"]), dw=torch.empty_like(s["w"]), db=torch.empty_like(s["b"]))
    need = max(_lib.lib().b2c_conv_workspace_bytes(ctypes.byref(desc), p) for p in (_lib.PASS_FPROP, _lib.PASS_DGRAD, _lib.PASS_WGRAD))
    s["ws"] = torch.empty(max(int(need), 256), dtype=torch.uint8, device="cuda")
    return s


def _prepare_fc(c, gen):
    dt = c["dtype"]
    s = dict(c, x=_randn(gen, (c["n"], c["n_in"]), dt), dy=_randn(gen, (c["n"], c["n_out"]), dt),
             w=_randn(gen, (c["n_in"], c["n_out"]), dt, math.sqrt(2.0 / c["n_in"])), b=_randn(gen, (c["n_out"],), dt))
    s.update(y=torch.empty_like(s["dy"]), dx=torch.empty_like(s["x"]), dw=torch.empty_like(s["w"]), db=torch.empty_like(s["b"]))
    need = _lib.lib().b2c_fc_workspace_bytes(_lib.dtype_code(dt), c["n"], c["n_in"], c["n_out"], _lib.ENGINE_AUTO)
    s["ws"] = torch.empty(max(int(need), 256), dtype=torch.uint8, device="cuda")
    return s


def run(state):
    s = state
    if s["kind"] == "train":
        m = s["model"]
        loss = m.train_batch(s["x"], s["labels"], s["optimizer"])
        out = {"totals": loss.totals.t, "probabilities": m.layers[-1].y.ary.t}
        for i, ch in enumerate(m.arena.chunks):
            out["parameters%d" % i], out["gradients%d" % i], out["velocities%d" % i] = ch.w[:ch.used], ch.dw[:ch.used], ch.v[:ch.used]
        # running averages of the batch norms, as many as an answer may hold
        out["running"] = [t.ary.t for l in s["norms"] for t in (l.running_mean, l.running_var)][:48]
        return out
    if s["kind"] == "infer":
        return s["model"].evaluate_batch(s["x"]).ary.t
    L = _lib.lib()
    stream = torch.cuda.current_stream().cuda_stream
    p = {k: s[k].data_ptr() for k in ("x", "dy", "w", "b", "y", "dx", "dw", "db", "ws")}
    nbytes = s["ws"].numel()
    if s["kind"] == "conv":
        d = ctypes.byref(s["desc"])
        _lib.check(L.b2c_conv_fprop(d, p["x"], p["w"], p["b"], None, 0, p["y"], p["ws"], nbytes, stream))
        _lib.check(L.b2c_conv_wgrad(d, p["x"], p["dy"], p["dw"], p["db"], p["ws"], nbytes, stream))
        _lib.check(L.b2c_conv_dgrad(d, p["dy"], p["w"], p["dx"], p["ws"], nbytes, stream))
    else:
        shape = (_lib.dtype_code(s["dtype"]), _lib.ENGINE_AUTO, s["n"], s["n_in"], s["n_out"])
        _lib.check(L.b2c_fc_forward(*shape, p["x"], p["w"], p["b"], p["y"], p["ws"], nbytes, stream))
        _lib.check(L.b2c_fc_backward(*shape, p["x"], p["dy"], p["w"], p["dw"], p["db"], p["dx"], p["ws"], nbytes, stream))
    return {k: s[k] for k in ("y", "dw", "db", "dx")}
