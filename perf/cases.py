"""The work that users have this library do, as cases that can be timed and compared.

Four kinds, all through the public Python front end:

* ``infer``  a network's forward pass over a batch: LeNet5 (the benchmark network) and the wide
             conv stack, from device tensors (``Model.forward_device``), from pinned host images
             (``Model.infer``) or from pinned u8 images (``Model.infer_u8``);
* ``train``  one SGD step: host batches through ``Model.train_step``, or device batches through
             ``Model.train_forward_backward`` + ``Model.apply_update`` (the data-parallel form);
* ``dot``    a product in one of the three layouts that forward and backward passes use;
* ``conv``   one Conv2 -> Relu -> MaxPool2 stage called operator by operator, forward and every
             backward edge, with the convolution options of the layer builder.
"""
import math

import torch

import autograph_b200 as ag
from autograph_b200 import data_parallel

_DTYPE = {"f32": torch.float32, "bf16": torch.bfloat16}
_SIZE = {"f32": 4, "bf16": 2}
_NETS = {"lenet5": ag.LENET5_SPEC, "wide": ag.WIDE_STACK_SPEC}
_IMAGE = {"lenet5": (1, 28, 28), "wide": (3, 64, 64)}
_LR = 0.01


def listed():
    return [
        # One image of a request that somebody waits for: copies, launches and waits are the cost.
        dict(name="infer_f32_1_host", kind="infer", net="lenet5", dtype="f32", source="host", batch=1),
        # The benchmark's step, images resident on the device.
        dict(name="infer_f32_1000", kind="infer", net="lenet5", dtype="f32", source="device", batch=1000),
        # The same step as a caller makes it: host images in, host logits out.
        dict(name="infer_f32_1000_host", kind="infer", net="lenet5", dtype="f32", source="host", batch=1000),
        # A whole dataset scored in one call.
        dict(name="infer_bf16_65536", kind="infer", net="lenet5", dtype="bf16", source="device", batch=65536),
        # The training benchmark: small batches from host memory, one loss read per step.
        dict(name="train_f32_100_host", kind="train", net="lenet5", dtype="f32", source="host", batch=100,
             momentum=0.0),
        # Larger-batch training on resident data with momentum, the batch not a round number.
        dict(name="train_bf16_509", kind="train", net="lenet5", dtype="bf16", source="device", batch=509,
             momentum=0.9),
        # Training a network whose layers fill the chip.
        dict(name="train_wide_bf16_256", kind="train", net="wide", dtype="bf16", source="device", batch=256,
             momentum=0.0),
        # A small Dense layer's product as an operator call.
        dict(name="dot_f32_100x256x128", kind="dot", dtype="f32", m=100, k=256, n=128, layout="nn"),
        # A weight-gradient layout at the largest f32 size in common use.
        dict(name="dot_f32_4096_tn", kind="dot", dtype="f32", m=4096, k=4096, n=4096, layout="tn"),
        # The bf16 product the library is judged by.
        dict(name="dot_bf16_4096_nn", kind="dot", dtype="bf16", m=4096, k=4096, n=4096, layout="nn"),
        # Sizes as data brings them: no dimension a multiple of anything.
        dict(name="dot_bf16_777x1009x333_nt", kind="dot", dtype="bf16", m=777, k=1009, n=333, layout="nt"),
        # A padded convolution stage of a mid-sized network in f32, every edge.
        dict(name="conv_f32_16to32_3x3", kind="conv", dtype="f32", batch=64, ic=16, hw=32, oc=32, filter=3,
             padding=1, stride=1),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["infer", "train", "dot", "conv"])
    dtype = rng.choice(["f32", "bf16"])
    if kind == "infer":
        net = rng.choice(["lenet5", "lenet5", "lenet5", "wide"])
        source = rng.choice(["device", "device", "host", "host_u8"] if net == "lenet5" else ["device", "host"])
        most = (65536 if source == "device" else 16384) if net == "lenet5" else (256 if dtype == "bf16" else 64)
        return dict(kind=kind, net=net, dtype=dtype, source=source, batch=_log_uniform(rng, 1, most))
    if kind == "train":
        net = rng.choice(["lenet5", "lenet5", "lenet5", "wide"])
        most = 4096 if net == "lenet5" else (256 if dtype == "bf16" else 48)
        return dict(kind=kind, net=net, dtype=dtype, source=rng.choice(["device", "host"]),
                    batch=_log_uniform(rng, 8, most), momentum=rng.choice([0.0, 0.9]))
    if kind == "dot":
        # half of the products have sizes a network's designer picks (multiples of 16), half
        # have whatever the data brings; at most as large as the largest listed one
        step = rng.choice([1, 16])
        while True:
            m, k, n = (max(step, _log_uniform(rng, 16, 8192) // step * step) for _ in range(3))
            if m * k * n <= 4096 ** 3 and m * n <= 4096 ** 2:
                return dict(kind=kind, dtype=dtype, m=m, k=k, n=n, layout=rng.choice(["nn", "nt", "tn"]))
    while True:
        f = rng.choice([3, 3, 5])
        c = dict(kind=kind, dtype=dtype, batch=_log_uniform(rng, 4, 256), ic=rng.choice([1, 3, 6, 16, 32, 64]),
                 hw=rng.randint(10, 64), oc=rng.choice([6, 16, 32, 64, 96, 128]), filter=f,
                 padding=rng.choice([0, f // 2]), stride=rng.choice([1, 1, 1, 2]))
        if work(c)["flops"] <= 2e10:
            return c


def _out_hw(case):
    return (case["hw"] + 2 * case["padding"] - case["filter"]) // case["stride"] + 1


_device = None


def _dev():
    """The one device object that a program keeps."""
    global _device
    if _device is None:
        _device = ag.Device(0)
    torch.cuda.set_stream(_device.stream)
    return _device


def prepare(case, seed):
    dev = _dev()
    gen = torch.Generator(device=dev.torch_device).manual_seed(seed)
    dtype = _DTYPE[case["dtype"]]

    def uniform(shape, lo, hi):
        t = torch.rand(shape, generator=gen, device=dev.torch_device)
        return t.mul_(hi - lo).add_(lo).to(dtype)

    def normal(shape):
        return torch.randn(shape, generator=gen, device=dev.torch_device).to(dtype)

    s = dict(case=case, dev=dev)
    if case["kind"] == "dot":
        m, k, n, layout = case["m"], case["k"], case["n"], case["layout"]
        a = uniform((k, m) if layout[0] == "t" else (m, k), -1.0, 1.0)
        b = uniform((n, k) if layout[1] == "t" else (k, n), -1.0, 1.0)
        s["a"] = a.t() if layout[0] == "t" else a
        s["b"] = b.t() if layout[1] == "t" else b
        return s
    if case["kind"] == "conv":
        bs, ic, hw, oc, f, o = (case["batch"], case["ic"], case["hw"], case["oc"], case["filter"], _out_hw(case))
        a = math.sqrt(2.0 / (ic * f * f))
        s["x"], s["w"], s["bias"] = normal((bs, ic, hw, hw)), uniform((oc, ic, f, f), -a, a), uniform((oc,), -a, a)
        # what an earlier forward pass kept for the backward edges, and the gradient that arrives
        s["pre"] = normal((bs, oc, o, o))
        s["act"] = s["pre"].clamp(min=0)
        s["dp"] = normal((bs, oc, o // 2, o // 2))
        s["opt"] = dict(padding=(case["padding"],) * 2, stride=(case["stride"],) * 2)
        return s

    s["model"] = model = ag.Model(dev, _NETS[case["net"]], dtype, seed=seed)
    shape = (case["batch"],) + _IMAGE[case["net"]]
    x = uniform(shape, 0.0, 1.0) if case["net"] == "lenet5" else normal(shape)
    if case["kind"] == "infer":
        if case["source"] == "device":
            s["x"] = x
            s["out"] = dev.empty((case["batch"], model.out_features), dtype)
        else:
            if case["source"] == "host_u8":
                x = torch.randint(0, 256, shape, generator=gen, device=dev.torch_device, dtype=torch.uint8)
            s["x"] = x.cpu().pin_memory()
            s["out"] = torch.empty((case["batch"], model.out_features), dtype=dtype).pin_memory()
        return s

    t = torch.randint(0, 10, (case["batch"],), generator=gen, device=dev.torch_device, dtype=torch.uint8)
    model.set_sgd(case["momentum"] or None)
    # a program that clips, logs or all-reduces gradients keeps a view of the model's bucket
    _, ptr, length = model.train_forward_backward(x[:1].contiguous(), t[:1].contiguous(), sync=False)
    s["grads"] = data_parallel.bucket_view(ptr, length, dtype, dev.torch_device)
    s["grads"].model = model  # the bucket is the model's memory: the view keeps its owner alive
    if case["source"] == "host":
        x, t = x.cpu().pin_memory(), t.cpu().pin_memory()
    s["x"], s["t"] = x, t
    return s


def run(state):
    case, dev = state["case"], state["dev"]
    if case["kind"] == "dot":
        return dev.dot(state["a"], state["b"])
    if case["kind"] == "infer":
        model = state["model"]
        if case["source"] == "device":
            return model.forward_device(state["x"], state["out"])
        if case["source"] == "host":
            return model.infer(state["x"], state["out"])
        return model.infer_u8(state["x"], out_host=state["out"])
    if case["kind"] == "train":
        model = state["model"]
        if case["source"] == "host":
            return {"loss": model.train_step(state["x"], state["t"], _LR), "grads": state["grads"]}
        model.train_forward_backward(state["x"], state["t"], sync=False)
        model.apply_update(_LR)
        return {"grads": state["grads"]}
    x, w, opt, f, hw = state["x"], state["w"], state["opt"], case["filter"], case["hw"]
    y = dev.conv2_forward(x, w, state["bias"], relu=True, **opt)
    p = dev.max_pool2(y)
    dr = dev.max_pool2_backward_from_input(state["act"], state["dp"])
    dy = dev.relu_backward(state["pre"], dr)
    db = dev.bias_grad(dy)
    dw = dev.conv2_backward_weight(x, dy, (f, f), **opt)
    dx = dev.conv2_backward_input(w, dy, (hw, hw), **opt)
    return {"y": y, "p": p, "db": db, "dw": dw, "dx": dx}


def _net_work(net):
    """Per image: forward flops, those of the first convolution, values in and out; parameters."""
    c, h, w = _IMAGE[net]
    values_in, flops, first, params = c * h * w, 0, 0, 0
    for layer in _NETS[net]:
        if layer[0] == "conv":
            _, ic, oc, (fh, fw), bias = layer
            h, w, c = h - fh + 1, w - fw + 1, oc
            fl = 2 * h * w * oc * ic * fh * fw
            first = first or fl
            flops += fl
            params += oc * ic * fh * fw + (oc if bias else 0)
        elif layer[0] == "pool":
            h, w = h // layer[1][0], w // layer[1][1]
        elif layer[0] == "dense":
            flops += 2 * layer[1] * layer[2]
            params += layer[1] * layer[2] + (layer[2] if layer[3] else 0)
            out = layer[2]
    return flops, first, values_in, out, params


def work(case):
    es = _SIZE[case["dtype"]]
    if case["kind"] == "dot":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": es * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    if case["kind"] == "conv":
        bs, ic, hw, oc, f, o = (case["batch"], case["ic"], case["hw"], case["oc"], case["filter"], _out_hw(case))
        x, w, y, p = bs * ic * hw * hw, oc * ic * f * f, bs * oc * o * o, bs * oc * (o // 2) ** 2
        # forward: x, w in, y and p out; backward: both activations, dp, x and w in, dx and dw out
        return {"bytes": es * (3 * x + 3 * w + 3 * y + 2 * p + 2 * oc), "flops": 3 * 2 * y * ic * f * f}
    flops, first, values_in, out, params = _net_work(case["net"])
    bs = case["batch"]
    if case["kind"] == "infer":
        return {"bytes": bs * (values_in * (1 if case["source"] == "host_u8" else es) + out * es) + params * es,
                "flops": bs * flops}
    # forward and both gradients of every product, except the first layer's input gradient; the
    # parameters are read and written once, their gradients written (and the velocity updated)
    return {"bytes": bs * (values_in * es + 1) + params * es * (5 if case["momentum"] else 3),
            "flops": bs * (3 * flops - first)}


def tolerance(case):
    f32 = case["dtype"] == "f32"
    if case["kind"] == "train":
        # Relu and pool gates turn on the last bit of an activation: in f32 one of the about 5000
        # per image moves now and then, and with it one row of a weight gradient.
        return {"rel": 1e-3, "max": 0.5} if f32 else {"rel": 1e-2, "max": 0.9}
    return {"rel": 1e-5} if f32 else {"rel": 1e-2}
