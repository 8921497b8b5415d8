"""What the library is used for, as measurable cases.

A case is one call sequence through the public entry points (`tiny_cnn_b200.ops`,
`tiny_cnn_b200.network`) with everything a program holds before the call already on
the GPU.  `listed()` names the representative ones, `draw()` gives others of the same
ranges, `prepare()` / `run()` execute one, `work()` and `tolerance()` say what a pass
cannot do without and how far two correct implementations may differ.
"""
from __future__ import annotations

import math

import torch

from tiny_cnn_b200 import _lib as L
from tiny_cnn_b200 import network, ops

CONV_FLOPS_MAX = 2.0 * 256 * 56 * 56 * 64 * 64 * 9   # one pass of the largest layer of the sweep
CONV_VALUES_MAX = 2 * 256 * 56 * 56 * 64             # its input and output values
MAP_VALUES_MAX = 256 * 64 * 32 * 32


def listed():
    return [
        # one sample through the smallest network: what a serving call or an on-line prediction costs,
        # all launches and host work
        {"name": "lenet_predict_1", "kind": "predict", "net": "lenet", "batch": 1},
        # LeNet-5, mini-batch 16, mse + adagrad: the MNIST example's training step
        {"name": "lenet_train_16", "kind": "train", "net": "lenet", "batch": 16},
        # the CIFAR-10 network, mini-batch 256, cross entropy + adam: the headline training step
        {"name": "cifar_train_256", "kind": "train", "net": "cifar", "batch": 256},
        # the same network trained from page-locked host rows through fit(), one epoch whose last
        # mini-batch is short: upload, steps and outputs back, end to end
        {"name": "cifar_fit_2000", "kind": "fit", "net": "cifar", "batch": 256, "samples": 2000},
        # 784-4096-4096-10 perceptron, mini-batch 1024, cross entropy + momentum: large matrix products
        {"name": "mlp_train_1024", "kind": "train", "net": "mlp", "hidden": 4096, "batch": 1024},
        # the same form at a size a user picks for MNIST, no dimension a multiple of a tile
        {"name": "mlp_train_77", "kind": "train", "net": "mlp", "hidden": 500, "batch": 77},
        # single convolution layers, forward then backward (dX, dW, db): the two ends of the sweep
        {"name": "conv_56x64", "kind": "conv", "w": 56, "h": 56, "c": 64, "oc": 64, "k": 3, "stride": 1, "same": True,
         "batch": 256},
        {"name": "conv_14x256", "kind": "conv", "w": 14, "h": 14, "c": 256, "oc": 256, "k": 3, "stride": 1, "same": True,
         "batch": 256},
        # a downsampling layer at odd sizes: stride 2, rectangular, channel counts and batch off every tile
        {"name": "conv_stride2_odd", "kind": "conv", "w": 55, "h": 39, "c": 24, "oc": 40, "k": 5, "stride": 2, "same": False,
         "batch": 33},
        # quantized inference: the 5x5 convolution and the fully-connected layer behind its stride-2 form
        {"name": "qconv_28x32", "kind": "qconv", "w": 28, "h": 28, "c": 32, "oc": 64, "k": 5, "stride": 1, "batch": 128},
        {"name": "qfc_9216", "kind": "qfc", "in": 9216, "out": 256, "batch": 128},
        # the layers between convolutions, called one by one, forward and backward: batch normalization
        # (train phase), relu, 2x2 max pooling on 64 maps of 32x32
        {"name": "maps_32x64", "kind": "maps", "w": 32, "h": 32, "c": 64, "pool": 2, "batch": 256},
    ]


def _log(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["predict", "train", "train", "fit", "conv", "conv", "qconv", "qfc", "maps"])
    if kind in ("predict", "train"):
        net = rng.choice(["lenet", "cifar", "mlp"])
        case = {"kind": kind, "net": net, "batch": _log(rng, 1, 1024 if net == "mlp" else 256)}
        if net == "mlp":
            case["hidden"] = _log(rng, 64, 4096)
        return case
    if kind == "fit":
        batch = _log(rng, 8, 256)
        return {"kind": kind, "net": rng.choice(["lenet", "cifar"]), "batch": batch,
                "samples": batch * rng.randint(2, 7) + rng.randint(0, batch - 1)}
    if kind == "conv":
        k = rng.choice([3, 3, 5])
        stride = rng.choice([1, 1, 1, 2])
        case = {"kind": kind, "w": _log(rng, 7, 64), "h": _log(rng, 7, 64), "c": _log(rng, 3, 256), "oc": _log(rng, 6, 256),
                "k": k, "stride": stride, "same": rng.random() < 0.6, "batch": _log(rng, 1, 256)}
        while True:  # no dearer than the largest layer of the sweep; strided layers follow small maps in a network
            flops, values = _conv_size(case)
            if flops <= CONV_FLOPS_MAX / (1 if stride == 1 else 8) and values <= CONV_VALUES_MAX:
                return case
            if case["batch"] > 1:
                case["batch"] = (case["batch"] + 1) // 2
            else:
                case["c"] = (case["c"] + 1) // 2
    if kind == "qconv":
        w = _log(rng, 8, 28)  # maps no higher than wide: the range scan of the quantized layer asks for that
        return {"kind": kind, "w": w, "h": _log(rng, 8, w), "c": _log(rng, 3, 32), "oc": _log(rng, 6, 64),
                "k": rng.choice([3, 5]), "stride": rng.choice([1, 2]), "batch": _log(rng, 1, 128)}
    if kind == "qfc":
        return {"kind": kind, "in": _log(rng, 64, 9216), "out": _log(rng, 10, 256), "batch": _log(rng, 1, 128)}
    case = {"kind": "maps", "w": _log(rng, 6, 56), "h": _log(rng, 6, 56), "c": _log(rng, 3, 128), "pool": rng.choice([2, 2, 3]),
            "batch": _log(rng, 1, 256)}
    while case["batch"] * case["c"] * case["w"] * case["h"] > MAP_VALUES_MAX:
        case["batch"] = (case["batch"] + 1) // 2
    return case


# ---- geometry ---------------------------------------------------------------------------------
def _conv_out(n, k, stride, same):
    return -(-n // stride) if same else (n - k) // stride + 1


def _conv_size(case):
    """(flops of one pass, input + output values) of a convolution layer."""
    same = case.get("same", False)
    ow, oh = (_conv_out(case[s], case["k"], case["stride"], same) for s in ("w", "h"))
    out = case["batch"] * case["oc"] * ow * oh
    return 2.0 * out * case["c"] * case["k"] ** 2, out + case["batch"] * case["c"] * case["w"] * case["h"]


# per network: input values, output values, parameters, multiply-adds of one forward pass of one sample
def _net_size(case):
    if case["net"] == "lenet":
        taps = int(network.LENET_TABLE.sum())
        macs = 6 * 28 * 28 * 25 + taps * 10 * 10 * 25 + 120 * 16 * 25 + 120 * 10 + 6 * 28 * 28 + 16 * 10 * 10
        return 1024, 10, 6 * 26 + 4 * 6 + 6 + 16 * (6 * 25 + 1) + 4 * 16 + 16 + 120 * (16 * 25 + 1) + 10 * 121, macs
    if case["net"] == "cifar":
        macs = 32 * 1024 * 75 + 32 * 256 * 800 + 64 * 64 * 800 + 1024 * 64 + 640
        return 3072, 10, 32 * 76 + 32 * 801 + 64 * 801 + 64 * 1025 + 650, macs
    h = case["hidden"]
    return 784, 10, h * 785 + h * (h + 1) + 10 * (h + 1), h * 784 + h * h + h * 10


# ---- states -----------------------------------------------------------------------------------
_shared = {}


def _context():
    """The one context a program of single operator calls keeps."""
    if "ctx" not in _shared:
        _shared["ctx"] = ops.Context(0)
    return _shared["ctx"]


class _Owner:
    """Gives a network's device memory back when the last one who reads it is gone."""

    def __init__(self, net):
        self.net = net

    def __del__(self):
        self.net.close()


class _Values(network.DevicePtr):
    """Device values of a network, as torch takes them; keeps the network for as long as the tensor lives."""

    def __init__(self, owner, address, n):
        super().__init__(address, n)
        self.owner = owner


class _Net:
    """A network with its optimizer and data."""

    def __init__(self, case, seed):
        kind, self.batch = case["net"], case["batch"]
        if kind == "lenet":
            # targets and weights as the MNIST example has them
            net, self.loss, self.opt, low = network.lenet5(), L.LOSS_MSE, network.adagrad(0.01), -1.0
        elif kind == "cifar":
            # the rates of this and the next are small ones, so that thousands of steps on the same few
            # mini-batches leave the weights in the range they have in training
            net, self.loss, self.opt, low = network.cifar10_net(), L.LOSS_CROSS_ENTROPY, network.adam(1e-5), 0.0
        else:
            net, low = network.mlp(hidden=case["hidden"]), 0.0
            self.loss, self.opt = L.LOSS_CROSS_ENTROPY, network.momentum(0.01 / 1024, 0.9)
        net.build(self.batch)
        self.net, owner = net, _Owner(net)

        def values(address, n):
            return torch.as_tensor(_Values(owner, address, n), device="cuda")

        g = torch.Generator(device="cuda").manual_seed(seed)
        flat = torch.zeros(net.n_params, device="cuda")
        weights = [t for t in zip(net.tensors(), net.fan_in_out())]
        for (off, n), (fan_in, fan_out) in weights[0::2]:  # every layer here has a bias, which starts at zero
            flat[off:off + n].uniform_(-1.0, 1.0, generator=g).mul_(math.sqrt(6.0 / (fan_in + fan_out)))
        net.set_params(flat.cpu().numpy())
        rows = case.get("samples", self.batch)
        x = torch.empty(rows, net.in_dim, device="cuda")
        if kind == "cifar":
            x.normal_(generator=g)
        else:
            x.uniform_(low, 1.0, generator=g)
        t = torch.full((rows, net.out_dim), low, device="cuda")
        t[torch.arange(rows, device="cuda"), torch.randint(0, net.out_dim, (rows,), device="cuda", generator=g)] = 1.0
        lib, handle = net.lib, net.handle
        self.params = values(lib.b200_net_params_ptr(handle), net.n_params)
        self.grads = values(lib.b200_net_grads_ptr(handle), net.n_params)
        if case["kind"] == "fit":
            self.x, self.t = x.cpu().pin_memory(), t.cpu().pin_memory()
            self.out = torch.zeros(rows, net.out_dim).pin_memory()
        else:
            self.x, self.t = x, t
            self.out = values(lib.b200_net_output_ptr(handle), rows * net.out_dim).view(rows, net.out_dim)


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind in ("predict", "train", "fit"):
        state["net"] = _Net(case, seed)
        return state
    ctx = state["ctx"] = _context()
    g = torch.Generator(device="cuda").manual_seed(seed)
    B = case["batch"]

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    def uniform(n, low, high):
        return torch.empty(n, device="cuda").uniform_(low, high, generator=g)

    if kind in ("conv", "qconv"):
        w, h, c, oc, k = (case[s] for s in ("w", "h", "c", "oc", "k"))
        d = state["desc"] = ops.conv_params(w, h, c, k, k, oc, case.get("same", False), True, case["stride"], case["stride"])
        state["b"] = uniform(oc, -0.1, 0.1)
        if kind == "conv":
            bound = math.sqrt(6.0 / (k * k * c + (k // case["stride"]) ** 2 * oc))
            state["W"] = uniform(oc * c * k * k, -bound, bound)
            state["x"] = normal(B, c * w * h)
            state["dy"] = normal(B, oc * d.out_w * d.out_h)
        else:
            state["W"] = uniform(oc * c * k * k, -0.5, 0.5)
            state["x"] = uniform(B * c * w * h, -1.0, 1.0).view(B, -1)
    elif kind == "qfc":
        state["in"], state["out"] = case["in"], case["out"]
        state["W"] = uniform(case["in"] * case["out"], -0.5, 0.5)
        state["b"] = uniform(case["out"], -0.1, 0.1)
        state["x"] = uniform(B * case["in"], -1.0, 1.0).view(B, -1)
    else:
        w, h, c, p = (case[s] for s in ("w", "h", "c", "pool"))
        state["desc"] = d = ops.maxpool_params(w, h, c, p)
        state["c"], state["area"] = c, w * h
        state["x"] = normal(B, c * w * h)
        state["dy"] = normal(B, c * w * h)
        state["dp"] = normal(B, c * d.out_w * d.out_h)
    return state


def run(state):
    kind = state["kind"]
    if kind == "predict":
        s = state["net"]
        s.net.forward(s.x)
        return s.out
    if kind == "train":
        s = state["net"]
        s.net.train_onebatch(s.opt, s.x, s.t, s.loss)
        return {"out": s.out, "grads": s.grads, "params": s.params}
    if kind == "fit":
        s = state["net"]
        s.net.fit(s.opt, s.x, s.t, s.batch, 1, s.loss, outputs=s.out)
        return {"out": s.out, "params": s.params}
    ctx = state["ctx"]
    if kind == "conv":
        d, x, W = state["desc"], state["x"], state["W"]
        y = ops.conv2d_op(ctx, d, x, W, state["b"])
        dx, dW, db = ops.conv2d_grad_op(ctx, d, x, W, state["dy"])
        return {"y": y, "dx": dx, "dW": dW, "db": db}
    if kind == "qconv":
        return ops.quantized_conv2d(ctx, state["desc"], state["x"], state["W"], state["b"])
    if kind == "qfc":
        return ops.quantized_fully_connected(ctx, state["in"], state["out"], state["x"], state["W"], state["b"])
    x, dy = state["x"], state["dy"]
    y, mean, variance, stddev = ops.batch_normalization_forward(ctx, state["c"], state["area"], 1e-5, x)
    dx = ops.batch_normalization_backward(ctx, state["c"], state["area"], y, dy, stddev)
    r = ops.forward_activation(ctx, L.ACT_RELU, x)
    dr = ops.backward_activation(ctx, L.ACT_RELU, r, dy)
    p, arg = ops.maxpool_op(ctx, state["desc"], r)
    dp = ops.maxpool_grad_op(ctx, state["desc"], state["dp"], arg)
    return {"y": y, "mean": mean, "variance": variance, "dx": dx, "relu": r, "relu_dx": dr, "pool": p, "argmax": arg, "pool_dx": dp}


def work(case):
    kind, B = case["kind"], case["batch"]
    if kind in ("predict", "train", "fit"):
        n_in, n_out, n_params, macs = _net_size(case)
        if kind == "predict":
            return {"bytes": 4.0 * (B * (n_in + n_out) + n_params), "flops": 2.0 * B * macs}
        # a step reads its rows and writes the outputs; weights and optimizer state are read and written
        # (adam keeps two values a weight, the others one), gradients are written
        state = 2 if case["net"] == "cifar" else 1
        step = 4.0 * (B * (n_in + 2 * n_out) + n_params * (2 + 2 * state + 1))
        steps = -(-case["samples"] // B) if kind == "fit" else 1
        return {"bytes": steps * step, "flops": steps * 6.0 * B * macs}
    if kind in ("conv", "qconv"):
        flops, values = _conv_size(case)
        weights = case["oc"] * (case["c"] * case["k"] ** 2 + 1)
        if kind == "qconv":
            return {"bytes": 4.0 * (values + weights), "flops": flops}
        return {"bytes": 4.0 * (2 * values + 2 * weights), "flops": 3.0 * flops}
    if kind == "qfc":
        n, m = case["in"], case["out"]
        return {"bytes": 4.0 * (B * (n + m) + n * m + m), "flops": 2.0 * B * n * m}
    maps = B * case["c"] * case["w"] * case["h"]
    pooled = B * case["c"] * (case["w"] // case["pool"]) * (case["h"] // case["pool"])
    # normalization x -> y and y, dy -> dx; relu the same; pooling in -> values + indices and back
    return {"bytes": 4.0 * (2 * maps + 3 * maps + 2 * maps + 3 * maps + (maps + 2 * pooled) + (maps + 2 * pooled)), "flops": 20.0 * maps}


def tolerance(case):
    kind = case["kind"]
    if kind in ("qconv", "qfc"):
        return "exact"  # whole-number accumulation and the reference's own double-precision range arithmetic
    if kind == "maps":
        return {"rel": 1e-5, "max": 1e-4}  # 32-bit sums over up to 262144 values; the rest is exact
    if kind == "conv":
        # 32-bit sums, of up to 800000 products for dW: the library's own matrix and scalar kernels differ
        # there by 2e-4
        return {"rel": 3e-4, "max": 2e-3}
    if kind == "predict":
        return {"rel": 3e-5, "max": 3e-4}
    if kind == "fit":
        return {"rel": 1e-3, "max": 2e-2}
    # gradients of one step: two summation orders agree on an output to 1e-6, but a relu gate or a pooling
    # winner decided by such a difference moves one position's whole contribution (the library's matrix and
    # scalar kernels: 2.6e-3, largest 0.25)
    return {"rel": 5e-3, "max": 0.5}
