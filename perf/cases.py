"""Performance cases of the framework: the calls a training or inference program makes, over the range of sizes it makes
them at, through the package's public entry points (bridges, networks and the C ABI's host-buffer calls).

A case is a dict of plain values.  `kind` says which entry point it exercises:
  conv       ConvolutionBridge: "train" = forward and backward (dX, dW, db), "forward" = forward with the ReLU folded in,
             "fused" = forward with ReLU, max pooling, and the backward pass with pooling and ReLU masks folded in
  conv_host  the host-buffer calls (cct_conv_forward_host / cct_conv_backward_host) on pinned host memory
  fc         FullyConnectedBridge: "train" or "forward"
  layers     the parameter-free bridges between two convolutions: ReLU, max pooling, LRN, forward and backward
  caffenet   one training iteration (forward, backward, SGD) of the network description in caffecontroll_b200/nets
  small_net  one training iteration of a two-convolution, two-inner-product network of LeNet's form
All tensors are fp32 and live on the GPU unless the kind says otherwise.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

from caffecontroll_b200 import Context, ConvolutionBridge, FullyConnectedBridge, Layer, LogicalCube, capi
from caffecontroll_b200.layers import LRNBridge, MaxPoolingBridge, ReLUBridge
from caffecontroll_b200.net import load_net

NETS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caffecontroll_b200", "nets")


def _conv(name, mode, B, D, n, o, k, s, p, g, x):
    return {"name": name, "kind": "conv", "mode": mode, "B": B, "D": D, "n": n, "o": o, "k": k, "s": s, "p": p, "g": g, "x": x}


def listed():
    return [
        # The smallest training call: LeNet's first layer on one mini-batch of digits; latency and launches count.
        _conv("lenet_conv1_b64", "train", 64, 1, 28, 20, 5, 1, 0, 1, "uniform"),
        # One image through a 3x3 layer (CaffeNet conv3): inference latency.
        _conv("conv3_forward_b1", "forward", 1, 256, 13, 384, 3, 1, 1, 1, "relu"),
        # A layer nobody tuned for: odd batch, channels that are not multiples of 16, stride 2.
        _conv("conv_ragged_b37", "train", 37, 50, 21, 75, 3, 2, 1, 1, "normal"),
        # AlexNet / CaffeNet conv1 at the reference's batch size: large images, few channels, stride 4.
        _conv("alexnet_conv1_b256", "train", 256, 3, 227, 96, 11, 4, 0, 1, "normal"),
        # CaffeNet conv2: grouped, with the ReLU and pooling bridges around it folded in as a network does it.
        _conv("caffenet_conv2_fused_b256", "fused", 256, 96, 27, 256, 5, 1, 2, 2, "relu"),
        # A caller that keeps its cubes in host memory, as the reference's ParallelizedBridge does: one partition of 32 images.
        {"name": "alexnet_conv1_host_b32", "kind": "conv_host", "B": 32, "D": 3, "n": 227, "o": 96, "k": 11, "s": 4, "p": 0, "g": 1},
        # The largest inner product of CaffeNet (37.7 M weights), forward and backward.
        {"name": "fc6_b256", "kind": "fc", "mode": "train", "B": 256, "D": 256, "n": 6, "o": 4096},
        # The classifier of a network fine-tuned to ten classes, forward and backward on a batch that is no multiple of 32.
        {"name": "fc_classifier_b50", "kind": "fc", "mode": "train", "B": 50, "D": 4096, "n": 1, "o": 10},
        # The bridges between CaffeNet's first two convolutions, run one by one (a program that does not fold them).
        {"name": "relu_pool_lrn_b128", "kind": "layers", "B": 128, "D": 96, "n": 55, "k": 3, "s": 2},
        # A training iteration of a small network: some forty short passes.
        {"name": "lenet_iteration_b64", "kind": "small_net", "B": 64, "c": 1, "n": 28, "f1": 20, "f2": 50, "h": 500, "classes": 10},
        # The CaffeNet iteration on one eighth of a 256-image batch (the share of one GPU of eight), and on the whole batch.
        {"name": "caffenet_iteration_b32", "kind": "caffenet", "B": 32},
        {"name": "caffenet_iteration_b256", "kind": "caffenet", "B": 256},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _channels(rng, lo, hi):
    """Half of the layers one meets have channel counts that are multiples of eight."""
    v = _log_int(rng, lo, hi)
    return v // 8 * 8 if v >= 8 and rng.random() < 0.5 else v


def _draw_conv(rng, batch_hi, flops_hi, elements_hi):
    while True:
        k, s = rng.choice([(1, 1), (3, 1), (3, 1), (3, 2), (5, 1), (5, 2), (7, 2), (11, 4)])
        p = rng.choice([0, k // 2])
        g = 2 if rng.random() < 0.2 else 1
        D, o, n = _channels(rng, 1, 384) * g, _channels(rng, 8, 384) * g, _log_int(rng, max(6, k), 227)
        if k >= 7:  # such windows are met in first layers, on images
            D, o, g = rng.choice([1, 3, 4]), o // g, 1
        c = {"B": _log_int(rng, 1, batch_hi), "D": D, "n": n, "o": o, "k": k, "s": s, "p": p, "g": g}
        if D <= 384 and o <= 384 and _conv_flops(c) <= flops_hi and max(_conv_elements(c)) <= elements_hi:
            return c


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(["conv", "conv", "conv", "conv_host", "fc", "fc", "layers", "small_net", "caffenet"])
    if kind == "conv":
        mode = rng.choice(["train", "forward", "fused"])
        while True:
            c = _draw_conv(rng, 256, 2e11, 8e7)
            if mode != "fused" or (6 <= _out(c) <= 112 and c["k"] > 1 and c["o"] // c["g"] >= 64):  # a pooled layer is a wide one
                return dict(c, kind="conv", mode=mode, x=rng.choice(["normal", "relu", "uniform"]))
    if kind == "conv_host":
        return dict(_draw_conv(rng, 64, 2e10, 1e7), kind="conv_host")
    if kind == "fc":
        n = rng.choice([1, 1, 4, 6, 7])
        return {"kind": "fc", "mode": rng.choice(["train", "forward"]), "B": _log_int(rng, 1, 256),
                "D": _channels(rng, 64, 9216 // (n * n)), "n": n, "o": _channels(rng, 10, 4096)}
    if kind == "layers":
        k, s = rng.choice([(3, 2), (3, 2), (2, 2), (3, 1)])
        return {"kind": "layers", "B": _log_int(rng, 1, 256), "D": _channels(rng, 16, 256), "n": _log_int(rng, 8, 57), "k": k, "s": s}
    if kind == "small_net":
        return {"kind": "small_net", "B": _log_int(rng, 8, 256), "c": rng.choice([1, 3]), "n": rng.randint(24, 48),
                "f1": rng.randint(6, 32), "f2": rng.randint(16, 64), "h": _channels(rng, 64, 1024), "classes": rng.randint(2, 100)}
    return {"kind": "caffenet", "B": _log_int(rng, 16, 256)}


# ------------------------------------------------------------------------------------------------ sizes and work

def _out(c):
    return (c["n"] + 2 * c["p"] - c["k"]) // c["s"] + 1


def _conv_elements(c):
    """Elements of X, Y, W."""
    m = _out(c)
    return c["B"] * c["D"] * c["n"] ** 2, c["B"] * c["o"] * m * m, c["o"] * (c["D"] // c["g"]) * c["k"] ** 2


def _conv_flops(c):
    """Multiply-adds x 2 of one contraction of the layer."""
    return 2.0 * _conv_elements(c)[2] * _out(c) ** 2 * c["B"]


def _pooled(m, k, s):
    return (m - k) // s + 1


_CAFFENET = [dict(D=3, n=227, o=96, k=11, s=4, p=0, g=1), dict(D=96, n=27, o=256, k=5, s=1, p=2, g=2),
             dict(D=256, n=13, o=384, k=3, s=1, p=1, g=1), dict(D=384, n=13, o=384, k=3, s=1, p=1, g=2),
             dict(D=384, n=13, o=256, k=3, s=1, p=1, g=2)]
_CAFFENET_FC = [(9216, 4096), (4096, 4096), (4096, 1000)]


def _small_net_layers(c):
    """Convolution geometries and inner-product sizes of a small_net case."""
    n2 = _pooled(c["n"] - 4, 2, 2)
    n3 = _pooled(n2 - 4, 2, 2)
    return ([dict(D=c["c"], n=c["n"], o=c["f1"], k=5, s=1, p=0, g=1), dict(D=c["f1"], n=n2, o=c["f2"], k=5, s=1, p=0, g=1)],
            [(c["f2"] * n3 * n3, c["h"]), (c["h"], c["classes"])])


def work(c):
    """What one pass cannot do without: inputs read once, outputs written once, each contraction counted once."""
    kind = c["kind"]
    if kind in ("conv", "conv_host"):
        nx, ny, nw = _conv_elements(c)
        F, o = _conv_flops(c), c["o"]
        if c.get("mode") == "forward":
            return {"bytes": 4.0 * (nx + nw + o + ny), "flops": F}
        if c.get("mode") == "fused":
            nP = c["B"] * o * _pooled(_out(c), 3, 2) ** 2
            return {"bytes": 4.0 * (2 * nx + 2 * nw + 2 * o + ny + 3 * nP), "flops": 3 * F}  # X, W, b, dP -> Y, P, index, dX, dW, db
        return {"bytes": 4.0 * (2 * nx + 2 * ny + 2 * nw + 2 * o), "flops": 3 * F}           # X, W, b, dY -> Y, dX, dW, db
    if kind == "fc":
        K, O, B = c["D"] * c["n"] ** 2, c["o"], c["B"]
        if c["mode"] == "forward":
            return {"bytes": 4.0 * (B * K + K * O + O + B * O), "flops": 2.0 * B * K * O}
        return {"bytes": 4.0 * (2 * B * K + 2 * K * O + 2 * O + 2 * B * O), "flops": 6.0 * B * K * O}
    if kind == "layers":
        na = c["B"] * c["D"] * c["n"] ** 2
        nP = c["B"] * c["D"] * _pooled(c["n"], c["k"], c["s"]) ** 2
        # X, dN -> A, P, index, N, dP, dA, dX
        return {"bytes": 4.0 * (4 * na + 5 * nP), "flops": 0.0}
    convs, fcs = (_CAFFENET, _CAFFENET_FC) if kind == "caffenet" else _small_net_layers(c)
    flops, params = 0.0, 0
    for i, g in enumerate(convs):
        flops += (3 if i else 2) * _conv_flops(dict(g, B=c["B"]))
        params += _conv_elements(dict(g, B=1))[2] + g["o"]
    for K, O in fcs:
        flops += 6.0 * c["B"] * K * O
        params += K * O + O
    # images and labels in, probabilities out; parameters and momentum read and written, gradients written
    images = c["B"] * convs[0]["D"] * convs[0]["n"] ** 2
    return {"bytes": 4.0 * (images + c["B"] + c["B"] * fcs[-1][1] + 5 * params), "flops": flops}


def tolerance(c):
    """Contractions run on split fp32 operands with fp32 accumulation over sums of up to some ten thousand terms: 1e-4, the
    figure the framework's parity tests state.  Where max pooling or a ReLU sits behind a contraction, an fp32 difference
    in the last places turns a near-tie of a window, or a sign near zero, now and then: that gradient then takes another
    way, and a gradient tensor that is a sum of n terms of random sign moves by sqrt(turned / n) - 1e-3 to 1e-2 where a
    few in 10^5 turn (the direct fp32 kernels and the tensor-core kernels differ by as much)."""
    if c["kind"] == "layers":
        return {"rel": 1e-5, "max": 1e-4}
    if c["kind"] in ("caffenet", "small_net"):
        return {"rel": 0.025, "max": 0.99}
    if c.get("mode") == "fused":
        return {"rel": 0.01, "max": 0.9, "differ": 1e-3}
    return {"rel": 1e-4, "max": 1e-3}


# ------------------------------------------------------------------------------------------------ states

_ctx = None


def _context():
    """The program's one context, on torch's current stream."""
    global _ctx
    if _ctx is None:
        _ctx = Context(0, stream=torch.cuda.current_stream().cuda_stream)
    return _ctx


class _Owner:
    """Closes what a state holds outside torch's allocator (plans, networks) once nothing refers to it any more."""

    def __init__(self, close):
        self._close = close

    def __del__(self):
        self._close()


class _Memory:
    """Device memory of the framework's own as a torch tensor; the tensor keeps `owner` alive."""

    def __init__(self, ptr, count, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _view(ptr, count, owner):
    return torch.as_tensor(_Memory(ptr, count, owner), device="cuda")


def _values(gen, shape, dist):
    if dist in ("uniform", "xavier"):
        t = torch.rand(shape, generator=gen, device="cuda")
        return t.sub_(0.5).mul_(2 * 0.01 * math.sqrt(3.0)) if dist == "xavier" else t  # standard deviation 0.01
    t = torch.randn(shape, generator=gen, device="cuda")
    return t.clamp_(min=0) if dist == "relu" else t


def _images(gen, B, D, n):
    """Mean-subtracted pixels: low frequencies with a standard deviation of some fifty grey levels, and some noise."""
    low = torch.randn((B, D, 14, 14), generator=gen, device="cuda")
    x = torch.nn.functional.interpolate(low, size=(n, n), mode="bilinear", align_corners=False)
    return 75 * x + 5 * torch.randn((B, D, n, n), generator=gen, device="cuda")


def _empty(*shape, dtype=torch.float32):
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _cube(ctx, t):
    """A cube over a torch tensor of shape (B, D, R, C)."""
    B, D, R, Cc = t.shape
    return LogicalCube(ctx, R, Cc, D, B, np.int32 if t.dtype == torch.int32 else np.float32, ptr=t.data_ptr())


def _with_parameters(br, W, b, dW, db):
    """The bridge's model, bias and gradient cubes over the caller's tensors."""
    for name, t in (("p_model_cube", W), ("p_bias_cube", b), ("p_model_gradient_cube", dW), ("p_bias_gradient_cube", db)):
        getattr(br, name).free()
        setattr(br, name, _cube(br.ctx, t))


def _prepare_conv(c, ctx, gen):
    B, D, n, o, k, g, m = c["B"], c["D"], c["n"], c["o"], c["k"], c["g"], _out(c)
    X, dX = _values(gen, (B, D, n, n), c["x"]), _empty(B, D, n, n)
    W, b = _values(gen, (o, D // g, k, k), "xavier"), 0.1 * _values(gen, (1, o, 1, 1), "normal")
    dW, db = torch.zeros_like(W), torch.zeros_like(b)
    Y, dY = _empty(B, o, m, m), _values(gen, (B, o, m, m), "normal") if c["mode"] == "train" else _empty(B, o, m, m)
    xin, out = Layer(_cube(ctx, X), _cube(ctx, dX)), Layer(_cube(ctx, Y), _cube(ctx, dY))
    br = ConvolutionBridge(xin, out, k, c["s"], c["p"], g, True, ctx=ctx)
    _with_parameters(br, W, b, dW, db)
    s = {"bridge": br, "tensors": (X, W, b, dY)}
    if c["mode"] == "train":
        s["out"] = [Y, dX, dW, db]
    elif c["mode"] == "forward":
        br.fuse_relu = True
        s["out"] = [Y]
    else:
        q = _pooled(m, 3, 2)
        P, dP, index = _empty(B, o, q, q), _values(gen, (B, o, q, q), "uniform") - 0.5, _empty(B, o, q, q, dtype=torch.int32)
        pool = MaxPoolingBridge(out, Layer(_cube(ctx, P), _cube(ctx, dP)), 3, 2, ctx)
        pool.max_index.free()
        pool.max_index = _cube(ctx, index)
        br.fuse_relu = br.fuse_relu_backward = True
        br.fuse_pool_relu_backward(pool.p_output_layer.p_gradient_cube, pool.max_index, 3, 2, pool.p_output_layer.p_data_cube)
        s.update(pool=pool, dP=dP, out=[Y, P, index, dX, dW, db])
    s["owner"] = _Owner(br.close)
    return s


def _prepare_conv_host(c, ctx, gen):
    B, D, n, o, k, g, m = c["B"], c["D"], c["n"], c["o"], c["k"], c["g"], _out(c)
    desc, plan = capi.ConvDesc(B, D, n, o, k, c["s"], c["p"], g, 1, capi.ALGO_AUTO), C.c_void_p()
    capi.check(ctx.lib.cct_conv_plan_create(ctx.h, C.byref(desc), C.byref(plan)), "cct_conv_plan_create", ctx.h)
    host = lambda t: t.cpu().pin_memory()  # noqa: E731
    X, dY = host(_values(gen, (B, D, n, n), "normal")), host(_values(gen, (B, o, m, m), "normal"))
    W, b = host(_values(gen, (o, D // g, k, k), "xavier")), host(0.1 * _values(gen, (o,), "normal"))
    out = [torch.zeros(t.shape).pin_memory() for t in (dY, X, W, b)]  # Y, dX, dW, db
    lib = ctx.lib
    return {"plan": plan, "inputs": (X, W, b, dY), "out": out, "owner": _Owner(lambda: lib.cct_conv_plan_destroy(plan))}


def _prepare_fc(c, ctx, gen):
    B, D, n, o = c["B"], c["D"], c["n"], c["o"]
    X, dX = _values(gen, (B, D, n, n), "relu"), _empty(B, D, n, n)
    W, b = _values(gen, (o, D, n, n), "xavier"), 0.1 * _values(gen, (1, o, 1, 1), "normal")
    dW, db = torch.zeros_like(W), torch.zeros_like(b)
    Y, dY = _empty(B, o, 1, 1), _values(gen, (B, o, 1, 1), "normal")
    br = FullyConnectedBridge(Layer(_cube(ctx, X), _cube(ctx, dX)), Layer(_cube(ctx, Y), _cube(ctx, dY)), True, ctx=ctx)
    holder = br._conv or br  # a layer outside the fully connected plan keeps its parameters in the convolution it runs as
    _with_parameters(holder, W, b, dW, db)
    return {"bridge": br, "tensors": (X, W, b, dY), "out": [Y, dX, dW, db] if c["mode"] == "train" else [Y], "owner": _Owner(br.close)}


def _prepare_layers(c, ctx, gen):
    B, D, n, k, s = c["B"], c["D"], c["n"], c["k"], c["s"]
    q = _pooled(n, k, s)
    X, dX, A, dA = _values(gen, (B, D, n, n), "normal"), _empty(B, D, n, n), _empty(B, D, n, n), _empty(B, D, n, n)
    X.mul_(20)  # activations of a first layer, large enough for the normalisation to matter
    P, dP, N, dN = _empty(B, D, q, q), _empty(B, D, q, q), _empty(B, D, q, q), _values(gen, (B, D, q, q), "normal")
    index = _empty(B, D, q, q, dtype=torch.int32)
    x, a, p, y = (Layer(_cube(ctx, u), _cube(ctx, v)) for u, v in ((X, dX), (A, dA), (P, dP), (N, dN)))
    relu, pool, lrn = ReLUBridge(x, a, ctx), MaxPoolingBridge(a, p, k, s, ctx), LRNBridge(p, y, 5, 1e-4, 0.75, ctx)
    pool.max_index.free()
    pool.max_index = _cube(ctx, index)
    return {"chain": (relu, pool, lrn), "tensors": (X, dN), "out": [A, P, index, N, dP, dA, dX], "owner": _Owner(lrn.close)}


_SMALL_NET = """
layer { name: "data" type: "Data" top: "data" top: "label" }
layer { name: "conv1" type: "Convolution" bottom: "data" top: "conv1" param { lr_mult: 1 } param { lr_mult: 2 }
  convolution_param { num_output: %(f1)d kernel_size: 5 weight_filler { type: "xavier" } bias_filler { type: "constant" } } }
layer { name: "pool1" type: "Pooling" bottom: "conv1" top: "pool1" pooling_param { pool: MAX kernel_size: 2 stride: 2 } }
layer { name: "conv2" type: "Convolution" bottom: "pool1" top: "conv2" param { lr_mult: 1 } param { lr_mult: 2 }
  convolution_param { num_output: %(f2)d kernel_size: 5 weight_filler { type: "xavier" } bias_filler { type: "constant" } } }
layer { name: "pool2" type: "Pooling" bottom: "conv2" top: "pool2" pooling_param { pool: MAX kernel_size: 2 stride: 2 } }
layer { name: "ip1" type: "InnerProduct" bottom: "pool2" top: "ip1" param { lr_mult: 1 } param { lr_mult: 2 }
  inner_product_param { num_output: %(h)d weight_filler { type: "xavier" } bias_filler { type: "constant" } } }
layer { name: "relu1" type: "ReLU" bottom: "ip1" top: "ip1" }
layer { name: "ip2" type: "InnerProduct" bottom: "ip1" top: "ip2" param { lr_mult: 1 } param { lr_mult: 2 }
  inner_product_param { num_output: %(classes)d weight_filler { type: "xavier" } bias_filler { type: "constant" } } }
layer { name: "loss" type: "SoftmaxWithLoss" bottom: "ip2" bottom: "label" top: "loss" }
"""
_SMALL_SOLVER = 'base_lr: 0.01 lr_policy: "inv" gamma: 0.0001 power: 0.75 momentum: 0.9 weight_decay: 0.0005'


def _prepare_net(c, ctx, gen, seed):
    if c["kind"] == "caffenet":
        with open(os.path.join(NETS, "caffenet_train.prototxt")) as f:
            text = f.read()
        with open(os.path.join(NETS, "caffenet_solver.prototxt")) as f:
            solver = f.read() + "\nbase_lr: 0.0005\n"  # a network being fine-tuned: small steps, batches of ten of the classes
        shape, classes = (3, 227), 10
    else:
        text, solver = _SMALL_NET % c, _SMALL_SOLVER
        shape, classes = (c["c"], c["n"]), c["classes"]
    net = load_net(ctx, text, solver + "\nrandom_seed: %d\n" % (seed % 1000003 + 1), c["B"], input_shape=shape)
    owner = _Owner(net.close)
    x, labels = net.input.p_data_cube, net.labels
    images = _images(gen, *x.shape[:3]) if c["kind"] == "caffenet" else _values(gen, x.shape, "uniform")
    _view(x.ptr, x.n_elements, owner).copy_(images.reshape(-1))
    _view(labels.ptr, labels.n_elements, owner).copy_(torch.randint(0, classes, (c["B"],), generator=gen, device="cuda").float())
    prob, loss = net.loss_bridge.p_output_layer.p_data_cube, net.loss_bridge.loss_cube
    out = [_view(prob.ptr, prob.n_elements, owner), _view(loss.ptr, 1, owner)]
    for _, pb in net.param_bridges():  # updated parameters, gradients, momentum: weights | bias of each layer
        out += [_view(p, pb.count, owner) for p in (pb.params, pb.grads, pb.hist)]
    return {"net": net, "out": out, "owner": owner}


def prepare(c, seed):
    ctx = _context()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    if c["kind"] in ("caffenet", "small_net"):
        s = _prepare_net(c, ctx, gen, int(seed))
    else:
        s = {"conv": _prepare_conv, "conv_host": _prepare_conv_host, "fc": _prepare_fc, "layers": _prepare_layers}[c["kind"]](c, ctx, gen)
    s["kind"], s["mode"], s["ctx"] = c["kind"], c.get("mode"), ctx
    return s


def run(s):
    """One pass; the outputs are the state's own buffers."""
    kind = s["kind"]
    if kind in ("conv", "fc"):
        br = s["bridge"]
        br.forward()
        if s["mode"] == "fused":
            s["pool"].forward()
        if s["mode"] != "forward":
            br.backward()
    elif kind == "conv_host":
        lib, h, plan = s["ctx"].lib, s["ctx"].h, s["plan"]
        X, W, b, dY = (t.data_ptr() for t in s["inputs"])
        Y, dX, dW, db = (t.data_ptr() for t in s["out"])
        capi.check(lib.cct_conv_forward_host(plan, X, W, b, Y, 0), "cct_conv_forward_host", h)
        capi.check(lib.cct_conv_backward_host(plan, None, None, dY, dX, dW, db), "cct_conv_backward_host", h)
    elif kind == "layers":
        for br in s["chain"]:
            br.forward()
        for br in reversed(s["chain"]):
            br.backward()
    else:
        s["net"].step()
    return s["out"]
