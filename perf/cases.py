"""Performance cases: what programs have this library compute, through its public entry points.

Five kinds of call, each with the sizes listed here and a range that ``draw`` takes more cases from:

  graph   ``compile(conv2d -> bias_add -> relu).run(x, w, b)``, the fused node of the graph API
  conv2d  eager ``conv2d`` as a drop-in for ``flag_dnn.ops.conv2d``, dense, grouped and depthwise
  conv1d  eager ``conv1d`` over long one-dimensional signals
  mm      eager ``mm``, a product of an activation matrix with a weight matrix
  stack   ``ResNet50ConvStack.forward``: the 53 convolutions and the max pooling of ResNet-50 with their folded
          scales and biases and fused shortcuts, then ``adaptive_avg_pool2d``

The library computes forward passes only; every path it has is a forward path.
"""
import math

import torch

import flagdnn_b200 as fd
from flagdnn_b200.convstack import ResNet50ConvStack, resnet50_conv_layers, stack_totals

_DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
_SIZES = {"f16": 2, "bf16": 2, "f32": 4}


def _conv(name, kind, dtype, layout, n, c, h, w, k, r, s, stride=1, pad=0, dil=1, groups=1, bias=True):
    return {"name": name, "kind": kind, "dtype": dtype, "layout": layout, "n": n, "c": c, "h": h, "w": w, "k": k, "r": r,
            "s": s, "stride": stride, "pad": pad, "dil": dil, "groups": groups, "bias": bias}


def listed():
    return [
        # one image through a small layer of an fp16 network: launches and host time are what it costs
        _conv("graph_one_image_f16", "graph", "f16", "nchw", 1, 64, 14, 14, 64, 3, 3, pad=1),
        # a small fp32 batch in torch's default layout, the benchmark's fp32 configuration
        _conv("graph_nchw_f32", "graph", "f32", "nchw", 4, 64, 56, 56, 64, 3, 3, pad=1),
        # the headline layer: the 3x3 convolution of a ResNet's third stage at a training-sized batch
        _conv("graph_3x3_bf16", "graph", "bf16", "nhwc", 256, 256, 14, 14, 256, 3, 3, pad=1),
        # the 7x7 stride-2 stem on RGB images
        _conv("graph_stem_bf16", "graph", "bf16", "nhwc", 256, 3, 224, 224, 64, 7, 7, stride=2, pad=3),
        # a whole ResNet-50's convolutions at the batch one of eight GPUs holds of 1024 images
        {"name": "resnet50_bf16", "kind": "stack", "dtype": "bf16", "n": 128, "image": 224},
        # an eager call on torch's default layout, as a model that was not converted to channels-last makes it
        _conv("conv2d_nchw_f16", "conv2d", "f16", "nchw", 32, 128, 28, 28, 128, 3, 3, pad=1),
        # channel counts and image sides that fit no tile
        _conv("conv2d_ragged_bf16", "conv2d", "bf16", "nhwc", 24, 100, 45, 37, 150, 3, 3, pad=1),
        # a temporal convolution over feature frames of odd length
        _conv("conv1d_ragged_bf16", "conv1d", "bf16", "nchw", 16, 80, 1, 1501, 256, 1, 5, pad=2),
        # depthwise layers in both layouts
        _conv("depthwise_nhwc_bf16", "conv2d", "bf16", "nhwc", 256, 64, 56, 56, 64, 3, 3, pad=1, groups=64),
        _conv("depthwise_nchw_bf16", "conv2d", "bf16", "nchw", 256, 64, 56, 56, 64, 3, 3, pad=1, groups=64),
        # a grouped layer with few groups
        _conv("grouped_nhwc_bf16", "conv2d", "bf16", "nhwc", 256, 64, 56, 56, 128, 3, 3, pad=1, groups=2),
        # a projection of many tokens
        {"name": "mm_bf16", "kind": "mm", "dtype": "bf16", "m": 8192, "kk": 4096, "nn": 4096},
    ]


def _log(rng, low, high):
    """An integer of [low, high], uniform in its logarithm."""
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def _channels(rng, low, high):
    """A channel count: mostly multiples of 8, as networks have them, one in four as it falls."""
    c = _log(rng, low, high)
    return c if rng.random() < 0.25 else max(8, c // 8 * 8)


def draw(rng):
    while True:
        case = _draw(rng)
        # between one small layer and the largest listed case in operations, bytes and memory
        flops, nbytes = work(case)["flops"], work(case)["bytes"]
        if 1e6 <= flops <= 1.0e12 and nbytes <= 1.0e9:
            return case


def _draw(rng):
    kind = rng.choice(["graph", "graph", "stem", "conv2d", "conv2d", "conv1d", "depthwise", "grouped", "mm", "stack"])
    dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
    layout = rng.choice(["nhwc", "nchw"])
    if kind == "stack":
        return {"kind": "stack", "dtype": rng.choice(["bf16", "f16"]), "n": _log(rng, 1, 128), "image": rng.choice([160, 192, 224])}
    if kind == "mm":
        return {"kind": "mm", "dtype": rng.choice(["bf16", "f16"]), "m": _log(rng, 64, 8192), "kk": _channels(rng, 64, 4096),
                "nn": _channels(rng, 64, 4096)}
    if kind == "conv1d":
        s = rng.choice([1, 3, 5, 7])
        case = _conv("", "conv1d", rng.choice(["bf16", "f16"]), "nchw", _log(rng, 1, 32), _channels(rng, 32, 512), 1,
                     _log(rng, 200, 4000), _channels(rng, 32, 512), 1, s, stride=rng.choice([1, 1, 2]), pad=s // 2)
    elif kind == "stem":
        h = 2 * rng.randint(48, 128)
        case = _conv("", "graph", rng.choice(["bf16", "f16"]), layout, _log(rng, 1, 256), 3, h, h, rng.choice([32, 64]), 7, 7,
                     stride=2, pad=3)
    elif kind == "depthwise":
        c, r, h = _channels(rng, 32, 1024), rng.choice([3, 3, 5]), _log(rng, 7, 112)
        case = _conv("", "conv2d", dtype, layout, _log(rng, 1, 256), c, h, h, c, r, r, stride=rng.choice([1, 1, 2]), pad=r // 2,
                     groups=c)
    elif kind == "grouped":
        g = rng.choice([2, 4, 8, 16, 32])
        cg, h = 8 * rng.randint(1, 8), _log(rng, 7, 56)
        case = _conv("", "conv2d", rng.choice(["bf16", "f16"]), layout, _log(rng, 1, 256), g * cg, h, h,
                     g * cg * rng.choice([1, 2]), 3, 3, stride=rng.choice([1, 1, 2]), pad=1, groups=g)
    else:
        r = rng.choice([1, 3, 3, 3, 5])
        dil = 2 if r == 3 and rng.random() < 0.15 else 1
        case = _conv("", kind, dtype, layout, _log(rng, 1, 256), _channels(rng, 16, 1024), _log(rng, 7, 112), _log(rng, 7, 112),
                     _channels(rng, 16, 1024), r, r, stride=rng.choice([1, 1, 1, 2]), pad=dil * (r // 2), dil=dil,
                     bias=kind == "graph" or rng.random() < 0.7)
    del case["name"]
    return case


def _out_hw(case):
    span_h, span_w = case["dil"] * (case["r"] - 1) + 1, case["dil"] * (case["s"] - 1) + 1
    if case["kind"] == "conv1d":
        return 1, (case["w"] + 2 * case["pad"] - span_w) // case["stride"] + 1
    return ((case["h"] + 2 * case["pad"] - span_h) // case["stride"] + 1,
            (case["w"] + 2 * case["pad"] - span_w) // case["stride"] + 1)


def work(case):
    es = _SIZES[case["dtype"]]
    if case["kind"] == "stack":
        layers = resnet50_conv_layers(case["image"])
        totals = stack_totals(layers, case["n"])
        last = layers[-1]
        # what must cross memory once: the images, the parameters, the last feature map and its means
        weights = sum(l.cout * l.cin * l.k * l.k + 2 * l.cout for l in layers)
        values = case["n"] * (3 * case["image"] ** 2 + last.cout * last.hw_out ** 2 + last.cout) + weights
        return {"bytes": float(es * values), "flops": totals["flops"]}
    if case["kind"] == "mm":
        m, k, n = case["m"], case["kk"], case["nn"]
        return {"bytes": float(es * (m * k + k * n + m * n)), "flops": 2.0 * m * k * n}
    oh, ow = _out_hw(case)
    n, c, k, taps = case["n"], case["c"], case["k"], case["r"] * case["s"]
    cg = c // case["groups"]
    values = n * c * case["h"] * case["w"] + k * cg * taps + (k if case["bias"] else 0) + n * k * oh * ow
    return {"bytes": float(es * values), "flops": 2.0 * n * oh * ow * k * cg * taps}


def tolerance(case):
    # Outputs are rounded once to the tensors' type after fp32 sums; fp32 tensors are multiplied as three TF32
    # products.  Stated: about four times the relative error measured against the same operation in fp64 (bf16
    # 1.66e-3, f16 2.1e-4, f32 4.0e-6; the whole stack 6.6e-3 in bf16 and 8.2e-4 in f16).
    if case["kind"] == "stack":
        return {"rel": {"bf16": 2.6e-2, "f16": 3.3e-3}[case["dtype"]]}
    return {"rel": {"bf16": 7.0e-3, "f16": 9.0e-4, "f32": 1.6e-5}[case["dtype"]]}


def _block(stride, padding, dilation):
    @fd.graph
    def conv_bias_relu(x, weight, bias):
        y = fd.conv2d(x, weight, stride=stride, padding=padding, dilation=dilation)
        return fd.relu(fd.bias_add(y, bias))

    return conv_bias_relu


def prepare(case, seed):
    dtype = _DTYPES[case["dtype"]]
    device = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=device).manual_seed(seed)

    def normal(shape, std=1.0):
        return (torch.randn(shape, generator=g, device=device) * std).to(dtype)

    state = {"case": case}
    if case["kind"] == "stack":
        state["model"] = ResNet50ConvStack(device, dtype, seed=seed, image=case["image"])
        x = normal((case["n"], 3, case["image"], case["image"]))
        state["x"] = x.contiguous(memory_format=torch.channels_last)
        return state
    if case["kind"] == "mm":
        state["x"] = normal((case["m"], case["kk"]))
        state["w"] = normal((case["kk"], case["nn"]), case["kk"] ** -0.5)
        return state
    cg = case["c"] // case["groups"]
    std = (cg * case["r"] * case["s"]) ** -0.5
    state["b"] = normal((case["k"],), 0.1) if case["bias"] else None
    if case["kind"] == "conv1d":
        state["x"] = normal((case["n"], case["c"], case["w"]))
        state["w"] = normal((case["k"], cg, case["s"]), std)
        return state
    fmt = torch.channels_last if case["layout"] == "nhwc" else torch.contiguous_format
    state["x"] = normal((case["n"], case["c"], case["h"], case["w"])).contiguous(memory_format=fmt)
    state["w"] = normal((case["k"], cg, case["r"], case["s"]), std).contiguous(memory_format=fmt)
    if case["kind"] == "graph":
        block = _block(case["stride"], case["pad"], case["dil"])
        state["compiled"] = fd.compile(block, inputs=[state["x"], state["w"], state["b"]])
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "graph":
        return state["compiled"].run(state["x"], state["w"], state["b"])
    if kind == "conv2d":
        return fd.conv2d(state["x"], state["w"], state["b"], stride=case["stride"], padding=case["pad"], dilation=case["dil"],
                         groups=case["groups"])
    if kind == "conv1d":
        return fd.conv1d(state["x"], state["w"], state["b"], stride=case["stride"], padding=case["pad"], dilation=case["dil"])
    if kind == "mm":
        return fd.mm(state["x"], state["w"])
    features = state["model"].forward(state["x"], fuse_residual=True)
    return features, fd.adaptive_avg_pool2d(features, 1)
