"""The inference work whose speed matters: whole networks and single layers, through the package's public entry points.

Whole networks are the three xnor networks Darknet ships, loaded from a .cfg and a .weights file and kept; a pass takes one
device-resident input batch to the activated heads (forward_network_gpu) or on to the detection rows on the host
(network_detections + rows_host, what a program that shows boxes does with every frame).  Single layers are the boundary a
Darknet build calls: one [convolutional] xnor=1 layer with its packed weights, fp32 in, fp32 out.

Weights and images are synthetic.  Images are 8-bit frames (multiples of 2^-8 in [0, 1)) and the weights of a network's first
convolution sit on a 2^-10 grid, so that layer's sums are exact in fp32 in any order; the binarisation behind it then has one
right answer and everything up to the heads can be compared closely.
"""
from __future__ import annotations

import math
import os
import struct
import tempfile

import numpy as np
import torch

from darknet_b200 import capi, cfgs
from darknet_b200 import layer as L
from darknet_b200 import network as N

DEVICE = "cuda:0"
CLASSES = 80                        # of both detectors' cfgs
ROWS = 1024                         # detection rows kept of one image
IMAGES = {                          # most pixels of one call: the batches the networks are run with, at their own resolution
    "yolov3-tiny_xnor": 64 * 416 * 416,
    "tiny-yolo_xnor": 256 * 416 * 416,
    "darknet53_448_xnor": 64 * 448 * 448,
}
LAYER_BYTES = 64 * (128 + 256) * 104 * 104 * 4     # most fp32 bytes in and out of a single-layer call
LAYER_BINOPS = 2 * 256 * 1152 * 64 * 104 * 104     # most binary operations of a single-layer call


def _net(name, network, width, height, batch, out):
    return {"name": name, "kind": "network", "network": network, "width": width, "height": height, "batch": batch, "out": out}


def _layer(name, c, h, w, n, size, stride, batch, activation):
    return {"name": name, "kind": "layer", "c": c, "h": h, "w": w, "n": n, "size": size, "stride": stride, "batch": batch,
            "activation": activation}


def listed():
    return [
        # one camera frame to boxes: the latency of the headline network
        _net("yolov3-tiny frame to boxes", "yolov3-tiny_xnor", 416, 416, 1, "rows"),
        # eight cameras served by one process
        _net("yolov3-tiny b8 to boxes", "yolov3-tiny_xnor", 416, 416, 8, "rows"),
        # a wide picture cut for a 16:9 source, an odd number of them, heads read on the device
        _net("yolov3-tiny 608x352 b3", "yolov3-tiny_xnor", 608, 352, 3, "heads"),
        # offline video: the batch that fills the GPU
        _net("yolov3-tiny b64", "yolov3-tiny_xnor", 416, 416, 64, "heads"),
        # a global batch of 256 on one GPU
        _net("tiny-yolo b256", "tiny-yolo_xnor", 416, 416, 256, "heads"),
        # classifying one picture: 52 dependent layers
        _net("darknet53 b1", "darknet53_448_xnor", 448, 448, 1, "heads"),
        # one GPU's share of a global batch of 512 on eight
        _net("darknet53 b64", "darknet53_448_xnor", 448, 448, 64, "heads"),
        # the single layer of the reference comparison
        _layer("layer 256-512 3x3 26x26 b1", 256, 26, 26, 512, 3, 1, 1, "leaky"),
        # the smallest call: a bottleneck on the coarsest map
        _layer("layer 1024-256 1x1 13x13 b1", 1024, 13, 13, 256, 1, 1, 1, "leaky"),
        # channels that fill no whole words: K = 675 and the plain [c][tap] bit order
        _layer("layer 75-64 3x3 52x52 b8", 75, 52, 52, 64, 3, 1, 8, "leaky"),
        # the largest fp32 tensors of the shape sweep a layer call is used with
        _layer("layer 128-256 3x3 104x104 b64", 128, 104, 104, 256, 3, 1, 64, "linear"),
    ]


def _log(rng, lo, hi):
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    if rng.random() < 0.5:
        network = rng.choice(sorted(IMAGES))
        step, lo, hi = 32, 7, 19                                   # 224 ... 608, each side on its own
        width, height = step * rng.randint(lo, hi), step * rng.randint(lo, hi)
        batch = _log(rng, 1, IMAGES[network] // (width * height))
        out = "rows" if network == "yolov3-tiny_xnor" and batch <= 16 and rng.random() < 0.5 else "heads"
        case = _net("", network, width, height, batch, out)
    else:
        while True:
            # three in four layers have whole words of channels, and whole words of filters, as networks do
            c = 32 * _log(rng, 1, 32) if rng.random() < 0.75 else _log(rng, 8, 1024)
            n = 32 * _log(rng, 1, 32) if rng.random() < 0.75 else _log(rng, 8, 1024)
            case = _layer("", c, _log(rng, 7, 208), _log(rng, 7, 208), n, rng.choice((1, 3)), 2 if rng.random() < 0.2 else 1,
                          _log(rng, 1, 64), rng.choice(("leaky", "linear")))
            oh, ow = _out_map(case)
            floats = case["batch"] * (c * case["h"] * case["w"] + n * oh * ow)
            if 4 * floats <= LAYER_BYTES and _layer_binops(case) <= LAYER_BINOPS:
                break
    del case["name"]
    return case


def _out_map(case):
    pad = case["size"] // 2
    return tuple((case[d] + 2 * pad - case["size"]) // case["stride"] + 1 for d in ("h", "w"))


def _layer_binops(case):
    oh, ow = _out_map(case)
    return 2 * case["batch"] * case["n"] * oh * ow * case["c"] * case["size"] ** 2


# ---- what a program has in hand before the call -------------------------------------------------------------------------


def _normal(gen, *shape, sigma=1.0):
    return torch.randn(*shape, generator=gen, device=DEVICE) * sigma


def _write_weights(net, path, gen):
    """A .weights file of the network's layout (header, then per convolution biases, batch-norm, weights; all fp32)."""
    def put(fh, t):
        fh.write(np.ascontiguousarray(t.cpu().numpy(), "<f4").tobytes())

    convs = [l for l in net.layers if l.type == "convolutional"]
    with open(path, "wb") as fh:
        fh.write(struct.pack("<iiiQ", 0, 2, 5, 0))
        for l in convs:
            fan_in = l.c * l.size * l.size
            biases = _normal(gen, l.n, sigma=0.01)
            weights = _normal(gen, l.n, fan_in, sigma=0.05 if l.xnor else fan_in ** -0.5)
            norm = [0.5 + torch.rand(l.n, generator=gen, device=DEVICE), _normal(gen, l.n, sigma=0.1),
                    0.25 + torch.rand(l.n, generator=gen, device=DEVICE)]
            if l is convs[0]:
                # exact sums in any order: a 2^-10 grid, and a batch-norm whose factor rounds to one
                biases, weights = (biases * 1024).round() / 1024, ((weights * 1024).round() / 1024).clamp(-0.25, 0.25)
                norm = [torch.ones(l.n), torch.zeros(l.n), torch.full((l.n,), 1.0 - 1e-5)]
            follows = net.layers[l.index + 1].type if l.index + 1 < len(net.layers) else ""
            if follows == "yolo":
                # a trained head: few cells hold an object, and an object is of few classes
                weights -= weights.mean(1, keepdim=True)
                entries = biases.view(-1, 5 + CLASSES)
                entries[:, 4] -= 5.0
                entries[:, 5:] -= 3.0
            put(fh, biases)
            if l.batch_normalize:
                for t in norm:
                    put(fh, t)
            put(fh, weights)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    if case["kind"] == "layer":
        act = capi.LEAKY if case["activation"] == "leaky" else capi.LINEAR
        layer = L.make_convolutional_layer(case["batch"], case["h"], case["w"], case["c"], case["n"], case["size"], case["stride"],
                                           case["size"] // 2, act, device=DEVICE)
        layer.load_weights(_normal(gen, case["n"], case["c"] * case["size"] ** 2, sigma=0.05), _normal(gen, case["n"], sigma=0.01))
        L.binary_align_weights(layer)
        return {"layer": layer, "x": _normal(gen, case["batch"], case["c"], case["h"], case["w"])}
    with tempfile.TemporaryDirectory() as folder:
        cfg, weights = os.path.join(folder, "net.cfg"), os.path.join(folder, "net.weights")
        with open(cfg, "w") as fh:
            fh.write(cfgs.CFGS[case["network"]](case["width"], case["height"]))
        _write_weights(N.parse_network_cfg(cfg, case["batch"], DEVICE), weights, gen)
        net = N.load_network_custom(cfg, weights, case["batch"], DEVICE)
    # pictures: shapes some tens of pixels wide, with fine detail on them
    shape = (case["height"], case["width"])
    coarse = torch.rand(case["batch"], 3, shape[0] // 32, shape[1] // 32, generator=gen, device=DEVICE)
    x = torch.nn.functional.interpolate(coarse, shape, mode="bilinear")
    x = ((0.8 * x + 0.2 * torch.rand(x.shape, generator=gen, device=DEVICE)) * 256).floor().clamp(0, 255) / 256
    state = {"net": net, "x": x}
    if case["out"] == "rows":
        state["dets"] = N.DetectionBuffers(case["batch"], CLASSES, device=DEVICE)
    return state


def run(state):
    if "layer" in state:
        return L.forward_convolutional_layer_gpu(state["layer"], state["x"])
    if "dets" in state:
        # rows of a fixed shape, as a message to the next process has; nothing is behind the last one
        out = np.zeros((state["net"].batch, ROWS, 7), np.float32)
        for shown, rows in zip(out, N.network_detections(state["net"], state["x"], dets=state["dets"]).rows_host()):
            shown[:len(rows)] = rows[:ROWS]
        return out
    return N.forward_network_gpu(state["net"], state["x"])


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------


def work(case):
    """Bytes: the input, the weights as they are kept (one bit each in an xnor layer, with a scale and a bias per filter) and
    the outputs.  Operations: a multiply and an add per weight and output position, binary or not."""
    if case["kind"] == "layer":
        oh, ow = _out_map(case)
        k = case["c"] * case["size"] ** 2
        floats = case["batch"] * (case["c"] * case["h"] * case["w"] + case["n"] * oh * ow)
        return {"bytes": 4 * floats + case["n"] * (k / 8 + 8), "flops": _layer_binops(case)}
    with tempfile.TemporaryDirectory() as folder:
        cfg = os.path.join(folder, "net.cfg")
        with open(cfg, "w") as fh:
            fh.write(cfgs.CFGS[case["network"]](case["width"], case["height"]))
        net = N.parse_network_cfg(cfg, case["batch"], DEVICE)
    nbytes, flops = 4.0 * case["batch"] * 3 * case["height"] * case["width"], 0.0
    for l in net.layers:
        if l.type == "convolutional":
            k = l.c * l.size * l.size
            nbytes += l.n * (k / 8 + 8 if l.xnor else 4 * k + 4)
            flops += 2.0 * case["batch"] * l.n * k * l.out_h * l.out_w
        elif l.type in ("yolo", "region", "softmax") and case["out"] == "heads":
            nbytes += 4.0 * case["batch"] * l.outputs
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "layer":
        return "exact"               # integer counts, then one multiply and one add in a fixed order
    # the float convolutions in front of the heads: fp32 sums over up to 2304 products, in any order
    return {"rel": 2e-5, "max": 2e-4}
