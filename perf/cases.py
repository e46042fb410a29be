"""The work that users of the data-graph path have it do, as cases to time.

Every case goes the way a host program goes: a graph is handed over as SPIR-V assembly with its constants, a session is
planned and bound (``prepare``: that is done once and kept), and a pass is one dispatch of that session over the inputs
it is bound to (``run``).  All arithmetic is integer, so outputs are compared byte for byte.

Kinds of case, and what each stands for in real use:
  conv       one CONV2D + per-channel RESCALE (benchmark configuration 0): a single layer that a host offloads by itself,
             enqueued without a captured graph; the smallest calls, where the launch counts
  matmul     batched MATMUL of two run-time inputs + RESCALE (benchmark configuration 1)
  resnet     the ResNet-50-shaped classifier (configuration 3): one image for latency, 64 for throughput; ``host`` is the
             serving form with the batch in pinned host memory and the logits read back (``run_host``)
  mobilenet  the MobileNetV2-shaped classifier (configuration 2): depthwise layers and narrow channel counts
  bert       the BERT-base-shaped encoder (configuration 4), padded sequences and ones of odd length
  segment    a per-pixel classifier over video frames: encoder, decoder with RESIZE, SLICE and CONCAT skips, a head with
             as many channels as there are classes, ARGMAX; frame sizes and class counts are seldom multiples of anything
  ops        the memory-bound operators of the benchmark, each result an output of the graph, so that nothing is fused
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

mlel = load_package()
from mlel_b200.graph_builder import GraphBuilder  # noqa: E402
from mlel_b200.model_graphs import (bert_graph, macs_of, matmul_rescale_graph, mobilenet_v2_graph,  # noqa: E402
                                    resnet50_graph)
from mlel_b200.runtime import GraphRunner  # noqa: E402

_TORCH = {np.dtype(np.int8): torch.int8, np.dtype(np.int16): torch.int16, np.dtype(np.int32): torch.int32}


def listed():
    return [
        # configuration 0: one 56x56x64 layer, a few microseconds of work
        {"name": "conv_56x56x64", "kind": "conv", "n": 1, "h": 56, "w": 56, "ic": 64, "oc": 64, "k": 3, "stride": 1,
         "replay": False},
        # configuration 1: 34 G multiply-adds on two activations
        {"name": "matmul_16x1024", "kind": "matmul", "n": 16, "h": 1024, "c": 1024, "w": 1024},
        # one image: the latency of 57 short kernels
        {"name": "resnet_1", "kind": "resnet", "n": 1, "image": 224, "classes": 1000, "host": False},
        # a request batch that arrives in host memory
        {"name": "resnet_16_host", "kind": "resnet", "n": 16, "image": 224, "classes": 1000, "host": True},
        # configuration 3: the throughput batch
        {"name": "resnet_64", "kind": "resnet", "n": 64, "image": 224, "classes": 1000, "host": False},
        {"name": "mobilenet_1", "kind": "mobilenet", "n": 1, "image": 224, "classes": 1000},
        # configuration 2
        {"name": "mobilenet_32", "kind": "mobilenet", "n": 32, "image": 224, "classes": 1000},
        # a few sequences, not padded to anything, through a shallow stack
        {"name": "bert_3x197", "kind": "bert", "n": 3, "seq": 197, "layers": 4},
        # configuration 4: 32 full sequences, 12 layers
        {"name": "bert_32x384", "kind": "bert", "n": 32, "seq": 384, "layers": 12},
        # one small video frame, 21 classes
        {"name": "segment_270x480", "kind": "segment", "n": 1, "h": 270, "w": 480, "width": 32, "classes": 21},
        # tensors that a cache keeps, sizes that no vector width divides
        {"name": "ops_odd", "kind": "ops", "n": 3, "hw": 57, "c": 36, "heads": 12, "seq": 197},
        # tensors well beyond the L2 cache, as the benchmark times its operators
        {"name": "ops_large", "kind": "ops", "n": 64, "hw": 112, "c": 64, "heads": 192, "seq": 384},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _channels(rng, lo, hi):
    """A channel count: mostly what layers have (a multiple of 8), otherwise any number (a head, a pruned layer)."""
    c = _log(rng, lo, hi)
    return c if rng.random() < 0.35 else max(8, (c + 7) // 8 * 8)


def draw(rng):
    kind = rng.choice(["conv", "matmul", "resnet", "mobilenet", "bert", "segment", "ops"])
    if kind == "conv":
        while True:
            c = {"kind": kind, "n": _log(rng, 1, 32), "h": _log(rng, 7, 112), "w": _log(rng, 7, 112),
                 "ic": _channels(rng, 3, 512), "oc": _channels(rng, 5, 512), "k": rng.choice([1, 3, 3, 5]),
                 "stride": rng.choice([1, 1, 2]), "replay": rng.random() < 0.5}
            if c["n"] * c["h"] * c["w"] * c["ic"] * c["oc"] * c["k"] ** 2 < 2e10:
                return c
    if kind == "matmul":
        def size(lo, hi):
            v = _log(rng, lo, hi)
            return v if rng.random() < 0.5 else max(16, v // 16 * 16)
        while True:
            c = {"kind": kind, "n": _log(rng, 1, 48), "h": size(16, 1024), "c": size(32, 1024), "w": size(16, 1024)}
            if c["n"] * c["h"] * c["c"] * c["w"] <= 16 * 1024 ** 3:
                return c
    if kind == "resnet":
        image, host = rng.randint(96, 256), rng.random() < 0.3
        n = min(_log(rng, 1, 64), int(64 * (224 / image) ** 2))
        return {"kind": kind, "n": n, "image": image, "classes": rng.choice([10, 100, 1000, 1001, rng.randint(2, 2000)]),
                "host": host}
    if kind == "mobilenet":
        image = rng.randint(96, 256)
        return {"kind": kind, "n": min(_log(rng, 1, 48), int(48 * (224 / image) ** 2)), "image": image,
                "classes": rng.choice([10, 100, 1000, 1001, rng.randint(2, 2000)])}
    if kind == "bert":
        seq = _log(rng, 16, 384)
        seq = seq if rng.random() < 0.5 else max(16, seq // 16 * 16)
        return {"kind": kind, "n": min(_log(rng, 1, 32), max(1, 6144 // seq)), "seq": seq, "layers": rng.choice([2, 4, 6])}
    if kind == "segment":
        h = _log(rng, 64, 540)
        w = _log(rng, max(64, h // 2), min(960, 2 * h))
        return {"kind": kind, "n": _log(rng, 1, max(1, min(8, 1000000 // (h * w)))), "h": h, "w": w,
                "width": rng.choice([16, 24, 32, 48]), "classes": rng.randint(2, 40)}
    hw, seq = _log(rng, 14, 112), _log(rng, 32, 384)
    n, heads = _log(rng, 1, 64), _log(rng, 1, 192)
    return {"kind": kind, "n": n, "hw": hw, "c": _channels(rng, 16, 96), "heads": heads,
            "seq": seq if rng.random() < 0.5 else max(32, seq // 16 * 16)}


# ---------------------------------------------------------------------------------------------------- the graphs

def _shift_for(k_elems):
    """A RESCALE shift that spreads sums of k products of random int8 values over the int8 range."""
    return 30 + max(1, math.ceil(math.log2(5460.0 * math.sqrt(k_elems) / 32.0)))


def _conv(g, rng, x, in_zp, oc, k, stride, out_zp, relu, depthwise=False):
    ic, pad = x.shape[3], k // 2
    if depthwise:
        w, oc, length = g.constant(rng.integers(-128, 128, (k, k, ic, 1), dtype=np.int8)), ic, k * k
    else:
        w, length = g.constant(rng.integers(-128, 128, (oc, k, k, ic), dtype=np.int8)), k * k * ic
    bias = g.constant(rng.integers(-(1 << 14), (1 << 14) + 1, (oc,), dtype=np.int32))
    mult = rng.integers(1 << 30, (1 << 31) - 1, (oc,), dtype=np.int64).astype(np.int32)
    shift = rng.integers(_shift_for(length), _shift_for(length) + 2, (oc,), dtype=np.int8)
    layer = g.depthwise_conv2d if depthwise else g.conv2d
    y = layer(x, w, bias, [pad] * 4, [stride] * 2, [1, 1], in_zp, 0)
    y = g.rescale(y, mult, shift, 0, out_zp, np.int8, double_round=True, per_channel=True)
    return g.clamp(y, out_zp, 127) if relu else y


def _conv_graph(seed, c):
    rng = np.random.Generator(np.random.PCG64(seed))
    g = GraphBuilder("conv2d_rescale")
    x = g.input(np.int8, (c["n"], c["h"], c["w"], c["ic"]))
    g.output(_conv(g, rng, x, -3, c["oc"], c["k"], c["stride"], 5, False))
    return g


def _segment_graph(seed, c):
    rng = np.random.Generator(np.random.PCG64(seed))
    g = GraphBuilder("segment")
    zp, width = -20, c["width"]
    x = g.input(np.int8, (c["n"], c["h"], c["w"], 3))

    def down(t):  # halves the frame, rounding up
        return g.max_pool2d(t, [2, 2], [2, 2], [0, t.shape[1] % 2, 0, t.shape[2] % 2])

    def up(t, skip):  # doubles the frame, cut to the skip connection's size, and joins the two
        t = g.resize(t, [4, 2, 4, 2], [0, 0], [2, 2], 1, np.int8)
        size = list(skip.shape[:3]) + [t.shape[3]]
        t = t if list(t.shape) == size else g.slice(t, [0, 0, 0, 0], size)
        return g.concat([t, skip], 3)

    a = _conv(g, rng, x, -3, width, 3, 1, zp, True)
    b = _conv(g, rng, down(a), zp, 2 * width, 3, 1, zp, True)
    t = _conv(g, rng, down(b), zp, 4 * width, 3, 1, zp, True)
    t = _conv(g, rng, up(t, b), zp, 2 * width, 3, 1, zp, True)
    t = _conv(g, rng, up(t, a), zp, width, 3, 1, zp, True)
    t = _conv(g, rng, t, zp, c["classes"], 1, 1, 0, False)
    g.output(t)
    g.output(g.argmax(t, 3))
    return g


def _ops_graph(seed, c):
    rng = np.random.Generator(np.random.PCG64(seed))
    g = GraphBuilder("ops")
    n, hw, ch, heads, seq = c["n"], c["hw"], c["c"], c["heads"], c["seq"]
    x = g.input(np.int8, (n, hw, hw, ch))
    s = g.input(np.int32, (heads, seq, seq))
    s16 = g.input(np.int16, (heads, seq, seq))
    row = g.input(np.int32, (heads, seq, 1))
    t = g.input(np.int8, (max(1, heads // 12), seq, 12, 64))
    g.output(g.clamp(x, -20, 127))
    g.output(g.table(x, rng.integers(-128, 128, (256,), dtype=np.int8)))
    g.output(g.max_pool2d(x, [3, 3], [2, 2], [1, 1, 1, 1]))
    g.output(g.avg_pool2d(x, [hw, hw], [hw, hw], [0, 0, 0, 0], -20, -20))
    g.output(_conv(g, rng, x, -5, ch, 3, 1, 0, False, depthwise=True))
    g.output(g.rescale(s, [1 << 30], [38], 0, 0, np.int8, double_round=True))
    g.output(g.sub(s, row))
    g.output(g.reduce("REDUCE_SUM", s, 2))
    g.output(g.table(s16, rng.integers(-32768, 32768, (513,), dtype=np.int16)))
    g.output(g.transpose(t, (0, 2, 1, 3)))
    g.output(g.transpose(t, (0, 2, 3, 1)))
    g.output(g.concat([t, t], 3))
    return g


def _graph(c, seed):
    kind = c["kind"]
    if kind == "conv":
        return _conv_graph(seed, c)
    if kind == "matmul":
        return matmul_rescale_graph(seed, c["n"], c["h"], c["c"], c["w"], double_round=True)[0]
    if kind == "resnet":
        return resnet50_graph(seed, c["n"], c["image"], classes=c["classes"])[0]
    if kind == "mobilenet":
        return mobilenet_v2_graph(seed, c["n"], c["image"], classes=c["classes"])[0]
    if kind == "bert":
        return bert_graph(seed, c["n"], c["seq"], layers=c["layers"])[0]
    return _segment_graph(seed, c) if kind == "segment" else _ops_graph(seed, c)


# ------------------------------------------------------------------------------------------------ one case's passes

def prepare(case, seed):
    runner = GraphRunner(_graph(case, seed))
    gen = torch.Generator("cuda").manual_seed(seed)
    for (_, _, value), t in zip(runner._in_keys, runner.inputs):
        if value.dtype == np.int32:  # accumulators of a few thousand products
            t.view(torch.int32).random_(-(1 << 20), 1 << 20, generator=gen)
        else:  # int8 and int16 over their whole range
            t.random_(0, 256, generator=gen)
    outputs = [t.view(_TORCH[v.dtype]).reshape(v.shape) for (_, _, v), t in zip(runner._out_keys, runner.outputs)]
    state = {"runner": runner, "outputs": outputs, "replay": case.get("replay", True), "host": case.get("host", False)}
    if state["host"]:
        keys = runner._in_keys + runner._out_keys
        pinned = [t.cpu().pin_memory() for t in runner.inputs + runner.outputs]
        state["pinned"] = pinned
        io = [(s, b, 0, p.data_ptr(), p.numel()) for (s, b, _), p in zip(keys, pinned)]
        state["in"], state["out"] = io[:len(runner.inputs)], io[len(runner.inputs):]
        state["outputs"] = [p.view(_TORCH[v.dtype]).reshape(v.shape)
                            for (_, _, v), p in zip(runner._out_keys, pinned[len(runner.inputs):])]
    torch.cuda.synchronize()
    return state


def run(state):
    if state["host"]:
        state["runner"].session.run_host(state["in"], state["out"], torch.cuda.current_stream().cuda_stream)
    else:
        state["runner"].dispatch(use_cuda_graph=state["replay"])
    return state["outputs"]


def work(case):
    """Inputs, constants and outputs once; two operations per multiply-add."""
    g = _graph(case, 0)
    size = lambda v: int(np.prod(v.shape)) * v.dtype.itemsize  # noqa: E731
    moved = sum(size(v) for v in g.inputs) + sum(size(v) for v, _, _ in g.outputs)
    moved += sum(a.nbytes for a in g.constants.values())
    return {"bytes": moved, "flops": 2 * macs_of(g)}


def tolerance(case):
    return "exact"
