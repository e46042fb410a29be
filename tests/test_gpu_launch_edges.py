"""Programmatic dependent launches: which launches ask for them, and contractions directly behind and in front of operators that a
replayed graph has on lanes of their own (several launches precede the first one behind them, and it takes no dependent launch)."""
import ctypes

import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate
from tests.test_gpu_attention import ATTENTION, attention_graph

pytestmark = pytest.mark.gpu

NORM = "ROWS(RESCALE+RESCALE+ADD+REDUCE_SUM+MUL+SUB+MUL+REDUCE_SUM+MUL+RESCALE+TABLE+MUL+RESCALE"
PIXEL_MAJOR, CHANNEL_MAJOR, PAIRED, SMALL, WINDOW = range(5)


def rng(seed):
    return np.random.Generator(np.random.PCG64(seed))


def conv(g, r, x, oc, k, in_zp=0, out_zp=0):
    w = g.constant(r.integers(-128, 128, (oc, k, k, x.shape[3]), dtype=np.int8))
    b = g.constant(r.integers(-(1 << 12), 1 << 12, (oc,), dtype=np.int32))
    y = g.conv2d(x, w, b, [k // 2] * 4, [1, 1], [1, 1], in_zp, 0)
    return g.rescale(y, r.integers(1 << 30, (1 << 31) - 1, (oc,), dtype=np.int64).astype(np.int32),
                     r.integers(38, 43, (oc,), dtype=np.int8), 0, out_zp, np.int8, True, True, True)


def product(g, r, x, columns):
    w = g.constant(r.integers(-128, 128, (1, x.shape[2], columns), dtype=np.int8))
    return g.rescale(g.matmul(x, w, 0, 0), [1 << 30], [39], 0, 0, np.int8)


def norm(g, r, x, y):
    from tests.test_gpu_vector_ops import _norm_chain
    t = g.add(g.rescale(x, [1 << 30], [24], 0, 0, np.int32), g.rescale(y, [1 << 30], [24], 0, 0, np.int32))
    return _norm_chain(g, r, t, x.shape[-1])[0]


# name -> (input shape, the contraction, the kernel it runs on or None)
BODIES = {
    "paired": ((1, 2048, 256), lambda g, r, x, y: product(g, r, x, 768), PAIRED),
    "small": ((1, 100, 256), lambda g, r, x, y: product(g, r, x, 256), SMALL),
    "channel-major pair": ((24, 28, 28, 256), lambda g, r, x, y: conv(g, r, conv(g, r, x, 256, 1), 256, 3), CHANNEL_MAJOR),
    "window": ((4, 56, 56, 64), lambda g, r, x, y: conv(g, r, x, 64, 3), WINDOW),
    "pixel-major": ((4, 56, 56, 96), lambda g, r, x, y: conv(g, r, x, 24, 1), PIXEL_MAJOR),
    "layer norm": ((1, 300, 256), norm, None),
}


def programmatic_edges(runner, dependent_launch, mlel):
    """Edges of that kind in what a dispatch puts into a capturing stream.  Nothing is launched."""
    import torch
    cudart = ctypes.CDLL("libcudart.so.12")
    stream = torch.cuda.Stream().cuda_stream
    graph, count = ctypes.c_void_p(), ctypes.c_size_t()
    assert mlel.lib().mlel_set_tuning(b"dependent_launch", dependent_launch) == 0
    try:
        assert cudart.cudaStreamBeginCapture(ctypes.c_void_p(stream), 1) == 0  # thread-local mode
        try:
            runner.session.dispatch(stream)
        finally:
            assert cudart.cudaStreamEndCapture(ctypes.c_void_p(stream), ctypes.byref(graph)) == 0
    finally:
        assert mlel.lib().mlel_set_tuning(b"dependent_launch", 1) == 0
    edges = cudart.cudaGraphGetEdges_v2
    assert edges(graph, None, None, None, ctypes.byref(count)) == 0
    assert count.value > 0
    source, target = (ctypes.c_void_p * count.value)(), (ctypes.c_void_p * count.value)()
    data = (ctypes.c_ubyte * (8 * count.value))()  # from_port, to_port, type (1: programmatic), five reserved
    assert edges(graph, source, target, data, ctypes.byref(count)) == 0
    assert cudart.cudaGraphDestroy(graph) == 0
    return sum(data[8 * k + 2] == 1 for k in range(count.value))


@pytest.mark.parametrize("name", list(BODIES) + ["attention"])
def test_dependent_launches_are_the_tunings_choice(mlel, name):
    """Every kernel asks the one function: with "dependent_launch" 0 no launch depends programmatically on the one before it."""
    from mlel_b200.runtime import GraphRunner
    if name == "attention":
        g, data = attention_graph(2, 4, 128, 128, 64)
    else:
        shape, body, _ = BODIES[name]
        g, r = GraphBuilder(), rng(5)
        a, b = g.input(np.int8, shape), g.input(np.int8, shape)
        a, b = g.reverse(a, 1), g.reverse(b, 1)
        g.output(body(g, r, a, b))
        g.output(b)
        data = [r.integers(-128, 128, shape, dtype=np.int8) for _ in range(2)]
    runner = GraphRunner(g)
    runner.run(data)
    assert programmatic_edges(runner, 1, mlel) > 0
    assert programmatic_edges(runner, 0, mlel) == 0


@pytest.mark.parametrize("name", BODIES)
@pytest.mark.parametrize("seed", range(2))
def test_contractions_between_lanes(mlel, name, seed):
    """Independent operators, of which the contraction reads two, then the contraction, then independent ones that read it."""
    from mlel_b200.runtime import GraphRunner
    lib = mlel.lib()
    lib.mlel_tensor_core_launches.restype = ctypes.c_longlong
    shape, body, kernel = BODIES[name]
    r = rng(seed)
    g = GraphBuilder()
    inputs = [g.input(np.int8, shape) for _ in range(3)]
    before = [g.clamp(x, -int(r.integers(60, 128)), int(r.integers(60, 127))) for x in inputs]
    before.append(g.table(inputs[0], r.integers(-128, 128, (256,), dtype=np.int8)))
    before.append(g.reverse(inputs[1], 1))
    y = body(g, r, before[3], before[4])
    after = [g.clamp(y, -50, 60), g.table(y, r.integers(-128, 128, (256,), dtype=np.int8)), g.reverse(y, 1), g.reverse(before[2], 1)]
    for v in [y, *before[:3], *after]:
        g.output(v)
    data = [r.integers(-128, 128, shape, dtype=np.int8) for _ in range(3)]
    want = evaluate(g, data)
    runner = GraphRunner(g)
    names = runner.pipeline.exec_names()
    assert kernel is not None or any(name.startswith(NORM) for name in names), names
    launches = lib.mlel_tensor_core_launches(kernel) if kernel is not None else 0
    for use_cuda_graph in (True, True, False):
        for t in runner.outputs:
            t.zero_()
        for a, b in zip(runner.run(data, use_cuda_graph=use_cuda_graph), want):
            np.testing.assert_array_equal(a, b)
    assert kernel is None or lib.mlel_tensor_core_launches(kernel) > launches


def test_attention_between_lanes(mlel):
    """The three inputs pass through independent operators, and two of the attention's inputs are read again behind it."""
    from mlel_b200.runtime import GraphRunner
    g, data = attention_graph(2, 4, 130, 130, 64, seed=3)
    context = g.outputs[0][0]
    for v in (g.reverse(context, 1), g.clamp(context, -3, 90), g.reverse(g.inputs[0], 1), g.clamp(g.inputs[2], -9, 9)):
        g.output(v)
    want = evaluate(g, data)
    runner = GraphRunner(g)
    assert ATTENTION in runner.pipeline.exec_names()
    for use_cuda_graph in (True, True, False):
        for t in runner.outputs:
            t.zero_()
        for a, b in zip(runner.run(data, use_cuda_graph=use_cuda_graph), want):
            np.testing.assert_array_equal(a, b)
