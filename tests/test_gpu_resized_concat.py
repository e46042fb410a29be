"""GPU parity of CONCAT along the channels whose inputs are enlarged (and cut) tensors, read where their pixels come from: channel
counts of every unit width, frame sizes that the enlargement overshoots, slices that start inside, several enlarged inputs; and
graphs in which a step is wanted elsewhere.  Bit-exact against the CPU oracle."""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate

pytestmark = pytest.mark.gpu


def check(g, r, launches=None):
    from mlel_b200.runtime import GraphRunner
    data = [r.integers(-128, 128, v.shape).astype(v.dtype) for v in g.inputs]
    want = evaluate(g, data)
    runner = GraphRunner(g)
    if launches is not None:
        assert runner.pipeline.exec_names() == launches
    for use_cuda_graph in (False, True):
        for a, b in zip(runner.run(data, use_cuda_graph=use_cuda_graph), want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("h,w", [(1, 1), (5, 8), (27, 31), (100, 67)])
@pytest.mark.parametrize("channels", [(32, 16), (24, 8), (4, 12), (6, 2), (3, 5)])
def test_enlarged_beside_a_skip(mlel, h, w, channels):
    r = np.random.Generator(np.random.PCG64(h * 100 + channels[0]))
    g = GraphBuilder()
    small = g.input(np.int8, (2, (h + 1) // 2, (w + 1) // 2, channels[0]))
    skip = g.input(np.int8, (2, h, w, channels[1]))
    t = g.resize(small, [4, 2, 4, 2], [0, 0], [2, 2], 1, np.int8)
    name = "RESIZE+CONCAT"
    if t.shape != (2, h, w, channels[0]):
        t = g.slice(t, [0, 0, 0, 0], [2, h, w, channels[0]])
        name = "SLICE+RESIZE+CONCAT"
    g.output(g.concat([t, skip], 3))
    check(g, r, [name])


@pytest.mark.parametrize("scale,offset,border,out", [([3, 2, 5, 2], [0, 0], [1, 1], None), ([4, 2, 6, 2], [-1, 2], [3, 1], None), ([1, 2, 1, 3], [0, 0], [0, 0], None)])
def test_other_scales_slices_and_orders(mlel, scale, offset, border, out):
    r = np.random.Generator(np.random.PCG64(scale[0]))
    g = GraphBuilder()
    a, b = g.input(np.int8, (1, 13, 19, 16)), g.input(np.int8, (1, 13, 19, 8))
    ra, rb = (g.resize(t, scale, offset, border, 1, np.int8) for t in (a, b))
    h, w = ra.shape[1], ra.shape[2]
    size = [1, max(1, h - 3), max(1, w - 2)]
    start = [0, min(2, h - size[1]), min(1, w - size[2]), 0]
    skip = g.input(np.int8, (1, size[1], size[2], 4))
    g.output(g.concat([g.slice(ra, start, size + [16]), skip, g.slice(rb, start, size + [8])], 3))
    check(g, r)


def test_steps_that_are_wanted_elsewhere_remain(mlel):
    r = np.random.Generator(np.random.PCG64(1))
    g = GraphBuilder()
    small, skip = g.input(np.int8, (1, 8, 8, 16)), g.input(np.int8, (1, 16, 16, 16))
    t = g.resize(small, [4, 2, 4, 2], [0, 0], [2, 2], 1, np.int8)
    g.output(g.concat([t, skip], 3))
    g.output(t)                       # the enlarged tensor is a result
    u = g.resize(skip, [4, 2, 4, 2], [0, 0], [2, 2], 1, np.int8)
    g.output(g.concat([u, u], 3))     # read twice
    v = g.resize(small, [4, 2, 4, 2], [0, 0], [2, 2], 1, np.int8)
    g.output(g.concat([v, skip], 2))  # along the columns
    check(g, r)
