"""GPU parity of the element-wise, movement and pooling kernels at sizes that no vector width divides.

Every size here leaves a remainder at one of the kernels' units: last groups of fewer than four or sixteen elements, rows
of odd length, channel counts that allow only 1-, 2-, 4- or 8-byte accesses, tiles of 64 x 64 with ragged edges, windows
cut by the image border.  All comparisons are bit-exact against the CPU oracle.
"""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.test_gpu_vector_ops import check, full_range, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 5, 7), (2, 33, 197), (1, 7, 128), (5, 4, 66)])
def test_elementwise_and_reductions(mlel, shape):
    r = rng(sum(shape))
    x8, x16 = full_range(r, np.int8, shape), full_range(r, np.int16, shape)
    x32, y32 = full_range(r, np.int32, shape), full_range(r, np.int32, shape)
    row = full_range(r, np.int32, shape[:2] + (1,))
    g = GraphBuilder()
    a8, a16, a32, b32 = (g.input(d.dtype, shape) for d in (x8, x16, x32, y32))
    rw = g.input(np.int32, row.shape)
    g.output(g.clamp(a8, -20, 99))
    g.output(g.table(a8, full_range(r, np.int8, (256,))))
    g.output(g.table(a16, full_range(r, np.int16, (513,))))
    g.output(g.add(a32, b32))
    g.output(g.sub(a32, rw))
    g.output(g.mul(a32, rw, 17))
    for x in (a8, a16, a32):
        for op in ("REDUCE_SUM", "REDUCE_MAX", "REDUCE_MIN"):
            g.output(g.reduce(op, x, 2))
    mult = r.integers(1 << 30, (1 << 31) - 1, (shape[2],), dtype=np.int64).astype(np.int32)
    shift = r.integers(31, 40, (shape[2],), dtype=np.int8)
    g.output(g.rescale(a32, mult, shift, 0, 3, np.int8, double_round=True, per_channel=True))
    g.output(g.rescale(a32, mult[:1], shift[:1], 5, -3, np.int16, double_round=True))
    g.output(g.rescale(a8, mult[:1], [20], 5, 0, np.int32))
    check(g, [x8, x16, x32, y32, row])


@pytest.mark.parametrize("dtype", [np.int8, np.int16, np.int32])
@pytest.mark.parametrize("shape,perms", [
    ((2, 65, 3, 64), (0, 2, 3, 1)),      # tiles with one row or column over
    ((3, 197, 12, 30), (0, 2, 1, 3)),    # runs of 30 elements
    ((5, 9, 7), (2, 1, 0)),              # too thin for tiles
    ((63, 129), (1, 0)),
    ((2, 3, 5, 8, 9), (4, 2, 0, 1, 3)),
])
def test_transpose(mlel, dtype, shape, perms):
    r = rng(len(shape))
    g = GraphBuilder()
    x = g.input(dtype, shape)
    g.output(g.transpose(x, perms))
    check(g, [full_range(r, dtype, shape)])


@pytest.mark.parametrize("channels", [1, 2, 3, 5, 8, 12, 16, 21, 48, 100, 130])
def test_channel_rows(mlel, channels):
    """CONCAT, SLICE, RESIZE, TILE, REVERSE, ARGMAX and the pools over every width of channel row."""
    r = rng(channels)
    shape, other = (2, 9, 7, channels), (2, 9, 7, channels + 3)
    g = GraphBuilder()
    x, y = g.input(np.int8, shape), g.input(np.int8, other)
    g.output(g.concat([x, y, x], 3))
    g.output(g.concat([x, x], 1))
    g.output(g.slice(x, [1, 2, 1, 0], [1, 5, 4, channels]))
    g.output(g.slice(y, [0, 0, 0, 2], [2, 9, 7, channels]))
    g.output(g.resize(x, [4, 2, 4, 2], [0, 0], [2, 2], 1, np.int8))
    g.output(g.resize(x, [3, 2, 5, 3], [-1, 1], [1, 0], 1, np.int8))
    g.output(g.tile(x, [1, 2, 1, 3]))
    g.output(g.reverse(x, 3))
    g.output(g.reverse(x, 1))
    g.output(g.argmax(x, 3))
    g.output(g.max_pool2d(x, [3, 3], [2, 2], [1, 1, 1, 1]))
    g.output(g.max_pool2d(x, [2, 2], [2, 2], [0, 1, 0, 1]))
    g.output(g.avg_pool2d(x, [9, 7], [9, 7], [0, 0, 0, 0], -20, 3))
    g.output(g.avg_pool2d(x, [5, 4], [2, 3], [2, 2, 1, 2], 7, -5))
    check(g, [full_range(r, np.int8, shape), full_range(r, np.int8, other)])


@pytest.mark.parametrize("n,hw,channels", [(1, 57, 36), (2, 64, 64), (1, 33, 1030), (1, 41, 257), (3, 12, 2048)])
def test_global_average_pool_split_over_blocks(mlel, n, hw, channels):
    r = rng(hw)
    g = GraphBuilder()
    x = g.input(np.int8, (n, hw, hw + 1, channels))
    g.output(g.avg_pool2d(x, [hw, hw + 1], [hw, hw + 1], [0, 0, 0, 0], -20, -20))
    g.output(g.avg_pool2d(x, [hw, hw], [hw, hw], [0, 0, 0, 0], -128, 5))  # rows of the window are not joined
    check(g, [full_range(r, np.int8, (n, hw, hw + 1, channels))])


@pytest.mark.parametrize("dtype", [np.int8, np.int16, np.int32])
@pytest.mark.parametrize("rows,length", [(1, 1), (257, 21), (300, 32), (70, 129), (5, 1000)])
def test_argmax_rows(mlel, dtype, rows, length):
    r = rng(length)
    data = full_range(r, dtype, (rows, length))
    data[rows // 2] = np.iinfo(dtype).min  # nothing above the start value: index 0
    data[0, :] = data[0, 0]                # ties: the first wins
    g = GraphBuilder()
    g.output(g.argmax(g.input(dtype, (rows, length)), 1))
    check(g, [data])


def test_consecutive_concat_passes_are_one_node(mlel):
    from mlel_b200.runtime import GraphRunner
    from tests.graph_eval import evaluate
    r = rng(3)
    g = GraphBuilder()
    xs = [g.input(np.int8, (2, 3, c)) for c in (4, 1, 16, 7, 32, 2)]
    g.output(g.concat([g.clamp(x, -100, 100) for x in xs], 2))
    inputs = [full_range(r, np.int8, x.shape) for x in xs]
    runner = GraphRunner(g)
    assert runner.pipeline.exec_names().count("CONCAT") == 1
    for a, b in zip(runner.run(inputs), evaluate(g, inputs)):
        np.testing.assert_array_equal(a, b)
