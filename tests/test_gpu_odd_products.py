"""GPU parity of int8 products whose row lengths are no multiple of 16: copies with padded rows, transposes by a cluster,
rows of output at odd addresses.  Bit-exact against the CPU oracle."""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.test_gpu_small import conv
from tests.test_gpu_vector_ops import check, check_fused

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,rows,k,n", [
    (1, 1, 1, 1), (1, 17, 33, 15), (3, 64, 100, 48), (2, 130, 197, 197), (5, 197, 64, 197), (1, 128, 127, 256), (2, 200, 1023, 272),
    (2, 129, 640, 129), (1, 31, 4100, 50), (3, 257, 144, 301),
])
@pytest.mark.parametrize("constant", [False, True])
def test_products_of_every_row_length(mlel, batch, rows, k, n, constant):
    r = np.random.Generator(np.random.PCG64(rows * k + n))
    a8, b8 = (r.integers(-128, 128, s, dtype=np.int8) for s in ((batch, rows, k), (batch, k, n)))
    g = GraphBuilder()
    a = g.input(np.int8, a8.shape)
    b = g.constant(b8) if constant else g.input(np.int8, b8.shape)
    g.output(g.matmul(a, b, -20, 0))
    for shift in (34, 40):
        g.output(g.rescale(g.matmul(a, b, 3, 0), [1 << 30 | 12345], [shift], 0, 1, np.int8, double_round=True))
    check(g, [a8] if constant else [a8, b8])


@pytest.mark.parametrize("channels", [5, 21, 34, 150])
def test_rows_at_odd_addresses_with_residual_tail(mlel, channels):
    r = np.random.Generator(np.random.PCG64(channels))
    g = GraphBuilder()
    x = g.input(np.int8, (2, 40, 41, channels))
    y = conv(g, r, x, channels, 1, 1, 0, 4, True)
    a = g.rescale(y, [int(r.integers(1 << 30, 1 << 31))], [23], 4, 0, np.int32)
    b = g.rescale(x, [int(r.integers(1 << 30, 1 << 31))], [23], -3, 0, np.int32)
    g.output(g.rescale(g.add(a, b), [int(r.integers(1 << 30, 1 << 31))], [40], 0, -20, np.int8, double_round=True))
    g.output(conv(g, r, x, channels, 3, 1, 1, 4, True))
    check(g, [r.integers(-128, 128, x.shape, dtype=np.int8)])


@pytest.mark.parametrize("n,hw,ic,oc,k,stride", [
    (2, 40, 64, 65, 1, 1), (8, 30, 256, 255, 1, 1), (4, 41, 128, 131, 3, 1), (3, 57, 48, 200 + 1, 3, 2), (1, 300, 16, 127, 1, 1),
    (9, 56, 32, 385, 1, 1), (2, 33, 50, 90, 1, 1),
])
def test_wide_convolutions_with_rows_at_odd_addresses(mlel, n, hw, ic, oc, k, stride):
    r = np.random.Generator(np.random.PCG64(hw + oc))
    g = GraphBuilder()
    x = g.input(np.int8, (n, hw, hw, ic))
    y = conv(g, r, x, oc, k, stride, k // 2, -7, True)
    g.output(conv(g, r, y, oc, 1, 1, 0, 4, False))
    g.output(conv(g, r, x, oc, k, stride, k // 2, 5, False, 33))
    check(g, [r.integers(-128, 128, x.shape, dtype=np.int8)])


@pytest.mark.parametrize("n,hw,ic,oc,k,stride", [
    (1, 17, 9, 51, 3, 1), (2, 23, 20, 48, 3, 1), (2, 30, 33, 32, 5, 2), (1, 14, 75, 125, 3, 2), (3, 28, 130, 64, 3, 1), (1, 40, 250, 200, 3, 1),
    (1, 9, 24, 144, 1, 1), (2, 19, 17, 64, 1, 2),
])
def test_convolutions_over_padded_channels(mlel, n, hw, ic, oc, k, stride):
    r = np.random.Generator(np.random.PCG64(hw + ic))
    g = GraphBuilder()
    x = g.input(np.int8, (n, hw, hw, ic))
    g.output(conv(g, r, x, oc, k, stride, k // 2, -7, True))
    g.output(conv(g, r, x, oc, k, stride, 0, 5, False, 33))
    w, b = g.constant(r.integers(-128, 128, (oc, k, k, ic), dtype=np.int8)), g.constant(r.integers(-999, 999, (oc,), dtype=np.int32))
    g.output(g.conv2d(x, w, b, [k // 2] * 4, [stride] * 2, [1, 1], 3, 0))
    check(g, [r.integers(-128, 128, x.shape, dtype=np.int8)])


@pytest.mark.parametrize("batch,rows,k,n,paired", [
    (37, 130, 70, 151, False), (38, 130, 70, 151, True), (1, 19 * 128, 33, 8 * 128 - 1, True), (3, 5000, 64, 255, True), (40, 200, 300, 385, True),
])
@pytest.mark.parametrize("constant", [False, True])
def test_products_with_rows_at_odd_addresses_where_the_paired_kernel_begins(mlel, batch, rows, k, n, paired, constant):
    """More 128 x 128 tiles than SMs (148); widths of all three tile sizes, one to four channel tiles."""
    import ctypes
    lib = mlel.lib()
    lib.mlel_tensor_core_launches.restype = ctypes.c_longlong
    r = np.random.Generator(np.random.PCG64(rows * k + n))
    a8, b8 = (r.integers(-128, 128, s, dtype=np.int8) for s in ((batch, rows, k), (batch, k, n)))
    g = GraphBuilder()
    a = g.input(np.int8, a8.shape)
    b = g.constant(b8) if constant else g.input(np.int8, b8.shape)
    for shift in (34, 40):
        y = g.rescale(g.matmul(a, b, 3, 0), [1 << 30 | 12345], [shift], 0, 1, np.int8, double_round=True)
        g.output(y)
    before = lib.mlel_tensor_core_launches(2)
    check_fused(mlel, g, [a8] if constant else [a8, b8], ["MATMUL+RESCALE"])
    assert (lib.mlel_tensor_core_launches(2) > before) == paired


@pytest.mark.parametrize("batch,rows,k,n", [(4, 17, 55, 384), (1, 9, 14, 272), (2, 300, 129, 640), (1, 1, 1, 144), (3, 40, 100, 128)])
def test_product_of_activations_with_copied_rows_as_a_session(mlel, batch, rows, k, n):
    """Three launches: enqueued where the second operand is read where it lies, replayed where it is transposed (the last).
    New inputs at every pass, both ways in turn."""
    from mlel_b200.runtime import GraphRunner
    from tests.graph_eval import evaluate
    r = np.random.Generator(np.random.PCG64(rows + n))
    g = GraphBuilder()
    a, b = g.input(np.int8, (batch, rows, k)), g.input(np.int8, (batch, k, n))
    g.output(g.rescale(g.matmul(a, b, 3, 0), [1 << 30 | 12345], [37], 0, 1, np.int8, double_round=True))
    runner = GraphRunner(g)
    for use_cuda_graph in (True, False, True, True):
        data = [r.integers(-128, 128, t.shape, dtype=np.int8) for t in (a, b)]
        np.testing.assert_array_equal(runner.run(data, use_cuda_graph=use_cuda_graph)[0], evaluate(g, data)[0])
