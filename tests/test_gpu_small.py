"""GPU parity of the small-problem kernel: pixel counts at and beside its 32- and 64-pixel tiles, K blocks fewer, equal
and more than the CTAs that share them, channel counts that are no multiple of 16, residual tails, border classes, shifts
on both sides of 32.  Bit-exact against the CPU oracle; a counter tells that the kernel took the case."""
import ctypes

import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate

pytestmark = pytest.mark.gpu


def run(mlel, g, inputs, expect_small=True):
    from mlel_b200.runtime import GraphRunner
    lib = mlel.lib()
    lib.mlel_tensor_core_launches.restype = ctypes.c_longlong
    want = evaluate(g, inputs)
    before = lib.mlel_tensor_core_launches(3)
    runner = GraphRunner(g)
    for use_cuda_graph in (False, True, True):
        for a, b in zip(runner.run(inputs, use_cuda_graph=use_cuda_graph), want):
            bad = np.argwhere(a != b)
            assert len(bad) == 0, (len(bad), a.size, bad[0].tolist(), bad[-1].tolist())
    assert (lib.mlel_tensor_core_launches(3) > before) == expect_small


def conv(g, r, x, oc, k, stride, pad, in_zp, relu, base_shift=37, dil=1):
    w = g.constant(r.integers(-128, 128, (oc, k, k, x.shape[3]), dtype=np.int8))
    b = g.constant(r.integers(-(1 << 14), 1 << 14, (oc,), dtype=np.int32))
    mult = r.integers(1 << 30, (1 << 31) - 1, (oc,), dtype=np.int64).astype(np.int32)
    y = g.conv2d(x, w, b, [pad] * 4, [stride] * 2, [dil] * 2, in_zp, 0)
    y = g.rescale(y, mult, r.integers(base_shift, base_shift + 3, (oc,), dtype=np.int8), 0, 4, np.int8, double_round=True,
                  per_channel=True)
    return g.clamp(y, 4, 127) if relu else y


@pytest.mark.parametrize("n,hw,ic,oc,k,stride,shift", [
    (1, 14, 256, 256, 3, 1, 38), (1, 7, 512, 512, 3, 1, 39), (1, 1, 64, 16, 1, 1, 36), (1, 5, 16, 21, 1, 1, 34),
    (2, 9, 144, 130, 3, 2, 37), (1, 33, 128, 128, 1, 1, 31), (3, 7, 2048, 1001, 1, 1, 38), (1, 56, 64, 64, 3, 1, 37),
    (1, 8, 32, 5, 5, 1, 29), (4, 14, 1024, 256, 1, 1, 38), (1, 13, 48, 96, 3, 1, 40),
])
def test_convolutions(mlel, n, hw, ic, oc, k, stride, shift):
    r = np.random.Generator(np.random.PCG64(hw * 1000 + oc))
    g = GraphBuilder()
    x = g.input(np.int8, (n, hw, hw, ic))
    g.output(conv(g, r, x, oc, k, stride, k // 2, -7, False, shift))
    g.output(conv(g, r, x, oc, k, stride, k // 2, 5, True, shift))
    run(mlel, g, [r.integers(-128, 128, x.shape, dtype=np.int8)])


@pytest.mark.parametrize("tile", [101, 102, 104, 108, 201, 202, 204, 208])
@pytest.mark.parametrize("hw,ic,oc", [(9, 1024, 256), (6, 272, 70), (15, 128, 128)])
def test_every_tile_and_split_with_residual_tail(mlel, tile, hw, ic, oc):
    """A bottleneck whose last convolution carries the residual add, on every tile width and cluster size."""
    r = np.random.Generator(np.random.PCG64(tile + hw))
    g = GraphBuilder()
    x = g.input(np.int8, (1, hw, hw, ic))
    t = conv(g, r, x, oc, 3, 1, 1, -3, True)
    y = conv(g, r, t, ic, 1, 1, 0, 4, False)
    a = g.rescale(y, [int(r.integers(1 << 30, 1 << 31))], [23], 4, 0, np.int32)
    b = g.rescale(x, [int(r.integers(1 << 30, 1 << 31))], [23], -3, 0, np.int32)
    y = g.rescale(g.add(a, b), [int(r.integers(1 << 30, 1 << 31))], [40], 0, -20, np.int8, double_round=True)
    g.output(g.clamp(y, -20, 127))
    lib = mlel.lib()
    try:
        assert lib.mlel_set_tuning(b"small_kernel", tile) == 0
        run(mlel, g, [r.integers(-128, 128, x.shape, dtype=np.int8)])
    finally:
        assert lib.mlel_set_tuning(b"small_kernel", 1) == 0


@pytest.mark.parametrize("tile,oc,relu", [(101, 70, True), (204, 130, False), (102, 16, False)])
def test_residual_tail_without_a_table(mlel, tile, oc, relu):
    """Behind a convolution over padded channels the tail has no table: its RESCALEs are evaluated."""
    r = np.random.Generator(np.random.PCG64(tile + oc))
    g = GraphBuilder()
    x, short = g.input(np.int8, (1, 9, 11, 40)), g.input(np.int8, (1, 9, 11, oc))
    y = conv(g, r, x, oc, 3, 1, 1, -3, relu)
    a = g.rescale(y, [int(r.integers(1 << 30, 1 << 31))], [23], 4, 0, np.int32)
    b = g.rescale(short, [int(r.integers(1 << 30, 1 << 31))], [23], -3, 0, np.int32)
    g.output(g.rescale(g.add(a, b), [int(r.integers(1 << 30, 1 << 31))], [40], 0, -20, np.int8, double_round=True))
    lib = mlel.lib()
    try:
        assert lib.mlel_set_tuning(b"small_kernel", tile) == 0
        run(mlel, g, [r.integers(-128, 128, v.shape, dtype=np.int8) for v in (x, short)])
    finally:
        assert lib.mlel_set_tuning(b"small_kernel", 1) == 0


@pytest.mark.parametrize("rows,k,n", [(1, 2048, 1000), (64, 768, 768), (33, 80, 10), (1, 16, 1), (130, 3072, 768)])
def test_products_with_constant_weights(mlel, rows, k, n):
    r = np.random.Generator(np.random.PCG64(rows + n))
    g = GraphBuilder()
    a = g.input(np.int8, (1, rows, k))
    w = g.constant(r.integers(-128, 128, (1, k, n), dtype=np.int8))
    mult = r.integers(1 << 30, (1 << 31) - 1, (n,), dtype=np.int64).astype(np.int32)
    g.output(g.rescale(g.matmul(a, w, -20, 0), mult, np.full((n,), 38, np.int8), 0, 1, np.int8, double_round=True, per_channel=True))
    run(mlel, g, [r.integers(-128, 128, a.shape, dtype=np.int8)])


def test_hand_over_between_channel_major_launches_without_the_small_kernel(mlel):
    """The chains of the tile-level hand-over on the kernels that implement it, whatever kernel small problems take."""
    from tests.test_gpu_tile_handover import CASES, bottleneck_chain, _run
    lib = mlel.lib()
    try:
        assert lib.mlel_set_tuning(b"small_kernel", 0) == 0
        for case in CASES:
            g, inputs = bottleneck_chain(*case)
            want = evaluate(g, inputs)
            _run(mlel, g, inputs, want, use_cuda_graph=False, times=2)
            _run(mlel, g, inputs, want, use_cuda_graph=True, times=3)
    finally:
        assert lib.mlel_set_tuning(b"small_kernel", 1) == 0


@pytest.mark.parametrize("ic", [640, 736, 752, 768])  # 45 K blocks at 4 to a tile of 32 pixels; 54 at 8 to one of 64
def test_tile_width_goes_by_the_blocks_of_a_cta(mlel, ic):
    from mlel_b200.runtime import GraphRunner
    r = np.random.Generator(np.random.PCG64(ic))
    g = GraphBuilder()
    x = g.input(np.int8, (2, 33, 33, ic))
    g.output(conv(g, r, x, 16, 3, 1, 1, -5, False, base_shift=41))
    data = [r.integers(-128, 128, x.shape, dtype=np.int8)]
    before = mlel.lib().mlel_tensor_core_launches(3)
    got = GraphRunner(g).run(data)[0]
    assert mlel.lib().mlel_tensor_core_launches(3) == before + 1
    np.testing.assert_array_equal(got, evaluate(g, data)[0])


@pytest.mark.parametrize("rows,k,n,small", [
    (1024, 256, 1152, True), (1025, 256, 1153, False), (2304, 1024, 512, True), (2304, 1040, 512, False), (1600, 64, 512, True),
    (4736, 129, 129, True), (4737, 129, 129, False), (4736, 128, 129, False), (6400, 64, 128, False),
])
def test_products_on_either_side_of_the_rule(mlel, rows, k, n, small):
    """Up to half as many tiles of 128 x 128 as SMs (148), with more than one channel tile and at most eight K blocks."""
    import torch
    from mlel_b200.runtime import GraphRunner
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are for 148 SMs")
    r = np.random.Generator(np.random.PCG64(rows + n))
    g = GraphBuilder()
    a = g.input(np.int8, (1, rows, k))
    w = g.constant(r.integers(-128, 128, (1, k, n), dtype=np.int8))
    mult = r.integers(1 << 30, (1 << 31) - 1, (n,), dtype=np.int64).astype(np.int32)
    g.output(g.rescale(g.matmul(a, w, -20, 0), mult, np.full((n,), 38, np.int8), 0, 1, np.int8, double_round=True, per_channel=True))
    data = [r.integers(-128, 128, a.shape, dtype=np.int8)]
    before = mlel.lib().mlel_tensor_core_launches(3)
    got = GraphRunner(g).run(data)[0]
    assert mlel.lib().mlel_tensor_core_launches(3) - before == small
    np.testing.assert_array_equal(got, evaluate(g, data)[0])
