"""GPU parity of the window kernel: both tile shapes, image sizes at and beside their edges, every pixel width (32, 64 and
128 bytes, whole and padded), one to several channel tiles, windows of other sizes and dilations, border classes, shifts
on both sides of 32, widths that are no multiple of 16.  Bit-exact against the CPU oracle; a counter tells that the kernel took the case."""
import ctypes

import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate
from tests.test_gpu_small import conv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,ic,oc,k,pad,dil,shift", [
    (2, 56, 56, 64, 64, 3, 1, 1, 37), (1, 16, 8, 128, 128, 3, 1, 1, 38), (3, 28, 28, 128, 128, 3, 1, 1, 38), (1, 45, 131, 96, 32, 3, 1, 1, 37),
    (1, 17, 9, 64, 64, 3, 1, 1, 37), (2, 40, 130, 32, 48, 3, 0, 1, 35), (1, 33, 257, 16, 16, 3, 1, 1, 34), (2, 23, 61, 48, 160, 3, 1, 1, 37),
    (1, 64, 70, 80, 96, 3, 1, 2, 37), (1, 30, 41, 32, 32, 5, 2, 1, 36), (2, 20, 120, 112, 16, 2, 0, 1, 30), (1, 50, 50, 16, 64, 7, 3, 1, 36),
    (5, 14, 14, 64, 256, 3, 1, 1, 29), (1, 3, 400, 32, 64, 3, 1, 1, 36), (1, 300, 2, 64, 16, 3, 1, 1, 36),
    (2, 56, 56, 64, 63, 3, 1, 1, 37), (1, 45, 131, 96, 21, 3, 1, 1, 37), (3, 28, 28, 128, 129, 3, 1, 1, 38), (1, 33, 70, 32, 5, 3, 1, 1, 31),
    (2, 23, 61, 48, 150, 3, 0, 1, 37),
])
def test_windows(mlel, n, h, w, ic, oc, k, pad, dil, shift):
    from mlel_b200.runtime import GraphRunner
    r = np.random.Generator(np.random.PCG64(h * 1000 + w))
    g = GraphBuilder()
    x = g.input(np.int8, (n, h, w, ic))
    g.output(conv(g, r, x, oc, k, 1, pad, -7, False, shift, dil))
    g.output(conv(g, r, x, oc, k, 1, pad, 5, True, shift, dil))
    data = r.integers(-128, 128, x.shape, dtype=np.int8)
    want = evaluate(g, [data])
    lib = mlel.lib()
    lib.mlel_tensor_core_launches.restype = ctypes.c_longlong
    try:
        assert lib.mlel_set_tuning(b"small_kernel", 0) == 0
        before = lib.mlel_tensor_core_launches(4)
        runner = GraphRunner(g)
        for use_cuda_graph in (False, True):
            for a, b in zip(runner.run([data], use_cuda_graph=use_cuda_graph), want):
                bad = np.argwhere(a != b)
                assert len(bad) == 0, (len(bad), a.size, bad[0].tolist(), bad[-1].tolist())
        assert lib.mlel_tensor_core_launches(4) > before
    finally:
        assert lib.mlel_set_tuning(b"small_kernel", 1) == 0


@pytest.mark.parametrize("n,h,w,ic,oc,k,stride,pad,shift", [
    (2, 56, 56, 3, 64, 7, 2, 3, 36), (1, 45, 131, 3, 32, 3, 1, 1, 33), (3, 33, 47, 3, 32, 3, 2, 1, 33), (1, 16, 8, 4, 16, 3, 1, 0, 33),
    (1, 20, 120, 1, 48, 5, 1, 2, 31), (2, 21, 257, 2, 16, 3, 2, 0, 32), (1, 40, 40, 3, 160, 7, 1, 3, 36), (1, 9, 300, 3, 64, 5, 2, 2, 29),
    (1, 5, 5, 4, 32, 2, 2, 0, 31), (2, 7, 7, 3, 16, 1, 2, 0, 30), (1, 70, 3, 3, 64, 3, 2, 2, 33),
    (2, 40, 50, 3, 37, 3, 1, 1, 33), (1, 56, 57, 3, 65, 7, 2, 3, 36), (3, 20, 21, 2, 1, 3, 2, 1, 31),
])
def test_windows_of_few_channels(mlel, n, h, w, ic, oc, k, stride, pad, shift):
    from mlel_b200.runtime import GraphRunner
    r = np.random.Generator(np.random.PCG64(h * 1000 + w))
    g = GraphBuilder()
    x = g.input(np.int8, (n, h, w, ic))
    g.output(conv(g, r, x, oc, k, stride, pad, -7, False, shift))
    g.output(conv(g, r, x, oc, k, stride, pad, 5, True, shift))
    data = r.integers(-128, 128, x.shape, dtype=np.int8)
    want = evaluate(g, [data])
    lib = mlel.lib()
    lib.mlel_tensor_core_launches.restype = ctypes.c_longlong
    before = lib.mlel_tensor_core_launches(4)
    runner = GraphRunner(g)
    for use_cuda_graph in (False, True):
        for a, b in zip(runner.run([data], use_cuda_graph=use_cuda_graph), want):
            bad = np.argwhere(a != b)
            assert len(bad) == 0, (len(bad), a.size, bad[0].tolist(), bad[-1].tolist())
    assert lib.mlel_tensor_core_launches(4) > before


@pytest.mark.parametrize("n,h,w,ic,oc,k,expected", [
    (1, 64, 74, 64, 64, 3, 3), (1, 64, 75, 64, 64, 3, 4),      # 37 and 38 tiles of 128 pixels
    (3, 28, 28, 16, 129, 3, 4), (2, 56, 56, 32, 32, 5, 4),     # channel tiles count; another window
    (1, 70, 90, 48, 63, 3, 4), (1, 56, 108, 64, 64, 2, 3),     # rows at any address; too few taps
    (1, 64, 75, 80, 64, 3, 3), (1, 64, 75, 144, 64, 3, 3),     # more channels than the rule takes, than a pixel row holds
    (1, 64, 75, 64, 64, 31, 3),                                # weights that do not fit beside the input
])
def test_window_kernel_before_the_small_one(mlel, n, h, w, ic, oc, k, expected):
    """From a quarter of the SMs on (148: 37 tiles), below half of which the small kernel would take them too."""
    from mlel_b200.runtime import GraphRunner
    r = np.random.Generator(np.random.PCG64(h * 1000 + w))
    g = GraphBuilder()
    x = g.input(np.int8, (n, h, w, ic))
    g.output(conv(g, r, x, oc, k, 1, k // 2, -7, True, 38))
    data = r.integers(-128, 128, x.shape, dtype=np.int8)
    want = evaluate(g, [data])[0]
    lib = mlel.lib()
    lib.mlel_tensor_core_launches.restype = ctypes.c_longlong
    runner = GraphRunner(g)
    before = [lib.mlel_tensor_core_launches(kernel) for kernel in range(5)]
    got = runner.run([data])[0]
    assert [lib.mlel_tensor_core_launches(kernel) - before[kernel] for kernel in range(5)] == [int(kernel == expected) for kernel in range(5)]
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n,h,w,ic,oc", [
    (5, 70, 110, 16, 64), (5, 70, 110, 32, 64), (5, 70, 110, 48, 64), (3, 75, 129, 64, 128),  # several tiles of 64 channels to a CTA
    (1, 135, 240, 64, 64), (12, 56, 56, 64, 64),                                             # 1.7 and 2 tiles to a CTA
    (3, 70, 110, 80, 64), (1, 70, 110, 64, 64), (3, 70, 110, 64, 63),                        # more channels, one tile, rows at any address
])
def test_both_forms_of_issue(mlel, n, h, w, ic, oc):
    from mlel_b200.runtime import GraphRunner
    r = np.random.Generator(np.random.PCG64(ic + oc))
    g = GraphBuilder()
    x = g.input(np.int8, (n, h, w, ic))
    g.output(conv(g, r, x, oc, 3, 1, 1, -7, True, 37))
    data = r.integers(-128, 128, x.shape, dtype=np.int8)
    lib = mlel.lib()
    lib.mlel_tensor_core_launches.restype = ctypes.c_longlong
    runner = GraphRunner(g)
    before = lib.mlel_tensor_core_launches(4)
    np.testing.assert_array_equal(runner.run([data])[0], evaluate(g, [data])[0])
    assert lib.mlel_tensor_core_launches(4) == before + 1
