"""GPU parity of fused contractions whose RESCALE subtracts an int32 zero point of any size: every kernel's one-multiply-add
form folds accumulator, correction and zero point into 32 bits, which only small zero points allow.  Bit-exact against the
CPU oracle; a counter tells which tensor-core kernel took the case."""
import ctypes

import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.test_gpu_vector_ops import check_fused

pytestmark = pytest.mark.gpu

ZERO_POINTS = (256, 257, 1 << 30, (1 << 31) - 1, -(1 << 31), -(1 << 30) - 257)


def rescales(g, r, make, channels, fill):
    """One contraction per zero point and rounding, at a shift that keeps the zero point's share of the result in sight and
    at one where it saturates; results on both sides of the zero point."""
    for zp in ZERO_POINTS:
        for shift in (37, 50):
            for double_round in (False, True):
                mult = r.integers(1 << 30, 1 << 31, (channels,), dtype=np.int64).astype(np.int32)
                g.output(g.rescale(make(np.int32(fill * (zp >> 1))), mult, np.full(channels, shift, np.int8), zp, -3, np.int8,
                                   double_round=double_round, per_channel=True))


def launches(mlel):
    lib = mlel.lib()
    lib.mlel_tensor_core_launches.restype = ctypes.c_longlong
    return [lib.mlel_tensor_core_launches(k) for k in range(5)]


@pytest.mark.parametrize("n,h,w,ic,oc,k,kernel", [
    (4, 56, 56, 64, 64, 1, 0), (4, 56, 56, 64, 256, 1, 1), (1, 7, 7, 64, 128, 1, 3), (6, 40, 41, 32, 48, 3, 4), (1, 45, 61, 3, 32, 3, 4),
])
@pytest.mark.parametrize("fill", [0, 1])
def test_convolutions(mlel, n, h, w, ic, oc, k, kernel, fill):
    """fill: a bias of half the zero point (a large correction with a large zero point) or a small one."""
    r = np.random.Generator(np.random.PCG64(h + oc))
    g = GraphBuilder()
    x = g.input(np.int8, (n, h, w, ic))

    def make(bias):
        weights = g.constant(r.integers(-127, 128, (oc, k, k, ic), dtype=np.int8))
        b = g.constant((r.integers(-3000, 3000, (oc,)) + int(bias)).astype(np.int32))
        return g.conv2d(x, weights, b, [k // 2] * 4, [1, 1], [1, 1], -7, 0)

    rescales(g, r, make, oc, fill)
    before = launches(mlel)
    check_fused(mlel, g, [r.integers(-128, 128, x.shape, dtype=np.int8)], ["CONV2D+RESCALE"])
    assert launches(mlel)[kernel] > before[kernel]


@pytest.mark.parametrize("stride,h,c", [(1, 40, 32), (2, 41, 36), (1, 5, 4)])
@pytest.mark.parametrize("fill", [0, 1])
def test_depthwise(mlel, stride, h, c, fill):
    r = np.random.Generator(np.random.PCG64(h + c))
    g = GraphBuilder()
    x = g.input(np.int8, (2, h, h, c))

    def make(bias):
        weights = g.constant(r.integers(-127, 128, (3, 3, c, 1), dtype=np.int8))
        b = g.constant((r.integers(-3000, 3000, (c,)) + int(bias)).astype(np.int32))
        return g.depthwise_conv2d(x, weights, b, [1] * 4, [stride, stride], [1, 1], -7, 0)

    rescales(g, r, make, c, fill)
    check_fused(mlel, g, [r.integers(-128, 128, x.shape, dtype=np.int8)], ["DEPTHWISE_CONV2D+RESCALE"])


@pytest.mark.parametrize("batch,rows,k,n,constant,kernel", [
    (1, 8000, 96, 64, True, 0), (1, 3000, 96, 384, True, 2), (2, 700, 128, 256, False, 2), (1, 40, 128, 128, True, 3),
])
def test_products(mlel, batch, rows, k, n, constant, kernel):
    r = np.random.Generator(np.random.PCG64(rows + n))
    a8, b8 = (r.integers(-128, 128, s, dtype=np.int8) for s in ((batch, rows, k), (batch, k, n)))
    g = GraphBuilder()
    a = g.input(np.int8, a8.shape)
    b = g.constant(b8) if constant else g.input(np.int8, b8.shape)
    rescales(g, r, lambda bias: g.matmul(a, b, 3, 0), n, 0)
    before = launches(mlel)
    check_fused(mlel, g, [a8] if constant else [a8, b8], ["MATMUL+RESCALE"])
    assert launches(mlel)[kernel] > before[kernel]
