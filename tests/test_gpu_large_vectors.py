"""GPU parity of the forms that the vectorised kernels take for large tensors only (vector_ops.cu): RESCALE by blocks of 512
elements a warp (from 606 208 elements) with its one-multiply-add forms, TABLE with a copy of the table per lane (from 2^23
elements), four groups in flight a thread (from 7.3 M int32 or 29 M int8 elements).  Bit-exact against the CPU oracle."""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.test_gpu_vector_ops import check, full_range, rng

pytestmark = pytest.mark.gpu

BLOCKS = 512 * 148 * 8  # elements from which RESCALE goes by blocks


def rescale_outputs(r, in_dtype, out_dtype, shape, out_zps, shifts, in_zp=0):
    """Every shift with and without double rounding, multipliers of both signs (double rounding: of both forms)."""
    g = GraphBuilder()
    x = g.input(in_dtype, shape)
    for out_zp in out_zps:
        for shift in shifts:
            for mult in (1 << 30, (1 << 31) - 1, int(r.integers(1 << 30, 1 << 31)), -int(r.integers(1 << 30, 1 << 31))):
                g.output(g.rescale(x, [mult], [shift], in_zp, out_zp, out_dtype, double_round=False))
            g.output(g.rescale(x, [(1 << 31) - 1], [shift], in_zp, out_zp, out_dtype, double_round=True))
            g.output(g.rescale(x, [-(1 << 30)], [shift], in_zp, out_zp, out_dtype, double_round=True))
    return g


@pytest.mark.parametrize("in_dtype,out_dtype,out_zps", [
    (np.int32, np.int16, (-32768, 32767, 3)), (np.int32, np.int32, (100000, -(1 << 31), (1 << 31) - 1)),
    (np.int32, np.int8, (-128, 127)), (np.int16, np.int16, (-32768,)), (np.int8, np.int32, (-100000,)), (np.int16, np.int8, (5,)),
])
@pytest.mark.parametrize("shifts", [(31, 32, 45), (46, 47, 48), (49, 50, 51)])
def test_rescale_by_blocks(mlel, in_dtype, out_dtype, out_zps, shifts):
    """Zero points times 2^shift that do not fit 64 bits beside the product; the shifts where the multiply-add forms (32 to
    50) begin and end; a last block, last groups of four and last elements."""
    r = rng(shifts[0])
    shape = (BLOCKS + 512 + 4 * 31 + 3,)
    in_zp = 0 if in_dtype == np.int32 else int(np.iinfo(in_dtype).min)
    check(rescale_outputs(r, in_dtype, out_dtype, shape, out_zps, shifts, in_zp), [full_range(r, in_dtype, shape)])


@pytest.mark.parametrize("elements", [BLOCKS - 1, BLOCKS, BLOCKS + 1])
def test_rescale_where_blocks_begin(mlel, elements):
    r = rng(elements & 7)
    g = rescale_outputs(r, np.int32, np.int16, (elements,), (-32768,), (48,))
    check(g, [full_range(r, np.int32, (elements,))])


@pytest.mark.parametrize("channels", [4, 7, 513])
def test_rescale_by_blocks_per_channel(mlel, channels):
    """Groups of four that cross the end of a channel row, shifts on both sides of 32."""
    r = rng(channels)
    shape = (BLOCKS // channels + 3, channels)
    g = GraphBuilder()
    x = g.input(np.int32, shape)
    mult = r.integers(1 << 30, 1 << 31, (channels,), dtype=np.int64).astype(np.int32)
    mult[::3] = -mult[::3]
    shift = r.integers(28, 52, (channels,), dtype=np.int8)
    for out_dtype, out_zp in ((np.int8, 5), (np.int16, -32768), (np.int32, 100000)):
        for double_round in (False, True):
            g.output(g.rescale(x, mult, shift, 0, out_zp, out_dtype, double_round=double_round, per_channel=True))
    check(g, [full_range(r, np.int32, shape)])


GROUPS = 4 * 148 * 16 * 256 + 1000  # groups of which every thread takes four at a time, some a fifth by itself


def test_int8_beyond_four_groups_a_thread(mlel):
    """CLAMP and TABLE: the unrolled part, the rest and the last elements."""
    r = rng(1)
    shape = (16 * GROUPS + 13,)
    g = GraphBuilder()
    x = g.input(np.int8, shape)
    g.output(g.clamp(x, -100, 93))
    g.output(g.table(x, full_range(r, np.int8, (256,))))
    check(g, [full_range(r, np.int8, shape)])


@pytest.mark.parametrize("elements", [(1 << 23) - 1, 1 << 23, (1 << 23) + 15, 16 * 4 * 148 * 2 * 1024 + 1])
def test_table_by_lanes(mlel, elements):
    """TABLE's copy per lane begins at 2^23 elements; its threads take four groups at a time from 14.5 M on."""
    r = rng(elements & 7)
    g = GraphBuilder()
    x = g.input(np.int8, (elements,))
    g.output(g.table(x, full_range(r, np.int8, (256,))))
    check(g, [full_range(r, np.int8, (elements,))])


def test_int16_table_beyond_four_groups_a_thread(mlel):
    r = rng(2)
    shape = (4 * GROUPS + 3,)
    g = GraphBuilder()
    x = g.input(np.int16, shape)
    g.output(g.table(x, full_range(r, np.int16, (513,))))
    check(g, [full_range(r, np.int16, shape)])


@pytest.mark.parametrize("length", [196, 197])
def test_int32_beyond_four_groups_a_thread(mlel, length):
    """ADD, SUB and MUL with an operand of the same shape, one value per row (of whole groups or not) and one value."""
    r = rng(length)
    shape = (4 * GROUPS // length + 1, length)
    same, row, one = (full_range(r, np.int32, s) for s in (shape, (shape[0], 1), (1, 1)))
    g = GraphBuilder()
    x, y, rw, v = g.input(np.int32, shape), g.input(np.int32, shape), g.input(np.int32, row.shape), g.input(np.int32, (1, 1))
    g.output(g.add(x, y))
    g.output(g.sub(x, rw))
    g.output(g.mul(x, rw, 17))
    g.output(g.mul(x, v, 31))
    check(g, [full_range(r, np.int32, shape), same, row, one])
