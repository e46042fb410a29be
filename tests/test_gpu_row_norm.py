"""GPU parity of the register-resident residual add + layer norm: rows at and beside its 128-element groups, scales that
the 32-bit forms take (powers of two) and scales that they do not, double rounding and zero points.  Bit-exact against
the CPU oracle, operator by operator."""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.test_gpu_vector_ops import check_fused, full_range, rng

pytestmark = pytest.mark.gpu

NORM = "ROWS(RESCALE+RESCALE+ADD+REDUCE_SUM+MUL+SUB+MUL+REDUCE_SUM+MUL+RESCALE+TABLE+MUL+RESCALE)"


@pytest.mark.parametrize("rows,length", [(1, 4), (3, 128), (37, 132), (5, 508), (2, 768), (9, 772), (3, 1024), (2, 2048), (2, 2052)])
@pytest.mark.parametrize("mult,shift,out_shift,in_zp,double_round", [
    (1 << 30, 24, 45, 0, True),            # 32-bit forms
    (3 << 28, 26, 44, -7, False),
    ((1 << 30) + 12345, 25, 46, 5, True),  # 64-bit forms
    (1 << 30, 33, 40, 0, True),            # double rounding on the inputs: 64-bit forms
])
def test_residual_layer_norm(mlel, rows, length, mult, shift, out_shift, in_zp, double_round):
    r = rng(length + shift)
    g = GraphBuilder()
    a, b = g.input(np.int8, (1, rows, length)), g.input(np.int8, (1, rows, length))
    t = g.add(g.rescale(a, [mult], [shift], in_zp, 0, np.int32, double_round=shift > 31),
              g.rescale(b, [1 << 30], [24], 0, 3, np.int32))
    inv = g.inline(np.asarray([(1 << 20) // length], np.int32).reshape(1, 1, 1))
    cen = g.sub(t, g.mul(g.reduce("REDUCE_SUM", t, 2), inv, 20))
    var = g.mul(g.reduce("REDUCE_SUM", g.mul(cen, cen, 8), 2), inv, 20)
    var16 = g.rescale(var, [1 << 30], [34], 0, -32768, np.int16)
    x = (np.arange(513, dtype=np.float64) - 256.0) * 128.0
    rsqrt = np.clip(np.round(32767.0 * 16.0 / np.sqrt(x + 32768.0 + 256.0)), 0, 32767).astype(np.int16)
    g.output(g.rescale(g.mul(cen, g.table(var16, rsqrt), 12), [mult], [out_shift], 0, -3, np.int8, double_round=double_round))
    check_fused(mlel, g, [full_range(r, np.int8, a.shape), full_range(r, np.int8, b.shape)], [NORM])


@pytest.mark.parametrize("tensor", ["first", "second", "result"])
@pytest.mark.parametrize("offset", [4, 8])
def test_tensors_off_16_byte_boundaries_are_refused(mlel, tensor, offset):
    """As by the row machine: both kernels load and store words.  Nothing is launched."""
    import torch
    from mlel_b200.runtime import GraphRunner
    from tests.test_gpu_vector_ops import _norm_chain
    shape = (1, 3, 128)
    g = GraphBuilder()
    a, b = g.input(np.int8, shape), g.input(np.int8, shape)
    t = g.add(g.rescale(a, [1 << 30], [24], 0, 0, np.int32), g.rescale(b, [1 << 30], [24], 0, 0, np.int32))
    g.output(_norm_chain(g, rng(1), t, shape[-1])[0])
    runner = GraphRunner(g)
    assert runner.pipeline.exec_names() == [NORM]
    set_, binding = {"first": runner._in_keys[0], "second": runner._in_keys[1], "result": runner._out_keys[0]}[tensor][:2]
    buffer = torch.zeros(3 * 128 + 16, dtype=torch.uint8, device="cuda")
    runner.session.set_external(set_, binding, buffer.data_ptr() + offset)
    for use_cuda_graph in (False, True):
        with pytest.raises(mlel.MlelError, match="not 16-byte aligned"):
            runner.dispatch(use_cuda_graph=use_cuda_graph)
    runner.session.set_external(set_, binding, buffer.data_ptr())  # a boundary is accepted again
    runner.dispatch()
    torch.cuda.synchronize()


@pytest.mark.parametrize("in_zp", [-(1 << 31), (1 << 31) - 1, -(1 << 30), 1 << 24, 256])
@pytest.mark.parametrize("mult,shift", [((1 << 31) - 1, 31), (1 << 30, 45)])
def test_result_scale_with_any_zero_point(mlel, in_zp, mult, shift):
    """The last RESCALE reads int32: bounds of the 32-bit form with zero points whose product leaves 64 bits."""
    from tests.test_gpu_vector_ops import _lut16
    r = rng(shift)
    shape = (1, 9, 132)
    g = GraphBuilder()
    a, b = g.input(np.int8, shape), g.input(np.int8, shape)
    t = g.add(g.rescale(a, [1 << 30], [24], 0, 0, np.int32), g.rescale(b, [1 << 30], [24], 0, 0, np.int32))
    inv = g.inline(np.asarray([(1 << 20) // shape[-1]], np.int32).reshape(1, 1, 1))
    cen = g.sub(t, g.mul(g.reduce("REDUCE_SUM", t, 2), inv, 20))
    var = g.mul(g.reduce("REDUCE_SUM", g.mul(cen, cen, 8), 2), inv, 20)
    factor = g.table(g.rescale(var, [1 << 30], [34], 0, -32768, np.int16), _lut16(r))
    g.output(g.rescale(g.mul(cen, factor, 12), [mult], [shift], in_zp, 3, np.int8))
    check_fused(mlel, g, [full_range(r, np.int8, shape), full_range(r, np.int8, shape)], [NORM])


@pytest.mark.parametrize("length", [4, 124, 768, 1028])
@pytest.mark.parametrize("up,norm_shift,out_shift,in_zp,out_zp,double_round,table", [
    ((24, 24), 12, 45, 0, 0, True, "any"),       # both products of the last step in one, table values of either sign and zero
    ((26, 21), 12, 42, -5, 100, True, "small"),  # factors below the MUL's rounding term; shifts that add up to 24
    ((24, 22), 9, 53, 3, -128, True, "any"),     # ... to 32
    ((24, 24), 9, 54, 0, 0, True, "any"),        # ... to 33: not in this form
    ((25, 24), 12, 31, 0, 7, False, "any"),      # no double rounding, a small shift: not in this form
    ((24, 24), 12, 46, 0, 0, False, "small"),
])
def test_whole_input_scales_and_a_power_of_two_on_the_result(mlel, length, up, norm_shift, out_shift, in_zp, out_zp, double_round, table):
    r = rng(length + out_shift)
    shape = (1, 11, length)
    g = GraphBuilder()
    a, b = g.input(np.int8, shape), g.input(np.int8, shape)
    t = g.add(g.rescale(a, [3 << 28], [up[0]], in_zp, 0, np.int32), g.rescale(b, [1 << 30], [up[1]], 0, 2, np.int32))
    inv = g.inline(np.asarray([(1 << 20) // length], np.int32).reshape(1, 1, 1))
    cen = g.sub(t, g.mul(g.reduce("REDUCE_SUM", t, 2), inv, 20))
    var = g.mul(g.reduce("REDUCE_SUM", g.mul(cen, cen, 8), 2), inv, 20)
    bound = 32768 if table == "any" else 8
    lut = r.integers(-bound, bound, (513,)).astype(np.int16)
    y = g.mul(cen, g.table(g.rescale(var, [1 << 30], [34], 0, -32768, np.int16), lut), norm_shift)
    g.output(g.rescale(y, [1 << 30], [out_shift], 0, out_zp, np.int8, double_round=double_round))
    check_fused(mlel, g, [full_range(r, np.int8, shape), full_range(r, np.int8, shape)], [NORM])


@pytest.mark.parametrize("length", [64, 132])
def test_layer_norm_with_gain_and_bias(mlel, length):
    """Per-channel gain and bias behind the normalisation: not the register kernel's program, the operators' results."""
    from mlel_b200.runtime import GraphRunner
    from tests.graph_eval import evaluate
    from tests.test_gpu_vector_ops import _lut16
    r = rng(length)
    shape = (1, 19, length)
    g = GraphBuilder()
    a, b = g.input(np.int8, shape), g.input(np.int8, shape)
    t = g.add(g.rescale(a, [1 << 30], [24], 0, 0, np.int32), g.rescale(b, [1 << 30], [24], 0, 0, np.int32))
    inv = g.inline(np.asarray([(1 << 20) // length], np.int32).reshape(1, 1, 1))
    cen = g.sub(t, g.mul(g.reduce("REDUCE_SUM", t, 2), inv, 20))
    var = g.mul(g.reduce("REDUCE_SUM", g.mul(cen, cen, 8), 2), inv, 20)
    y = g.mul(cen, g.table(g.rescale(var, [1 << 30], [34], 0, -32768, np.int16), _lut16(r)), 12)
    gain, bias = (g.constant(r.integers(lo, hi, (1, 1, length)).astype(np.int32)) for lo, hi in ((200, 300), (-99, 99)))
    g.output(g.rescale(g.add(g.mul(y, gain, 8), bias), [1 << 30], [45], 0, 3, np.int8, double_round=True))
    data = [full_range(r, np.int8, shape), full_range(r, np.int8, shape)]
    runner = GraphRunner(g)
    assert NORM not in runner.pipeline.exec_names()
    for use_cuda_graph in (False, True):
        np.testing.assert_array_equal(runner.run(data, use_cuda_graph=use_cuda_graph)[0], evaluate(g, data)[0])
