"""GPU parity of the 3x3 depthwise convolution from a table of channel constants: channel counts beside multiples of four,
images at and beside a thread's 4 x 4 and 4 x 2 outputs, strides and padding, shifts at the ends of what the table takes,
bounds at and off the ends of int8, operands at any address; and parameters that no table describes.  Bit-exact against the CPU
oracle."""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate

pytestmark = pytest.mark.gpu


def graph(r, shape, stride=1, pad=1, in_zp=-3, out_zp=5, shift=(37, 40), double_round=True, per_channel=True, clamp=None,
          rescale_zp=0, low_mult=1 << 30, one_bias=False):
    g = GraphBuilder()
    c = shape[3]
    x = g.input(np.int8, shape)
    w = g.constant(r.integers(-128, 128, (3, 3, c, 1), dtype=np.int8))
    b = g.constant(r.integers(-(1 << 14), 1 << 14, (1 if one_bias else c,), dtype=np.int32))
    y = g.depthwise_conv2d(x, w, b, [pad] * 4, [stride] * 2, [1, 1], in_zp, 0)
    n = c if per_channel else 1
    mult = r.integers(low_mult, (1 << 31) - 1, (n,), dtype=np.int64).astype(np.int32)
    y = g.rescale(y, mult, r.integers(shift[0], shift[1] + 1, (n,), dtype=np.int8), rescale_zp, out_zp, np.int8,
                  double_round=double_round, per_channel=per_channel)
    g.output(g.clamp(y, *clamp) if clamp else y)
    return g


def check(g, r, offsets=((0, 0),)):
    import torch
    from mlel_b200.runtime import GraphRunner
    data = r.integers(-128, 128, g.inputs[0].shape, dtype=np.int8)
    want = evaluate(g, [data])[0]
    runner = GraphRunner(g)
    assert runner.session.launch_count() == 1
    source = torch.zeros(data.size + 4, dtype=torch.uint8, device="cuda")
    result = torch.zeros(want.size + 8, dtype=torch.uint8, device="cuda")
    for a, b in offsets:
        source[a:a + data.size] = torch.from_numpy(data.reshape(-1).view(np.uint8)).cuda()
        result.fill_(0x55)
        runner.session.set_external(*runner._in_keys[0][:2], source.data_ptr() + a)
        runner.session.set_external(*runner._out_keys[0][:2], result.data_ptr() + 4 + b)
        runner.dispatch()
        torch.cuda.synchronize()
        got = result.cpu().numpy()
        np.testing.assert_array_equal(got[4 + b:4 + b + want.size].view(np.int8).reshape(want.shape), want)
        assert (got[:4 + b] == 0x55).all() and (got[4 + b + want.size:] == 0x55).all()


@pytest.mark.parametrize("c", [1, 2, 3, 4, 5, 18, 63, 64])
@pytest.mark.parametrize("hw,stride,pad", [((1, 1), 1, 1), ((5, 4), 1, 0), ((9, 13), 2, 1), ((8, 7), 2, 0), ((16, 16), 1, 1)])
def test_channels_and_sizes(mlel, c, hw, stride, pad):
    r = np.random.Generator(np.random.PCG64(c * 100 + hw[1]))
    check(graph(r, (2, *hw, c), stride, pad), r)


@pytest.mark.parametrize("c,stride", [(36, 1), (35, 1), (64, 2), (66, 2)])
def test_images_that_fill_the_gpu(mlel, c, stride):
    r = np.random.Generator(np.random.PCG64(c))
    check(graph(r, (16, 100, 99, c), stride, clamp=(5, 127)), r)


@pytest.mark.parametrize("offsets", [(1, 0), (0, 1), (2, 2), (3, 1)])
@pytest.mark.parametrize("c", [16, 17])
def test_any_address(mlel, c, offsets):
    r = np.random.Generator(np.random.PCG64(sum(offsets)))
    check(graph(r, (1, 6, 7, c)), r, [(0, 0), offsets])


@pytest.mark.parametrize("kw", [
    dict(shift=(33, 33)), dict(shift=(50, 50)),                      # the table's ends where the sign counts
    dict(shift=(32, 32), double_round=False), dict(shift=(32, 32), clamp=(5, 127)),  # and where it does not
    dict(shift=(32, 32)), dict(shift=(28, 31)), dict(shift=(51, 60)),  # beyond
    dict(low_mult=1), dict(per_channel=False, one_bias=True), dict(rescale_zp=(1 << 30) + 5), dict(rescale_zp=-77),
    dict(clamp=(-50, 60)), dict(clamp=(-128, 60)), dict(clamp=(-50, 127)), dict(clamp=(5, 100), double_round=False),
    dict(in_zp=-128, out_zp=127), dict(in_zp=127, out_zp=-128),
])
@pytest.mark.parametrize("c", [20, 21])
def test_parameters(mlel, c, kw):
    r = np.random.Generator(np.random.PCG64(c))
    check(graph(r, (2, 9, 10, c), **kw), r)
