"""GPU parity of narrow outputs whose rows are whole words, or not, with a residual tail: the shortcut at any address, tiles that
end inside.  Bit-exact against the CPU oracle."""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate
from tests.test_gpu_small import conv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("oc", [4, 20, 24, 60, 21, 63, 100])
@pytest.mark.parametrize("ic,k", [(64, 1), (32, 3), (144, 1)])
@pytest.mark.parametrize("tail", [True, False])
def test_rows_of_words_and_of_bytes(mlel, oc, ic, k, tail):
    import torch
    from mlel_b200.runtime import GraphRunner
    r = np.random.Generator(np.random.PCG64(oc + ic))
    g = GraphBuilder()
    n, hw = 7, 75  # 308 tiles of 128 pixels and a rest: two or three rounds on every SM
    inputs = [g.input(np.int8, (n, hw, hw, c)) for c in ((ic, oc) if tail else (ic,))]
    x = inputs[0]
    y = conv(g, r, x, oc, k, 1, k // 2, 4, True)
    if tail:
        a = g.rescale(y, [int(r.integers(1 << 30, 1 << 31))], [23], 4, 0, np.int32)
        b = g.rescale(inputs[1], [int(r.integers(1 << 30, 1 << 31))], [23], -3, 0, np.int32)
        y = g.rescale(g.add(a, b), [int(r.integers(1 << 30, 1 << 31))], [40], 0, -20, np.int8, double_round=True)
    g.output(y)
    data = [r.integers(-128, 128, v.shape, dtype=np.int8) for v in inputs]
    want = evaluate(g, data)[0]
    runner = GraphRunner(g)
    runner.set_inputs(data)
    short = data[-1].reshape(-1).view(np.uint8)
    buffer = torch.zeros(short.size + 16, dtype=torch.uint8, device="cuda")
    for offset in (0, 4, 1) if tail else (0,):
        if tail:
            buffer[offset:offset + short.size] = torch.from_numpy(short).cuda()
            runner.session.set_external(*runner._in_keys[1][:2], buffer.data_ptr() + offset)
        runner.outputs[0].zero_()
        runner.dispatch()
        assert np.array_equal(runner.get_outputs()[0], want), offset
