"""GPU parity of residual tails whose shortcut is an application tensor at any byte address: convolutions that the channel-
major, the pixel-major, the small and the paired kernel take, and the add on its own.  Bit-exact against the CPU oracle."""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate
from tests.test_gpu_small import conv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,hw,ic,oc,k", [(4, 56, 64, 256, 1), (4, 56, 64, 64, 1), (4, 40, 32, 48, 3), (1, 7, 64, 128, 1), (2, 30, 20, 32, 3)])
@pytest.mark.parametrize("pair", [1, 2])
def test_shortcut_at_any_address(mlel, n, hw, ic, oc, k, pair):
    import torch
    from mlel_b200.runtime import GraphRunner
    r = np.random.Generator(np.random.PCG64(hw + oc))
    g = GraphBuilder()
    x, short = g.input(np.int8, (n, hw, hw, ic)), g.input(np.int8, (n, hw, hw, oc))
    y = conv(g, r, x, oc, k, 1, k // 2, 4, True)
    a = g.rescale(y, [int(r.integers(1 << 30, 1 << 31))], [23], 4, 0, np.int32)
    b = g.rescale(short, [int(r.integers(1 << 30, 1 << 31))], [23], -3, 0, np.int32)
    g.output(g.rescale(g.add(a, b), [int(r.integers(1 << 30, 1 << 31))], [40], 0, -20, np.int8, double_round=True))
    data = [r.integers(-128, 128, v.shape, dtype=np.int8) for v in (x, short)]
    want = evaluate(g, data)[0]
    lib = mlel.lib()
    try:
        assert lib.mlel_set_tuning(b"pair_kernel", pair) == 0
        runner = GraphRunner(g)
        assert runner.session.launch_count() == 1 and "ADD+RESCALE" in runner.pipeline.exec_names()[0]
        runner.set_inputs(data)
        buffer = torch.zeros(data[1].size + 16, dtype=torch.uint8, device="cuda")
        for offset in (0, 8, 4, 1):
            buffer[offset:offset + data[1].size] = torch.from_numpy(data[1].reshape(-1).view(np.uint8)).cuda()
            runner.session.set_external(*runner._in_keys[1][:2], buffer.data_ptr() + offset)
            for use_cuda_graph in (False, True):
                runner.outputs[0].zero_()
                runner.dispatch(use_cuda_graph=use_cuda_graph)
                assert np.array_equal(runner.get_outputs()[0], want), offset
    finally:
        assert lib.mlel_set_tuning(b"pair_kernel", 1) == 0
