"""GPU parity of products whose RESCALE feeds an int8 TABLE: looked up in the small and the paired kernel's epilogue, applied
in place behind the other kernels (run-time operand, NO_TENSOR_CORE), left alone where the rows are no whole 16 bytes.
Bit-exact against the CPU oracle."""
import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.test_gpu_vector_ops import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,rows,k,n,constant,fused", [
    (1, 5, 64, 144, True, True), (1, 200, 96, 256, True, True), (2, 300, 128, 400, True, True), (1, 1500, 768, 3072, True, True),
    (1, 4000, 70, 272, True, True), (3, 257, 64, 512, False, True), (2, 65, 50, 160, False, True), (1, 64, 64, 128, True, False),
    (1, 64, 64, 150, True, False),
])
@pytest.mark.parametrize("clamp", [False, True])
def test_product_with_table(mlel, batch, rows, k, n, constant, fused, clamp):
    from mlel_b200.runtime import GraphRunner
    r = np.random.Generator(np.random.PCG64(rows + n))
    a8, b8 = (r.integers(-128, 128, s, dtype=np.int8) for s in ((batch, rows, k), (batch, k, n)))
    g = GraphBuilder()
    a = g.input(np.int8, a8.shape)
    b = g.constant(b8) if constant else g.input(np.int8, b8.shape)
    lut = r.integers(-128, 128, (256,), dtype=np.int8)
    for shift in (37, 31):
        y = g.rescale(g.matmul(a, b, 3, 0), [1 << 30 | 12345], [shift], 0, 1, np.int8, double_round=True)
        g.output(g.table(g.clamp(y, -100, 90) if clamp else y, lut))
    names = GraphRunner(g).pipeline.exec_names()
    assert all(x.endswith("+TABLE") for x in names) == fused, names
    check(g, [a8] if constant else [a8, b8])


@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("k,n", [(256, 256), (256, 144), (250, 256), (256, 128)])
def test_product_of_activations_dispatched_by_either_way(mlel, table, k, n):
    """Enqueued (column sums and the paired kernel) or replayed (anything else), by the kernel that takes it: with the paired
    kernel and without, with a TABLE as third launch, with addresses that go to the generic kernel."""
    import torch
    from mlel_b200.runtime import GraphRunner
    from tests.graph_eval import evaluate
    r = np.random.Generator(np.random.PCG64(k + n))
    a8, b8 = (r.integers(-128, 128, s, dtype=np.int8) for s in ((2, 300, k), (2, k, n)))
    g = GraphBuilder()
    a, b = g.input(np.int8, a8.shape), g.input(np.int8, b8.shape)
    y = g.rescale(g.matmul(a, b, 3, 0), [1 << 30 | 12345], [37], 0, 1, np.int8, double_round=True)
    g.output(g.table(y, r.integers(-128, 128, (256,), dtype=np.int8)) if table else y)
    want = evaluate(g, [a8, b8])[0]
    lib = mlel.lib()
    runner = GraphRunner(g)
    buffer = torch.zeros(b8.size + 16, dtype=torch.uint8, device="cuda")
    try:
        for pair in (1, 0, 1):
            assert lib.mlel_set_tuning(b"pair_kernel", pair) == 0
            for use_cuda_graph in (True, False):
                assert np.array_equal(runner.run([a8, b8], use_cuda_graph=use_cuda_graph)[0], want)
    finally:
        assert lib.mlel_set_tuning(b"pair_kernel", 1) == 0
    buffer[1:1 + b8.size] = torch.from_numpy(b8.reshape(-1).view(np.uint8)).cuda()
    runner.session.set_external(*runner._in_keys[1][:2], buffer.data_ptr() + 1)
    assert np.array_equal(runner.run([a8, b8], use_cuda_graph=True)[0], want)


@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("dispatched_before", [False, True])
def test_product_of_activations_inside_a_capture(mlel, table, dispatched_before):
    """A host that captures its stream gets the kernels, whichever way the session dispatches otherwise."""
    import torch
    from mlel_b200.runtime import GraphRunner
    from tests.graph_eval import evaluate
    r = np.random.Generator(np.random.PCG64(5))
    a8, b8 = (r.integers(-128, 128, s, dtype=np.int8) for s in ((2, 300, 256), (2, 256, 256)))
    g = GraphBuilder()
    a, b = g.input(np.int8, a8.shape), g.input(np.int8, b8.shape)
    y = g.rescale(g.matmul(a, b, 3, 0), [1 << 30 | 12345], [37], 0, 1, np.int8, double_round=True)
    g.output(g.table(y, r.integers(-128, 128, (256,), dtype=np.int8)) if table else y)
    runner = GraphRunner(g)
    runner.run([a8, b8])  # uploads the constants
    if dispatched_before:
        runner.dispatch(use_cuda_graph=True)
    torch.cuda.synchronize()
    runner.outputs[0].zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        runner.dispatch(use_cuda_graph=True)
    assert not np.array_equal(runner.get_outputs()[0], evaluate(g, [a8, b8])[0])  # captured, not run
    graph.replay()
    assert np.array_equal(runner.get_outputs()[0], evaluate(g, [a8, b8])[0])
