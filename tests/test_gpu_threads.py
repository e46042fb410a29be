"""Sessions of several host threads, each on a stream of its own, dispatched at the same time: enqueued (every thread keeps
its own encoded tensor maps) and replayed.  Bit-exact against the CPU oracle."""
import threading

import numpy as np
import pytest

from mlel_b200.model_graphs import bert_graph, matmul_rescale_graph, resnet50_graph
from tests.graph_eval import evaluate

pytestmark = pytest.mark.gpu


def test_sessions_of_several_threads(mlel):
    import torch
    from mlel_b200.runtime import GraphRunner
    graphs = [resnet50_graph(seed=1, n=2, image=64, width=16, blocks=(1, 1, 1, 1), classes=40),
              bert_graph(seed=2, n=2, seq=48, hidden=64, heads=2, ffn=128, layers=2),
              matmul_rescale_graph(seed=3, n=2, h=300, c=256, w=272)]
    graphs.append(graphs[0])  # the same graph, a session of its own
    failures = []

    def work(graph, inputs, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                runner = GraphRunner(graph)
                for k in range(40):
                    runner.set_inputs(inputs)
                    runner.outputs[0].zero_()
                    runner.dispatch(use_cuda_graph=k % 2 == 1)
                    torch.cuda.current_stream().synchronize()
                    got = runner.outputs[0].cpu().numpy().view(want.dtype).reshape(want.shape)
                    if not np.array_equal(got, want):
                        failures.append((graph.name, k))
        except Exception as error:  # a thread's exception would be lost
            failures.append((graph.name, repr(error)))

    threads = [threading.Thread(target=work, args=(g, i, evaluate(g, i)[0])) for g, i in graphs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
