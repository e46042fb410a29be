"""GPU parity of projections that run as one product in front of a fused attention node: all three of one activation, two of
three, per-tensor and per-channel scales, contraction lengths with and without a copy in front, an application tensor at an odd
address, and the forms that stay separate.  Bit-exact against the CPU oracle."""
import math

import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate

pytestmark = pytest.mark.gpu


def projected_attention(n, heads, sq, sk, d, width, sources, seed, scales="channel", zps=(3, 3, 3), extra=None):
    """Q, K and V as products of the inputs `sources` names; `extra`: "output" makes K a graph output besides, "clamp" gives V
    another upper bound."""
    rng = np.random.Generator(np.random.PCG64(seed))
    x = (np.arange(513, dtype=np.float64) - 256.0) * 128.0
    exp_lut = np.round(32767.0 * np.exp(np.minimum(x, 0.0) / 4096.0)).astype(np.int16)
    recip_lut = np.clip(np.round(32767.0 * 256.0 / (x + 32768.0 + 256.0)), 0, 32767).astype(np.int16)
    g = GraphBuilder("projections")
    rows = {s: n * t for s, t in zip(sources, (sq, sk, sk))}
    xs = {s: g.input(np.int8, (1, rows[s], width)) for s in sorted(rows)}
    data = [rng.integers(-128, 128, (1, rows[s], width), dtype=np.int8) for s in sorted(rows)]
    hidden = heads * d

    def project(k):
        w = g.constant(rng.integers(-128, 128, (1, width, hidden), dtype=np.int8))
        y = g.matmul(xs[sources[k]], w, zps[k], 0)
        shift = 36 + int(math.log2(width) / 2)
        if scales == "channel":
            mult = rng.integers(1 << 30, (1 << 31) - 1, (hidden,), dtype=np.int64).astype(np.int32)
            y = g.rescale(y, mult, rng.integers(shift, shift + 2, (hidden,), dtype=np.int8), 0, 0, np.int8, double_round=True,
                          per_channel=True)
        else:
            y = g.rescale(y, [int(rng.integers(1 << 30, 1 << 31))], [shift + k % 2], 0, 0, np.int8, double_round=True)
        y = g.clamp(y, -128, 100) if extra == "clamp" and k == 2 else y
        if extra == "output" and k == 1:
            g.output(y)
        return g.reshape(y, (n, sq if k == 0 else sk, heads, d))

    q, k, v = (project(i) for i in range(3))
    q = g.reshape(g.transpose(q, (0, 2, 1, 3)), (n * heads, sq, d))
    k = g.reshape(g.transpose(k, (0, 2, 3, 1)), (n * heads, d, sk))
    v = g.reshape(g.transpose(v, (0, 2, 1, 3)), (n * heads, sk, d))
    s = g.matmul(q, k, 0, 0)
    diff = g.sub(s, g.reduce("REDUCE_MAX", s, 2))
    e = g.table(g.rescale(diff, [1 << 30], [30 + max(2, int(math.log2(d)) - 2)], 0, 0, np.int16), exp_lut)
    log_keys = max(1, math.ceil(math.log2(sk)))
    r = g.table(g.rescale(g.reduce("REDUCE_SUM", e, 2), [1 << 30], [37 + log_keys], 0, -32768, np.int16), recip_lut)
    p = g.rescale(g.mul(e, r, 22), [1 << 30], [37 + log_keys], 0, -128, np.int8)
    c = g.rescale(g.matmul(p, v, -128, 0), [int(rng.integers(1 << 30, 1 << 31))], [38], 0, 3, np.int8, double_round=True)
    g.output(g.clamp(g.transpose(g.reshape(c, (n, heads, sq, d)), (0, 2, 1, 3)), -127, 126))
    return g, data


@pytest.mark.parametrize("products,n,heads,sq,sk,d,width,sources,form", [
    (1, 2, 4, 33, 33, 32, 128, "aaa", {}), (1, 1, 12, 197, 197, 64, 768, "aaa", {}), (1, 3, 1, 40, 40, 64, 64, "aaa", {}),
    (1, 1, 2, 130, 130, 96, 200, "aaa", {}), (1, 8, 4, 384, 384, 64, 256, "aaa", {}), (1, 1, 2, 7, 7, 32, 49, "aaa", {}),
    (1, 2, 3, 65, 65, 64, 192, "aaa", {"scales": "tensor"}), (2, 2, 4, 50, 77, 32, 128, "abb", {}),
    (2, 2, 4, 64, 64, 32, 128, "aab", {}), (2, 2, 4, 64, 64, 32, 128, "aba", {}), (3, 1, 2, 64, 64, 32, 64, "abc", {}),
    (2, 2, 2, 64, 64, 64, 128, "aaa", {"zps": (3, 3, -3)}), (2, 2, 2, 64, 64, 64, 128, "aaa", {"extra": "clamp"}),
    (2, 2, 2, 64, 64, 64, 128, "aaa", {"extra": "output"}),
])
def test_projections_as_one_product(mlel, products, n, heads, sq, sk, d, width, sources, form):
    import torch
    from mlel_b200.runtime import GraphRunner
    g, data = projected_attention(n, heads, sq, sk, d, width, sources, seed=sk + width, **form)
    runner = GraphRunner(g)
    names = runner.pipeline.exec_names()
    assert sum(name.startswith("MATMUL+RESCALE") for name in names) == products and sum("ATTENTION" in name for name in names) == 1, names
    want = evaluate(g, data)
    assert np.unique(want[-1]).size > 8
    for use_cuda_graph in (False, True):
        for got, expected in zip(runner.run(data, use_cuda_graph=use_cuda_graph), want):
            np.testing.assert_array_equal(got, expected)
    # the application's activation at an odd address (no tensor core)
    if data[0].size * heads * d < 1 << 24:
        shifted = torch.zeros(data[0].size + 1, dtype=torch.uint8, device="cuda")
        shifted[1:] = torch.from_numpy(data[0].reshape(-1).view(np.uint8)).cuda()
        runner.session.set_external(*runner._in_keys[0][:2], shifted.data_ptr() + 1)
        for t in runner.outputs:
            t.zero_()
        runner.dispatch()
        for got, expected in zip(runner.get_outputs(), want):
            np.testing.assert_array_equal(got, expected)
