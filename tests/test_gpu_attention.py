"""GPU parity of the fused attention node: key counts at and beside the tensor core's steps of 32, the tile of 128, the
two-blocks-per-SM limit of 192 and the largest row of 512; query counts with ragged tiles; every head dimension; signed
and unsigned probabilities.  Bit-exact against the CPU oracle, which evaluates the twenty operators one by one."""
import math

import numpy as np
import pytest

from mlel_b200.graph_builder import GraphBuilder
from tests.graph_eval import evaluate

pytestmark = pytest.mark.gpu

ATTENTION = "ATTENTION(MATMUL+SOFTMAX+MATMUL+RESCALE)"


def attention_graph(n, heads, sq, sk, d, prob_zp=-128, double_round=False, merge=True, pow2=False, seed=0):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = (np.arange(513, dtype=np.float64) - 256.0) * 128.0
    exp_lut = np.round(32767.0 * np.exp(np.minimum(x, 0.0) / 4096.0)).astype(np.int16)
    recip_lut = np.clip(np.round(32767.0 * 256.0 / (x + 32768.0 + 256.0)), 0, 32767).astype(np.int16)
    g = GraphBuilder("attention")
    xs = [g.input(np.int8, (n, s, heads, d)) for s in (sq, sk, sk)]
    data = [rng.integers(-128, 128, v.shape, dtype=np.int8) for v in xs]
    q, k, v = (g.clamp(t, -128, 127) for t in xs)  # session tensors, as projections leave them
    q = g.reshape(g.transpose(q, (0, 2, 1, 3)), (n * heads, sq, d))
    k = g.reshape(g.transpose(k, (0, 2, 3, 1)), (n * heads, d, sk))
    v = g.reshape(g.transpose(v, (0, 2, 1, 3)), (n * heads, sk, d))
    s = g.matmul(q, k, 0, 0)
    diff = g.sub(s, g.reduce("REDUCE_MAX", s, 2))
    e = g.table(g.rescale(diff, [1 << 30 if pow2 else int(rng.integers(1 << 30, 1 << 31))], [30 + max(2, int(math.log2(d)) - 2)], 0, 0, np.int16,
                          double_round=double_round), exp_lut)
    log_keys = max(1, math.ceil(math.log2(sk)))
    denom = g.rescale(g.reduce("REDUCE_SUM", e, 2), [1 << 30], [37 + log_keys], 0, -32768, np.int16)
    r = g.table(denom, recip_lut)
    p = g.rescale(g.mul(e, r, 22), [1 << 30 if pow2 else (1 << 30) + 12345], [37 + log_keys - (0 if prob_zp else 1)], 0, prob_zp, np.int8,
                  double_round=double_round)
    c = g.rescale(g.matmul(p, v, prob_zp, 0), [int(rng.integers(1 << 30, 1 << 31))], [38], 0, 3, np.int8, double_round=True)
    if merge:
        c = g.transpose(g.reshape(c, (n, heads, sq, d)), (0, 2, 1, 3))
    g.output(g.clamp(c, -127, 126))
    return g, data


@pytest.mark.parametrize("n,heads,sq,sk,d", [
    (1, 1, 128, 128, 64), (1, 2, 32, 32, 32), (2, 3, 197, 197, 64), (1, 1, 130, 33, 128), (1, 2, 1, 512, 64),
    (3, 2, 129, 191, 96), (1, 4, 192, 192, 64), (1, 2, 100, 193, 64), (1, 1, 300, 384, 64), (1, 2, 65, 256, 32),
    (2, 1, 511, 511, 128), (20, 12, 257, 65, 64), (1, 1, 40, 16, 64), (3, 2, 19, 19, 64), (1, 2, 7, 1, 32),
])
@pytest.mark.parametrize("prob_zp,double_round,pow2", [(-128, False, False), (0, True, False), (-128, True, True), (0, False, True)])
def test_attention_matches_the_operators(mlel, n, heads, sq, sk, d, prob_zp, double_round, pow2):
    from mlel_b200.runtime import GraphRunner
    g, data = attention_graph(n, heads, sq, sk, d, prob_zp, double_round, merge=(sq % 2 == 0 or n > 1), pow2=pow2, seed=sk)
    runner = GraphRunner(g)
    assert ATTENTION in runner.pipeline.exec_names(), runner.pipeline.exec_names()
    want = evaluate(g, data)[0]
    assert np.unique(want).size > 8
    for use_cuda_graph in (False, True):
        got = runner.run(data, use_cuda_graph=use_cuda_graph)[0]
        bad = np.argwhere(got != want)
        assert len(bad) == 0, (len(bad), got.size, bad[:4].tolist())


@pytest.mark.parametrize("n,heads,sq,sk,d", [(1, 1, 16, 513, 32), (1, 2, 48, 48, 16)])
def test_attention_outside_the_kernel_stays_with_the_operators(mlel, n, heads, sq, sk, d):
    from mlel_b200.runtime import GraphRunner
    g, data = attention_graph(n, heads, sq, sk, d, seed=7)
    runner = GraphRunner(g)
    assert ATTENTION not in runner.pipeline.exec_names()
    np.testing.assert_array_equal(runner.run(data)[0], evaluate(g, data)[0])


def softmax_variant(form, n, heads, s, d, seed):
    """An attention that is not the fused node's: a mask added to the scores, the factors of MUL the other way round, a
    second reader of the probabilities."""
    rng = np.random.Generator(np.random.PCG64(seed))
    x = (np.arange(513, dtype=np.float64) - 256.0) * 128.0
    exp_lut = np.round(32767.0 * np.exp(np.minimum(x, 0.0) / 4096.0)).astype(np.int16)
    recip_lut = np.clip(np.round(32767.0 * 256.0 / (x + 32768.0 + 256.0)), 0, 32767).astype(np.int16)
    g = GraphBuilder("attention_variant")
    q, k, v = g.input(np.int8, (n * heads, s, d)), g.input(np.int8, (n * heads, d, s)), g.input(np.int8, (n * heads, s, d))
    data = [rng.integers(-128, 128, t.shape, dtype=np.int8) for t in (q, k, v)]
    q, k, v = (g.clamp(t, -128, 127) for t in (q, k, v))
    scores = g.matmul(q, k, 0, 0)
    if form == "mask":
        mask = g.input(np.int32, (n * heads, 1, s))
        data.append(np.where(rng.random((n * heads, 1, s)) < 0.3, -(1 << 22), 0).astype(np.int32))
        scores = g.add(scores, mask)
    diff = g.sub(scores, g.reduce("REDUCE_MAX", scores, 2))
    e = g.table(g.rescale(diff, [1 << 30], [30 + max(2, int(math.log2(d)) - 2)], 0, 0, np.int16), exp_lut)
    log_keys = max(1, math.ceil(math.log2(s)))
    r = g.table(g.rescale(g.reduce("REDUCE_SUM", e, 2), [1 << 30], [37 + log_keys], 0, -32768, np.int16), recip_lut)
    p = g.rescale(g.mul(r, e, 22) if form == "swapped" else g.mul(e, r, 22), [1 << 30], [37 + log_keys], 0, -128, np.int8)
    if form == "read twice":
        g.output(g.clamp(p, -100, 100))
    g.output(g.rescale(g.matmul(p, v, -128, 0), [(1 << 30) + 3], [38], 0, 3, np.int8, double_round=True))
    return g, data


@pytest.mark.parametrize("form", ["mask", "swapped", "read twice"])
@pytest.mark.parametrize("n,heads,s,d", [(2, 3, 64, 32), (1, 2, 197, 64)])
def test_attention_of_another_form_stays_with_the_operators(mlel, form, n, heads, s, d):
    from mlel_b200.runtime import GraphRunner
    g, data = softmax_variant(form, n, heads, s, d, s)
    runner = GraphRunner(g)
    assert ATTENTION not in runner.pipeline.exec_names()
    want = evaluate(g, data)
    for use_cuda_graph in (False, True):
        for a, b in zip(runner.run(data, use_cuda_graph=use_cuda_graph), want):
            np.testing.assert_array_equal(a, b)
