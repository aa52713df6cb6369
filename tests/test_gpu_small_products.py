"""Products with fewer rows than a tensor-core tile (single requests, short sequences): the shapes around the line between
the tiled and the SIMT kernel, and attention over sequences shorter than one key block.

Tolerances: |a - b| / max(|b|, rms) <= 1e-5 against float64 for a product (fp32 sums of at most 3072 terms), 1e-4 for the
attention block (a softmax between two products), as in the other contraction tests.
"""
import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with pytest.MonkeyPatch.context() as m:
        m.setenv("SAGE_VERBOSE_NAMES", "1")  # the launch list tells the kernels apart
        c = S.Context(0)
    yield c
    c.close()


def rms_err(got, ref):
    a, b = np.asarray(got, np.float64), np.asarray(ref, np.float64)
    assert a.shape == b.shape
    return float((np.abs(a - b) / np.maximum(np.abs(b), np.sqrt((b ** 2).mean()))).max())


@pytest.mark.parametrize("m,n,k,tiled", [(1, 4128, 129, True), (2, 2049, 768, True), (24, 768, 768, True), (63, 96, 1000, True), (33, 200, 3072, True),
                                         (1, 4096, 768, False), (40, 100, 512, False), (63, 511, 127, False)])
def test_products_with_few_rows(ctx, m, n, k, tiled):
    rng = np.random.default_rng(8001)
    x = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    w = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    b = rng.uniform(-1, 1, (n,)).astype(np.float32)
    y = S.relu(S.matmul(ctx.var(x), ctx.var(w)) + ctx.var(b))
    ctx.clear()
    ctx.trace_begin()
    got = y.eval(ctx)
    assert any(t.startswith("gemm_tc") for t in ctx.trace()) == tiled
    assert rms_err(got, np.maximum(x.astype(np.float64) @ w.astype(np.float64) + b, 0.0)) <= 1e-5
    assert ctx.status_word() == 0


@pytest.mark.parametrize("n,heads,l,d", [(1, 12, 24, 64), (2, 4, 2, 64), (3, 2, 31, 32), (1, 1, 63, 64), (5, 3, 9, 16)])
def test_attention_over_short_sequences(ctx, n, heads, l, d):
    rng = np.random.default_rng(8002)
    q, k, v = (rng.standard_normal((n, l, heads * d)).astype(np.float32) for _ in range(3))
    mask = np.ones((n, l), np.float32)
    mask[-1, l - l // 3:] = 0

    def split(t):
        return S.transpose(S.view(t, [n, l, heads, d]), 2, 1)
    scores = S.matmul_batched(split(ctx.var(q)), S.transpose(split(ctx.var(k)), -1, -2)) / float(np.sqrt(np.float32(d)))
    p = S.softmax(scores + (-(S.view(ctx.var(mask), [n, 1, 1, l])) + 1.0) * -1e5, [3])
    y = S.view(S.transpose(S.matmul_batched(p, split(ctx.var(v))), 2, 1), [n, l, heads * d])
    ctx.clear()
    ctx.trace_begin()
    got = y.eval(ctx)
    assert any(t.startswith("attention_tc_h2[") for t in ctx.trace())
    q64, k64, v64 = (t.astype(np.float64).reshape(n, l, heads, d).transpose(0, 2, 1, 3) for t in (q, k, v))
    s = q64 @ k64.transpose(0, 1, 3, 2) / np.sqrt(d) + (1.0 - mask)[:, None, None, :] * -1e5
    e = np.exp(s - np.maximum(s.max(-1, keepdims=True), 0.0))
    ref = ((e / e.sum(-1, keepdims=True)) @ v64).transpose(0, 2, 1, 3).reshape(n, l, heads * d)
    assert rms_err(got, ref) <= 1e-4
    assert ctx.status_word() == 0
