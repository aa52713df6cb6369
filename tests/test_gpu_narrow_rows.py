"""Rows of fewer than 32 columns as generated programs, a warp each (graph/rowfuse.cc: row_space_narrow)."""
import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu


def reference(x, labels):
    z = x.astype(np.float64)
    m = z.max(1, keepdims=True)
    lse = np.log(np.exp(z - m).sum(1, keepdims=True)) + m
    p = np.exp(z - lse)
    p[np.arange(len(z)), labels[:, 0]] -= 1
    return (lse - np.take_along_axis(z, labels.astype(np.int64), 1))[:, 0], p


def close(got, want):
    # Sums of at most 31 fp32 terms and a few roundings of exponentials of arguments up to ~10: 16 roundings of 6e-8 each,
    # of the value or of the rms.
    return (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-6 * 4


# One vector of four and fewer, columns that are and are not whole vectors, the last narrow width; one warp, several rounds, and the first
# count of rows that is left to the other kernels.
@pytest.mark.parametrize("rows,cols", [(2, 2), (128, 10), (33, 4), (5, 31), (7, 28), (4097, 3), (262144, 2), (262145, 2)])
def test_cross_entropy_and_gradient(rows, cols):
    rng = np.random.default_rng(100 * cols + rows)
    x = (3 * rng.standard_normal((rows, cols))).astype(np.float32)
    labels = rng.integers(0, cols, (rows, 1)).astype(np.uint32)
    ctx = S.Context(0)
    try:
        xv = ctx.var(x)
        loss = S.softmax_cross_entropy(xv, ctx.var(labels))
        gx = xv.grad(loss)
        ctx.trace_begin()
        ctx.eval(loss, gx)
        assert (ctx.trace() == ["sage_narrow_rows"]) == (rows <= 262144)
        want, grad = reference(x, labels)
        assert close(ctx.read(loss).reshape(-1), want) and close(ctx.read(gx), grad)
        assert ctx.status_word() == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("rows", [4096, 4097])
def test_few_exchanges(rows):
    """Without an element picked, only up to 4096 rows."""
    x = np.random.default_rng(rows).random((rows, 5), dtype=np.float32) + 0.5
    ctx = S.Context(0)
    try:
        xv = ctx.var(x)
        y = xv / xv.sum([1], True)
        ctx.trace_begin()
        ctx.eval(y)
        assert ("sage_narrow_rows" in ctx.trace()) == (rows <= 4096)
        assert close(ctx.read(y), x.astype(np.float64) / x.astype(np.float64).sum(1, keepdims=True))
    finally:
        ctx.close()


@pytest.mark.parametrize("rows,cols", [(32, 2), (128, 10), (96, 31)])
def test_loss_of_a_training_step(rows, cols):
    """Inside a training program: the mean loss, and the gradient of the logits, which products read."""
    rng = np.random.default_rng(cols)
    a, w = (rng.standard_normal(s).astype(np.float32) / 8 for s in ((rows, 64), (64, cols)))
    labels = rng.integers(0, cols, (rows, 1)).astype(np.uint32)
    ctx = S.Context(0)
    try:
        av, wv = ctx.var(a), ctx.var(w)
        loss = S.softmax_cross_entropy(av.matmul(wv), ctx.var(labels)).mean([0], False)
        ga, gw = av.grad(loss), wv.grad(loss)
        for _ in range(2):
            ctx.clear()
            ctx.trace_begin()
            ctx.eval(loss, ga, gw)
            assert ctx.trace().count("sage_narrow_rows") == 2
            per_row, p = reference(a.astype(np.float64) @ w, labels)
            p /= rows
            assert abs(float(ctx.read(loss).reshape(-1)[0]) - per_row.mean()) <= 4e-6 * per_row.mean()
            assert close(ctx.read(ga), p @ w.T.astype(np.float64)) and close(ctx.read(gw), a.T.astype(np.float64) @ p)
        assert ctx.status_word() == 0
    finally:
        ctx.close()


def test_infinite_logits():
    """A masked class (-inf) has probability 0 and gradient 0; as the kernels one by one give it."""
    x = np.array([[0.5, -np.inf, 1.0], [-np.inf, 2.0, -np.inf], [np.finfo(np.float32).min, 0.0, 1.0]], np.float32)
    labels = np.array([[0], [1], [2]], np.uint32)
    got = []
    for fusion in (1, 5):
        ctx = S.Context(0, pattern_fusion=fusion)
        try:
            xv = ctx.var(x)
            loss = S.softmax_cross_entropy(xv, ctx.var(labels))
            gx = xv.grad(loss)
            ctx.eval(loss, gx)
            got.append((ctx.read(loss).reshape(-1), ctx.read(gx)))
        finally:
            ctx.close()
    for a, b in zip(*got):
        np.testing.assert_allclose(a, b, rtol=4e-6, atol=1e-7)
