"""Attention of few short sequences (kernels/attn_small_device.inc): rows and keys that fill neither a warp's lanes nor its four rows, head
widths off the chunks of eight, an operand of the expression per row, all three forms of the result, rows whose weights are all 0."""
import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with pytest.MonkeyPatch.context() as m:
        m.setenv("SAGE_VERBOSE_NAMES", "1")
        c = S.Context(0)
    yield c
    c.close()


# (n, heads, queries, keys, head width); the last: one more key than the form takes, two blocks of queries
@pytest.mark.parametrize("n,heads,lq,lk,d,small", [(1, 12, 24, 24, 64, True), (2, 3, 1, 1, 64, True), (1, 2, 33, 47, 64, True), (3, 2, 31, 32, 32, True), (70, 6, 5, 16, 64, True),
                                                   (40, 12, 17, 30, 64, True), (1, 1, 32, 33, 20, True), (5, 3, 9, 13, 12, True), (1, 2, 64, 48, 64, True), (2, 2, 64, 49, 64, False)])
@pytest.mark.parametrize("per_row", [False, True])
def test_attention(ctx, n, heads, lq, lk, d, small, per_row):
    """Products and sums in fp32: within 2^-20 of the largest value a head has, and the following product's bound for the pieces."""
    rng = np.random.default_rng(n + lq + lk)
    w = heads * d
    q, k, v = (rng.standard_normal((n, l, w)).astype(np.float32) * s for l, s in ((lq, 1), (lk, 1), (lk, 3)))
    mask = np.where(rng.random((n, 1, lq if per_row else 1, lk)) < 0.2, -1e5, 0).astype(np.float32)
    mask[..., 0] = 0
    if n > 1:
        mask[-1] = -1e5  # nothing left: 0 / 0, as the reference's max(m, 0) has it

    def split(t, l):
        return S.transpose(S.view(t, [n, l, heads, d]), 2, 1)
    scores = S.matmul_batched(split(ctx.var(q), lq), S.transpose(split(ctx.var(k), lk), -1, -2)) / float(np.sqrt(np.float32(d)))
    p = S.softmax(scores + ctx.var(mask), [3])
    y = S.view(S.transpose(S.matmul_batched(p, split(ctx.var(v), lk)), 2, 1), [n * lq, w])
    wo = (rng.standard_normal((w, 64)) / np.sqrt(w)).astype(np.float32)
    z = S.matmul(y, ctx.var(wo))
    ctx.clear()
    ctx.trace_begin()
    ctx.eval(y)
    got = ctx.read(y)
    names = [t for t in ctx.trace() if t.startswith("attention")]
    if names:  # (the smallest products stay by themselves)
        assert all(t.startswith("attention_tc_h2[") and t.endswith(",small]") == small for t in names), names
    got_z = z.eval(ctx)
    ctx.clear()
    ctx.eval(z)  # the pieces alone
    again = ctx.read(z)
    q64, k64, v64 = (t.astype(np.float64).reshape(n, -1, heads, d).transpose(0, 2, 1, 3) for t in (q, k, v))
    s = q64 @ k64.transpose(0, 1, 3, 2) / np.sqrt(d) + mask
    with np.errstate(invalid="ignore"):
        e = np.exp(s - np.maximum(s.max(-1, keepdims=True), 0.0))
        ref = ((e / e.sum(-1, keepdims=True)) @ v64).transpose(0, 2, 1, 3).reshape(n * lq, w)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert np.abs(got[ok] - ref[ok]).max() <= 2.0 ** -20 * np.abs(v).max() * 4  # (scores of up to 5: their rounding, 2^-24 of 5, in the exponent)
    rows = ok.all(1)
    for a in (got_z, again):
        assert np.abs(a[rows] - ref[rows] @ wo.astype(np.float64)).max() <= 2.0 ** -18 * (np.abs(ref[rows]) @ np.abs(wo.astype(np.float64))).max() + 2.0 ** -18 * np.abs(v).max()
    assert ctx.status_word() == 0


@pytest.mark.parametrize("lq,lk", [(24, 24), (33, 47)])
def test_what_is_not_finite(ctx, lq, lk):
    """Infinities and nan in queries, keys, values and the expression's operand: in the places where e / sum(e) of exp(s - max(s, 0)) has them, and
    every other value as close as ever."""
    n, heads, d = 1, 2, 64
    rng = np.random.default_rng(lq)
    w = heads * d
    q, k, v = (rng.standard_normal((n, l, w)).astype(np.float32) for l in (lq, lk, lk))
    mask = np.zeros((n, 1, lq, lk), np.float32)
    mask[0, 0, :, 3] = -np.inf       # a key nobody looks at
    mask[0, 0, 5, 7] = np.nan
    mask[0, 0, 6, :] = -np.inf       # a row of nothing
    mask[0, 0, 8, 2] = np.inf
    q[0, 10, 4], q[0, 11, 70] = np.nan, np.inf  # a row of one head each
    k[0, 9, 20] = -np.inf            # a key of the first head: rows of either sign
    v[0, 3, 100], v[0, 12, 101], v[0, 13, 102] = np.inf, np.inf, np.nan  # one under weights of 0, two that count, in the second head

    def split(t, l):
        return S.transpose(S.view(t, [n, l, heads, d]), 2, 1)
    scores = S.matmul_batched(split(ctx.var(q), lq), S.transpose(split(ctx.var(k), lk), -1, -2)) / float(np.sqrt(np.float32(d)))
    y = S.view(S.transpose(S.matmul_batched(S.softmax(scores + ctx.var(mask), [3]), split(ctx.var(v), lk)), 2, 1), [n * lq, w])
    ctx.clear()
    ctx.trace_begin()
    ctx.eval(y)
    got = ctx.read(y)
    assert [t for t in ctx.trace() if t.startswith("attention")] == ["attention_tc_h2[%dx%dx%dx%d,small]" % (lq, lk, d, heads)]
    with np.errstate(invalid="ignore", over="ignore"):
        q64, k64, v64 = (t.astype(np.float64).reshape(n, -1, heads, d).transpose(0, 2, 1, 3) for t in (q, k, v))
        s = np.einsum("bhqd,bhkd->bhqk", q64, k64) / np.sqrt(d) + mask
        e = np.exp(s - np.maximum(s.max(-1, keepdims=True), 0.0))
        ref = np.einsum("bhqk,bhkd->bhqd", e / e.sum(-1, keepdims=True), v64).transpose(0, 2, 1, 3).reshape(n * lq, w)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
    ok = np.isfinite(ref)
    assert 0.3 < ok.mean() < 0.97 and np.abs(got[ok] - ref[ok]).max() <= 2.0 ** -20 * np.abs(v[np.isfinite(v)]).max() * 4
    assert ctx.status_word() == 0
