"""What a training step's plan leaves out: copies of the attention heads that only products read (they read them through the view),
the copy behind a product whose transpose has the wanted layout, and passes of a softmax's gradient beside its row program."""
import numpy as np
import pytest

import sage_b200 as S


def gradients(ctx, heads, d, length, batch, layers=1, seed=0):
    w = heads * d
    rng = np.random.default_rng(seed)
    model = S.Bert(embed_dim=w, num_vocabs=50, max_num_tokens=max(length, 4), hidden_dim=2 * w, num_layers=layers, num_heads=heads, num_classes=2)
    for i, p in enumerate(model.params()):
        ctx.set(p, (rng.standard_normal(p.extents) * 0.2 + (1.0 if p.extents == (1,) and i % 2 == 0 else 0.0)).astype(np.float32))
    ids = ctx.var(rng.integers(0, 50, (batch, length)).astype(np.uint32))
    mask = np.ones((batch, length), np.float32)
    mask[0, length - length // 4:] = 0
    loss = S.softmax_cross_entropy(model.pass_(ids, ctx.var(mask)), ctx.var(rng.integers(0, 2, (batch, 1)).astype(np.uint32))).mean([0], False)
    return [loss] + list(S.grad_param(loss, model).values())


@pytest.mark.parametrize("heads,d,length", [(12, 64, 128), (3, 64, 72)])
def test_no_copies_of_heads_are_left(heads, d, length):
    c = S.Context(-1)
    targets = gradients(c, heads, d, length, 4)
    c.eval(*targets)
    plan = c.describe()
    copies = [line for line in plan.splitlines() if "map{(x0)}" in line and "permute" in line]
    assert not copies, copies
    assert plan.count("permute(reshape(state))") >= 4 and "[store]" in plan
    assert "14 maps, 2 reductions" in plan  # the softmax's gradient, scale included, is one row program
    c.close()


# (34 elements a head: rows off the 16-byte grid, which TMA cannot read: the copies stay)
@pytest.mark.gpu
@pytest.mark.parametrize("heads,d,length,batch", [(2, 64, 64, 2), (3, 36, 72, 3), (3, 20, 72, 2), (2, 34, 65, 2), (1, 32, 128, 2), (4, 64, 33, 5)])
def test_gradients_are_those_of_the_plain_evaluation(heads, d, length, batch):
    """Against the same graph evaluated operator by operator.  Gradients are sums of a few thousand products through two row
    normalisations: the largest difference stays below 2^-14 of the gradient's largest element (rounding 2^-24 x sqrt(terms) ~ 2^-18,
    times the amplification of two LayerNorms); of LayerNorm's scalars, sums over all n ~ 10^4 elements that cancel, sqrt(n) ~ 2^7 less."""
    got = []
    for fusion in (1, 0):
        c = S.Context(0, pattern_fusion=fusion)
        try:
            targets = gradients(c, heads, d, length, batch, layers=2)
            for _ in range(2):
                c.clear()
                c.eval(*targets)
            got.append([c.read(t).copy() for t in targets])
            assert c.status_word() == 0
        finally:
            c.close()
    assert np.abs(got[0][0] - got[1][0]).max() <= 1e-5 * max(1.0, np.abs(got[1][0]).max())
    scale = max(np.abs(g).max() for g in got[1][1:])
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.abs(a - b).max() <= 2.0 ** (-14 if a.size > 1 else -14 + 7) * max(np.abs(b).max(), 2.0 ** -10 * scale)


def views(c, kind, shift, seed=0):
    """A value, read by products alone, that starts `shift` elements into the storage it lies in."""
    rng = np.random.default_rng(seed)
    m, k = 256, 128
    x = rng.standard_normal({"flat": (m * k + 8,), "columns": (m, k + 8), "rows": (m + 8, k)}[kind]).astype(np.float32)
    a = c.var(x) * 2.0 + 1.0
    v = S.view(a.slice(0, shift, shift + m * k), [m, k]) if kind == "flat" else a.slice(1, shift, shift + k) if kind == "columns" else a.slice(0, shift, shift + m)
    w, u, g = (rng.standard_normal(s).astype(np.float32) for s in ((k, 96), (k, 64), (m, 96)))
    x = x * 2.0 + 1.0
    x = x[shift:shift + m * k].reshape(m, k) if kind == "flat" else x[:, shift:shift + k] if kind == "columns" else x[shift:shift + m]
    return v, [v.matmul(c.var(w)), v.matmul(c.var(u)), S.transpose(v, 1, 0).matmul(c.var(g))], [x @ w, x @ u, x.T @ g], [np.abs(x) @ np.abs(w), np.abs(x) @ np.abs(u), np.abs(x).T @ np.abs(g)]


@pytest.mark.parametrize("kind", ["flat", "columns", "rows"])
@pytest.mark.parametrize("shift", [0, 1, 2, 4])
def test_what_products_alone_read_keeps_values_only_where_they_need_them(kind, shift):
    """Products read planes where a view's rows lie on 16 bytes, whatever state the view is; else they gather its values."""
    for more in (None, "value", "sum"):
        c = S.Context(-1)
        v, products, _, _ = views(c, kind, shift)
        c.eval(*products, *([v] if more == "value" else [v.exp().sum([0], False)] if more == "sum" else []))
        first = c.describe().splitlines()[0]
        direct = shift % 4 == 0 or kind == "rows"
        assert ("=planes" in first) == (direct and more is None) and ("+planes" in first) == (direct and more is not None), first
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["flat", "columns", "rows"])
@pytest.mark.parametrize("shift", [0, 1, 2, 4])
def test_products_of_views_that_start_anywhere(kind, shift):
    """Within 2^-19 of |a| |b|, the bound of the products."""
    c = S.Context(0)
    try:
        _, products, want, size = views(c, kind, shift)
        for _ in range(2):
            c.clear()
            c.eval(*products)
        for p, w, s in zip(products, want, size):
            assert (np.abs(c.read(p) - w) <= 2.0 ** -19 * s).all()
        assert c.status_word() == 0
    finally:
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,d,length,batch", [(2, 64, 64, 2), (3, 36, 72, 3), (3, 20, 72, 2), (2, 34, 65, 2), (1, 32, 128, 2), (4, 64, 33, 5)])
def test_gradients_of_scalars(heads, d, length, batch):
    """LayerNorm's scalars against the same graph evaluated operator by operator: sums over all n ~ 10^4 elements that may cancel, so below
    2^-14 of the largest element of all gradients, not of themselves (2^-14.9 ... 2^-21.7 seen)."""
    got = []
    for fusion in (1, 0):
        c = S.Context(0, pattern_fusion=fusion)
        try:
            targets = gradients(c, heads, d, length, batch, layers=2)[1:]
            c.eval(*targets)
            got.append([c.read(t).copy() for t in targets])
            assert c.status_word() == 0
        finally:
            c.close()
    scale = max(np.abs(g).max() for g in got[1])
    scalars = [(a, b) for a, b in zip(*got) if a.size == 1]
    assert len(scalars) == 10 and all(np.abs(a - b).max() <= 2.0 ** -14 * scale for a, b in scalars), len(scalars)


@pytest.mark.parametrize("levels", [1, 7, 8, 9, 12])
def test_products_at_the_end_of_a_chain_of_views(levels):
    """Views of views, each a state: a product on the 16-byte grid reads every one of them, and two off it the last, which gather values."""
    c = S.Context(-1)
    m, k = 256, 64

    def matrix(v, at):
        return S.view(v.slice(0, at, at + m * k), [m, k])
    size = m * k + 4 * levels + 8
    v = (c.var(np.zeros(size + 1, np.float32)) * 2.0 + 1.0).slice(0, 1, size + 1)
    w, g = c.var(np.zeros((k, 96), np.float32)), c.var(np.zeros((m, 96), np.float32))
    targets = []
    for _ in range(levels):
        targets.append(matrix(v, 3).matmul(w))
        v = v.slice(0, 4, v.extents[0])
    c.eval(*targets, matrix(v, 0).matmul(w), S.transpose(matrix(v, 0), 1, 0).matmul(g))
    first = c.describe().splitlines()[0]
    assert "+planes" in first and "=planes" not in first, first
    c.close()
