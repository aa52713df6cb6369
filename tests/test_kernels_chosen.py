"""Which kernels the rules choose: the verbose launch lists of planning contexts.  The values of the same sizes are compared on the device
(test_gpu_attention_small.py, test_gpu_conv_gradients.py, test_gpu_few_outputs.py, test_gpu_store_loops.py), where a rule that stopped
choosing a kernel would leave them right."""
import numpy as np
import pytest

import sage_b200 as S


@pytest.fixture
def ctx(monkeypatch):
    monkeypatch.setenv("SAGE_VERBOSE_NAMES", "1")
    c = S.Context(-1)
    yield c
    c.close()


def launches(ctx, *targets):
    ctx.clear()
    ctx.trace_begin()
    ctx.eval(*targets)
    return ctx.trace()


def var(ctx, *shape):
    return ctx.var(np.zeros(shape, np.float32))


@pytest.mark.parametrize("n,heads,lq,lk,d,small", [(1, 12, 24, 24, 64, True), (2, 3, 1, 1, 64, True), (1, 2, 33, 47, 64, True), (3, 2, 31, 32, 32, True), (70, 6, 5, 16, 64, True),
                                                   (40, 12, 17, 30, 64, True), (1, 1, 32, 33, 20, True), (5, 3, 9, 13, 12, True), (1, 2, 64, 48, 64, True), (2, 2, 64, 49, 64, False)])
@pytest.mark.parametrize("per_row", [False, True])
def test_small_attention(ctx, n, heads, lq, lk, d, small, per_row):
    def split(l):
        return S.transpose(S.view(var(ctx, n, l, heads * d), [n, l, heads, d]), 2, 1)
    scores = S.matmul_batched(split(lq), S.transpose(split(lk), -1, -2)) / float(np.sqrt(np.float32(d)))
    p = S.softmax(scores + var(ctx, n, 1, lq if per_row else 1, lk), [3])
    y = S.view(S.transpose(S.matmul_batched(p, split(lk)), 2, 1), [n * lq, heads * d])
    assert [t for t in launches(ctx, y) if t.startswith("attention")] == ["attention_tc_h2[%dx%dx%dx%d%s]" % (lq, lk, d, n * heads, ",small" if small else "")]


# three column matrices (a rectifier is part of its own, a tanh too long to be worked out for every tap), and the maps behind every gradient of
# an image; channels off the fours keep their own maps; a K long enough for slices, which the map behind the product adds up
@pytest.mark.parametrize("b,hw,c,ker,stride,pad,residual", [(4, 9, 32, 3, 1, 1, True), (3, 12, 64, 3, 2, 1, False), (2, 7, 34, 3, 1, 1, True), (8, 4, 256, 3, 1, 1, True), (16, 5, 36, 5, 1, 2, False)])
@pytest.mark.parametrize("smooth", [False, True])
def test_maps_of_column_matrices(ctx, b, hw, c, ker, stride, pad, residual, smooth):
    xv, wv, bv = var(ctx, b, hw, hw, c), [var(ctx, ker, ker, c, c) for _ in range(3)], [var(ctx, c) for _ in range(3)]
    act = (lambda v: v.tanh()) if smooth else S.relu
    h = act(S.conv_2d(xv * 1.5, wv[0], stride, pad, 1) + bv[0])
    h1 = S.conv_2d(h, wv[1], 1, pad, 1) + bv[1]
    h2 = act(h1 + h if residual else h1)
    y = S.conv_2d(h2, wv[2], 1, pad, 1) + bv[2]
    loss = (y * y).sum([0, 1, 2, 3], False)
    names = [t.split("{")[0] + "{map}" if "{map}" in t else t for t in launches(ctx, loss, *[v.grad(loss) for v in [xv] + wv + bv])]
    assert names.count("im2col{map}") == (0 if c % 4 else 1 if smooth else 3), names
    assert ("col2im{map}" in names, "col2im" in names) == (c % 4 == 0, c % 4 != 0), names
    assert any(t.startswith("map{") and ",ZG" in t for t in names) == (c == 256), names


# (the last is a tensor-core product)
@pytest.mark.parametrize("m,n,k", [(1, 1000, 512), (32, 2, 768), (1, 2, 1024), (3, 33, 129), (7, 32, 255), (128, 10, 512), (16, 100, 257), (1, 8192, 128)])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
def test_products_of_few_outputs(ctx, m, n, k, ta, tb):
    x, y = var(ctx, *((k, m) if ta else (m, k))), var(ctx, *((n, k) if tb else (k, n)))
    assert launches(ctx, S.gemm(x, y, ta, tb))[-1].split("x")[0] == ("gemm_tc_h2[1" if n == 8192 else "gemm_simt[skinny]" if tb or n < 32 else "gemm_simt[columns]")


@pytest.mark.parametrize("shape,ker,stride,pad", [((1, 7, 7, 512), 7, 1, 0), ((2, 9, 8, 36), 4, 2, 1), ((1, 20, 20, 68), 9, 6, 3), ((3, 5, 5, 64), 5, 1, 2), ((400, 7, 7, 128), 7, 1, 0), ((1, 7, 7, 66), 7, 1, 0)])
@pytest.mark.parametrize("is_max", [False, True])
def test_pooling_of_large_windows(ctx, shape, ker, stride, pad, is_max):
    window = shape[0] < 400 and shape[3] % 4 == 0
    assert launches(ctx, (S.max_pool_2d if is_max else S.avg_pool_2d)(var(ctx, *shape), ker, stride, pad, 1)) == [("max_pool2d" if is_max else "avg_pool2d") + ("[window]" if window else "")]


@pytest.mark.parametrize("m,k,n,single", [(129, 256, 192, True), (200, 320, 97, True), (462, 768, 3072, True), (4096, 512, 2048, False), (130, 64, 130, True), (5000, 256, 1000, False)])
@pytest.mark.parametrize("long", [False, True])
def test_stores_in_a_loop(ctx, m, k, n, single, long):
    h = var(ctx, m, k).matmul(var(ctx, k, n)) + var(ctx, n)
    y = h * 0.5 * ((h * 0.70710678).erf() + 1.0) if long else S.relu(h)
    z = y.matmul(var(ctx, n, 64))
    for targets in ((y,), (z,), (y, z)):
        names = [t for t in launches(ctx, *targets) if t.startswith("gemm_tc_h2[%dx%dx%d," % (m, n, k))]
        assert len(names) == 1 and (",rolled" in names[0]) == (single or long), names


# `kind`: the tile of those that take the residual through the ring; None: several tiles to a CTA, or slices
@pytest.mark.parametrize("m,k,n,kind", [(129, 64, 64, ",bn64,pair"), (200, 320, 100, None), (300, 256, 128, None), (4096, 768, 768, ",bn256/0+4x192,pair"), (1536, 128, 192, ",bn64,pair"), (2000, 200, 516, ",bn64,pair"),
                                        (6000, 128, 1024, None), (130, 96, 260, ",bn64,pair"), (1100, 200, 1000, ",bn128,pair"), (1100, 64, 1024, ",bn128,pair"), (4096, 200, 1000, ",bn256,pair"),
                                        (3000, 96, 1000, ",bn256/0+6x192,pair"), (120, 96, 260, ",bn64")])
@pytest.mark.parametrize("wider,shift", [(0, 0), (8, 4), (8, 1)])
def test_residuals_through_the_ring(ctx, m, k, n, kind, wider, shift):
    rv = var(ctx, m, n + wider)
    if wider:
        rv = rv.slice(1, shift, shift + n)
    names = [t for t in launches(ctx, var(ctx, m, k).matmul(var(ctx, k, n)) + var(ctx, n) + rv) if t.startswith("gemm_tc_h2[%dx%dx%d," % (m, n, k))]
    assert len(names) == 1 and (",residual1]" in names[0]) == (kind is not None and shift != 1), names
    assert kind is None or kind + (",residual1" if shift != 1 else "") + "]" in names[0], names
