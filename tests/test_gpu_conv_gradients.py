"""Column matrices and their inverses with the map before or behind them spliced in (kernels/conv_cols_device.inc), and products in K slices
whose sum is part of the map that follows: gradients of small convolution chains against torch in float64."""
import numpy as np
import pytest
import torch

import sage_b200 as S

pytestmark = pytest.mark.gpu


# (batch, size, channels, kernel, stride, padding): whole rows and ragged ones, channels off the fours (which keep their own map), windows
# larger than the image's rows, a residual, K long enough for slices
@pytest.mark.parametrize("b,hw,c,ker,stride,pad,residual", [(4, 9, 32, 3, 1, 1, True), (3, 12, 64, 3, 2, 1, False), (2, 7, 34, 3, 1, 1, True), (8, 4, 256, 3, 1, 1, True), (16, 5, 36, 5, 1, 2, False)])
@pytest.mark.parametrize("smooth", [False, True])
def test_gradients(b, hw, c, ker, stride, pad, residual, smooth):
    """Every tensor within 2^-15 of its largest element: products of two convolutions' 2^-20 each, sums of up to b hw^2 = 10^3 terms."""
    rng = np.random.default_rng(c + ker)
    x = rng.standard_normal((b, hw, hw, c)).astype(np.float32)
    w = [(rng.standard_normal((ker, ker, c, c)) / np.sqrt(ker * ker * c)).astype(np.float32) for _ in range(3)]
    bias = [rng.standard_normal(c).astype(np.float32) * np.float32(0.1) for _ in range(3)]
    ctx = S.Context(0)
    try:
        xv, wv, bv = ctx.var(x), [ctx.var(v) for v in w], [ctx.var(v) for v in bias]
        act = (lambda v: v.tanh()) if smooth else S.relu
        h = act(S.conv_2d(xv * 1.5, wv[0], stride, pad, 1) + bv[0])
        h1 = S.conv_2d(h, wv[1], 1, pad, 1) + bv[1]
        h2 = act(h1 + h if residual else h1)
        y = S.conv_2d(h2, wv[2], 1, pad, 1) + bv[2]
        loss = (y * y).sum([0, 1, 2, 3], False)
        targets = [loss] + [v.grad(loss) for v in [xv] + wv + bv]
        for _ in range(2):
            ctx.clear()
            ctx.eval(*targets)
        got = [ctx.read(t).copy() for t in targets]
        assert ctx.status_word() == 0
    finally:
        ctx.close()
    tx, tw, tb = torch.from_numpy(x).double().requires_grad_(), [torch.from_numpy(v).double().requires_grad_() for v in w], [torch.from_numpy(v).double().requires_grad_() for v in bias]

    def conv(v, i, s):
        return torch.nn.functional.conv2d(v.permute(0, 3, 1, 2), tw[i].permute(3, 2, 0, 1), tb[i], s, pad).permute(0, 2, 3, 1)
    tact = torch.tanh if smooth else torch.relu
    t = tact(conv(tx * 1.5, 0, stride))
    t1 = conv(t, 1, 1)
    t2 = tact(t1 + t if residual else t1)
    out = conv(t2, 2, 1)
    tl = (out * out).sum()
    tl.backward()
    for g, ref in zip(got, [tl.detach()] + [v.grad for v in [tx] + tw + tb]):
        ref = ref.numpy()
        assert np.abs(g.reshape(ref.shape) - ref).max() <= 2.0 ** -15 * np.abs(ref).max()


@pytest.fixture
def verbose(monkeypatch):
    monkeypatch.setenv("SAGE_VERBOSE_NAMES", "1")  # the launch list tells the kernels apart


# (rows, K, columns) of products in K slices whose sum is part of the map behind them: whole 16-byte loads, and rows that are not
@pytest.mark.parametrize("m,k,n,vec", [(128, 4096, 64, 4), (129, 4096, 36, 4), (100, 4096, 34, 1), (64, 8192, 65, 1), (128, 4160, 33, 1)])
@pytest.mark.usefixtures("verbose")
def test_slices_in_the_map(m, k, n, vec):
    """The product within (2^-22 + 128 x 2^-23 + (K / 128 + 1) 2^-24) |x| |w|: the dropped low x low products, a chain's truncating additions, a
    rounding for every chain and slice; its bias and rectifier add 2^-23 of what they read."""
    rng = np.random.default_rng(m + n)
    x, w, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    ctx = S.Context(0)
    try:
        xv, wv, bv = ctx.var(x), ctx.var(w), ctx.var(b)
        y = S.relu(xv.matmul(wv) + bv)
        loss = (y * y).sum([0, 1], False)
        targets = [y, loss, wv.grad(loss), xv.grad(loss)]
        for _ in range(2):
            ctx.clear()
            ctx.trace_begin()
            ctx.eval(*targets)
        assert any(t.startswith("map{") and ",v%d,ZG" % vec in t for t in ctx.trace()), ctx.trace()
        got = ctx.read(y).copy()
        assert ctx.status_word() == 0
    finally:
        ctx.close()
    x64, w64 = x.astype(np.float64), w.astype(np.float64)
    size = np.abs(x64) @ np.abs(w64) + np.abs(b)
    assert (np.abs(got - np.maximum(x64 @ w64 + b, 0)) <= (2.0 ** -22 + 128 * 2.0 ** -23 + (k / 128 + 1) * 2.0 ** -24 + 2.0 ** -22) * size).all()


@pytest.mark.parametrize("shift", [1, 4])
@pytest.mark.usefixtures("verbose")
def test_images_that_start_anywhere(shift):
    """An image that starts off the 16-byte grid has its map worked out by itself, before the column matrix and behind the gradient of the image:
    the same values, the same sums in the same order."""
    b, hw, c = 2, 6, 8
    n = b * hw * hw * c
    rng = np.random.default_rng(shift)
    x, w, bias = rng.standard_normal(n).astype(np.float32), rng.standard_normal((3, 3, c, 32)).astype(np.float32), rng.standard_normal(32).astype(np.float32)
    got = []
    for start in (0, shift):
        ctx = S.Context(0)
        try:
            flat = np.zeros(n + 8, np.float32)
            flat[start:start + n] = x
            image = S.view(ctx.var(flat).slice(0, start, start + n), [b, hw, hw, c])
            wv = ctx.var(w)
            y = S.conv_2d(S.relu(image), wv, 1, 1, 1) + ctx.var(bias)
            loss = (y * y).sum([0, 1, 2, 3], False)
            targets = [loss, wv.grad(loss), image.grad(loss)]
            for _ in range(2):
                ctx.clear()
                ctx.trace_begin()
                ctx.eval(*targets)
            names = ctx.trace()
            on_grid = start % 4 == 0
            assert (("im2col{map}=planes" in names), ("im2col=planes" in names), ("col2im{map}" in names), ("col2im" in names)) == (on_grid, not on_grid, on_grid, not on_grid), names
            got.append([ctx.read(t).copy() for t in targets])
            assert ctx.status_word() == 0
        finally:
            ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
