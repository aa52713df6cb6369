"""Operands that are views, on the host side (a planning context: launches are recorded, nothing is computed)."""
import numpy as np
import pytest

import sage_b200 as S


@pytest.fixture()
def ctx():
    c = S.Context(-1)
    yield c
    c.close()


@pytest.mark.parametrize("off,tail", [(0, 5), (1, 0), (4, 0), (32, 5)])
@pytest.mark.parametrize("ker,stride,chan", [(3, 1, 64), (1, 2, 64), (3, 2, 128), (3, 1, 32), (7, 2, 3)])
def test_convolutions_of_views_are_accepted(ctx, off, tail, ker, stride, chan):
    """An image anywhere inside a storage of any length, alone and behind a pool or in front of another convolution."""
    shape = (4, 32, 32, chan)
    n = int(np.prod(shape))
    x = S.view(ctx.var(np.zeros((off + n + tail,), np.float32)).slice(0, off, off + n), list(shape))
    f, f2 = ctx.var(np.zeros((ker, ker, chan, 64), np.float32)), ctx.var(np.zeros((3, 3, 64, 64), np.float32))
    y = S.conv_2d(x, f, stride, ker // 2, 1)
    ctx.eval(y)
    ctx.eval(S.conv_2d(S.relu(y), f2, 1, 1, 1))
    ctx.eval(S.conv_2d(S.max_pool_2d(x, 2, 2, 0, 1), f, stride, ker // 2, 1))


@pytest.mark.parametrize("off", [0, 1, 32])
def test_products_of_parts_of_a_result_are_accepted(ctx, off):
    """A result that only a product reads may exist as operand pieces alone, unless the product's view of it (here behind a
    reshape) starts inside a group of 64: then it has to be gathered from the fp32 values."""
    n = 2 * 32 * 32 * 64
    w, f = ctx.var(np.zeros((64, 64), np.float32)), ctx.var(np.zeros((3, 3, 64, 64), np.float32))
    for result in (lambda: S.matmul(ctx.var(np.zeros((4096, 64), np.float32)), w), lambda: S.relu(S.conv_2d(ctx.var(np.zeros((4, 32, 32, 64), np.float32)), f, 1, 1, 1))):
        ctx.eval(S.conv_2d(S.view(S.view(result(), [2 * n]).slice(0, off, off + n), [2, 32, 32, 64]), f, 1, 1, 1))
        ctx.eval(S.matmul(S.view(S.view(result(), [2 * n]).slice(0, off, off + n), [2048, 64]), w))
        part = S.view(S.view(result(), [2 * n]).slice(0, off, off + n), [8, 4, 64, 64])
        ctx.eval(S.matmul_batched(S.softmax(S.matmul_batched(part, S.transpose(part, -1, -2)), [3]), part))


# (a slice along axis 0 of a matrix, or of the flat value), seen under another shape
RESHAPED_SLICES = [("rows", 3, 40), ("rows", 1, 65), ("flat", 2, 2 + 40 * 96), ("flat", 1, 1 + 64 * 96)]


def reshaped_slice(M, x, kind, start, end):
    """sum(y * y) of a reshaped slice, and what its gradient is: twice the slice, zeros around it."""
    v = M[0](x)
    y = M[2](M[1](v, 0, start, end), [(end - start) // 2 if (end - start) % 2 == 0 else end - start, -1]) if kind == "rows" else M[2](M[1](M[2](v, [x.size]), 0, start, end), [-1, 96])
    want = np.zeros(x.size, np.float32)
    lo, hi = (start * x.shape[1], end * x.shape[1]) if kind == "rows" else (start, end)
    want[lo:hi] = 2 * x.reshape(-1)[lo:hi]
    return v, y, want.reshape(x.shape)


@pytest.mark.parametrize("kind,start,end", RESHAPED_SLICES)
def test_gradients_of_reshaped_slices_in_the_oracle(kind, start, end):
    from oracle import sage_ref as R
    x = np.random.default_rng(start).standard_normal((70, 96)).astype(np.float32)
    v, y, want = reshaped_slice((lambda a: R.Var.new(R.Tensor.new(a)), R.slice_, R.view), x, kind, start, end)
    assert np.array_equal(R.evaluate([v.grad(R.sum_(y * y, [0, 1]))])[0].numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("fusion", [0, 1])
@pytest.mark.parametrize("kind,start,end", RESHAPED_SLICES)
def test_gradients_of_reshaped_slices(kind, start, end, fusion):
    """The gradient starts where it starts, not where the slice does; also of a slice that a product reads (as a matrix of its own)."""
    rng = np.random.default_rng(start)
    x = rng.standard_normal((70, 96)).astype(np.float32)
    c = S.Context(0, pattern_fusion=fusion)
    try:
        v, y, want = reshaped_slice((c.var, lambda a, axis, lo, hi: a.slice(axis, lo, hi), S.view), x, kind, start, end)
        got = v.grad((y * y).sum([0, 1], False)).eval(c)
        assert np.array_equal(got.reshape(x.shape), want)
        if kind == "rows":
            w = rng.standard_normal((96, 64)).astype(np.float32)
            got = v.grad(v.slice(0, start, end).matmul(c.var(w)).sum([0, 1], False)).eval(c).reshape(x.shape)
            row = w.astype(np.float64).sum(1)
            assert not got[:start].any() and not got[end:].any()
            assert (np.abs(got[start:end] - row) <= 2.0 ** -19 * np.abs(w).sum(1)).all()
        assert c.status_word() == 0
    finally:
        c.close()
