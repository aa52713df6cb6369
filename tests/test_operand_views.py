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
