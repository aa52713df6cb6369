"""Copies that operators keep between passes, on the host side (a planning context: launches are recorded, nothing is computed)."""
import numpy as np
import pytest

import sage_b200 as S


@pytest.fixture()
def ctx():
    c = S.Context(-1)
    yield c
    c.close()


def launches(ctx, y, name):
    ctx.clear()
    ctx.trace_begin()
    ctx.eval(y)
    return ctx.trace().count(name)


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("computed", [True, False])
def test_a_computed_filter_is_packed_on_every_pass(ctx, stride, computed):
    """The packed form of a first convolution's filter belongs to the values it was made from: a filter that is computed anew on
    every pass is packed anew, wherever its memory comes from; one that stays is packed once."""
    x, f, m = ctx.var(np.zeros((2, 64, 64, 3), np.float32)), ctx.var(np.zeros((7, 7, 3, 64), np.float32)), ctx.var(np.zeros((64,), np.float32))
    y = S.conv_2d(x, f * m if computed else f, stride, 3, 1)
    assert [launches(ctx, y, "pack_small_c_filter") for _ in range(12)] == [1] + [int(computed)] * 11


def replace(ctx, v):
    """Two new tensors one after the other: a variable whose tensor something else holds gets another one when it is assigned."""
    for _ in range(2):
        ctx.clear()
        ctx.eval(S.view(v, [-1]))
        ctx.set(v, np.zeros(v.extents, np.float32))


def test_a_replaced_filter_is_packed_again(ctx):
    x, f = ctx.var(np.zeros((2, 64, 64, 3), np.float32)), ctx.var(np.zeros((7, 7, 3, 64), np.float32))
    y = S.conv_2d(x, f, 2, 3, 1)
    for _ in range(6):
        replace(ctx, f)
        assert launches(ctx, y, "pack_small_c_filter") == 1


@pytest.mark.parametrize("k", [128, 96])
def test_replaced_weights_of_grouped_products_are_copied_again(ctx, k):
    """Three products of one operand run as one launch over a joint copy of their weights, in half-precision pieces (k in whole
    groups of 64, an operand made by a kernel that writes them) or as tf32 planes."""
    x = ctx.var(np.zeros((2, 64, k), np.float32)) * 2.0
    w = [ctx.var(np.zeros((k, k), np.float32)) for _ in range(3)]
    b = [ctx.var(np.zeros((k,), np.float32)) for _ in range(3)]
    a = S.layer_norm(x, [2], ctx.var(np.ones(1, np.float32)), ctx.var(np.zeros(1, np.float32)), 1e-5)
    q, key, v = [S.transpose(S.view(S.matmul(a, w[i]) + b[i], [2, 64, 2, k // 2]), 2, 1) for i in range(3)]
    y = S.matmul_batched(S.softmax(S.matmul_batched(q, S.transpose(key, -1, -2)), [3]), v)
    first = launches(ctx, y, "split_tf32")
    assert "gemm_grouped" in ctx.describe() and first >= 3 and launches(ctx, y, "split_tf32") == first - 3
    for _ in range(6):
        for v in w:
            replace(ctx, v)
        assert launches(ctx, y, "split_tf32") == first
