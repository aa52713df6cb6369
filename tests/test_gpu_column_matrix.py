"""The explicit column matrix of a convolution (graph/ops_conv.cc: Im2colOp) with its tf32 planes: alone where products are its only
readers, beside the fp32 values where anything else reads it."""
import numpy as np
import pytest

import sage_b200 as S


def _weight_gradient(ctx, x, g):
    col = S.im2col(ctx.var(x), 3, 1, 1, 1)
    pixels, k = x.shape[0] * x.shape[1] * x.shape[2], 9 * x.shape[3]
    return col, S.gemm(S.view(col, [pixels, k]), ctx.var(g), True, False)


def _context(device):
    with pytest.MonkeyPatch.context() as m:
        m.setenv("SAGE_VERBOSE_NAMES", "1")
        return S.Context(device)


def test_forms_that_are_written():
    x, g = np.zeros((2, 20, 20, 64), np.float32), np.zeros((800, 96), np.float32)
    ctx = _context(-1)
    try:
        for second, name in ((False, "im2col=planes"), (True, "im2col+planes")):
            col, p = _weight_gradient(ctx, x, g)
            ctx.trace_begin()
            ctx.eval(*([p, col * 2.0] if second else [p]))
            assert [n for n in ctx.trace() if n.startswith("im2col")] == [name] and name + "(" in ctx.describe()
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,hw,c", [(2, 20, 64), (1, 9, 4), (3, 7, 12)])
def test_readers_of_a_column_matrix(n, hw, c):
    """The product by itself, and beside a map of the matrix: the same bits; the map's exactly.  Product: 22 bits of an operand (two
    planes) and sums of up to 48 truncated terms and then fp32, 64 x 2^-23 of the sum of magnitudes."""
    rng = np.random.default_rng(hw)
    x, g = rng.standard_normal((n, hw, hw, c), dtype=np.float32), rng.standard_normal((n * hw * hw, 96), dtype=np.float32)
    pad = np.pad(x, ((0, 0), (1, 1), (1, 1), (0, 0)))
    want = np.stack([np.stack([pad[:, i:i + hw, j:j + hw] for j in range(3)], 3) for i in range(3)], 3)  # [n, h, w, kh, kw, c]
    a = want.reshape(n * hw * hw, -1).astype(np.float64)
    ctx = _context(0)
    try:
        col, p = _weight_gradient(ctx, x, g)
        alone = p.eval(ctx)
        assert (np.abs(alone - a.T @ g) <= 64 * 2.0 ** -23 * (np.abs(a).T @ np.abs(g).astype(np.float64))).all()
        ctx.clear()
        twice = col * 2.0
        ctx.eval(p, twice)
        assert np.array_equal(ctx.read(p), alone) and np.array_equal(ctx.read(twice).reshape(want.shape), 2 * want)
        assert ctx.status_word() == 0
    finally:
        ctx.close()
