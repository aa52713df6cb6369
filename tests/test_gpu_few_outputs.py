"""Kernels for few outputs: products of a warp or a lane per output (kernels/gemm_simt.cu), pooling whose windows are shared between threads
(kernels/conv.cu)."""
import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu


# fewer k than a round of loads and one more than two; columns of one block, cut, and of several; both orders of each operand
@pytest.mark.parametrize("m,n,k", [(1, 1000, 512), (32, 2, 768), (1, 2, 1024), (3, 33, 129), (7, 32, 255), (128, 10, 512), (16, 100, 257), (1, 8192, 128)])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
def test_products_of_few_outputs(m, n, k, ta, tb):
    """Within (k / 8 + 16) 2^-24 of |a| |b|: a lane's share of the terms, and the sums that meet."""
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    ctx = S.Context(0)
    try:
        x, y = ctx.var(np.ascontiguousarray(a.T) if ta else a), ctx.var(np.ascontiguousarray(b.T) if tb else b)
        got = S.gemm(x, y, ta, tb).eval(ctx) if hasattr(S, "gemm") else (S.transpose(x, 1, 0) if ta else x).matmul(S.transpose(y, 1, 0) if tb else y).eval(ctx)
        assert ctx.status_word() == 0
    finally:
        ctx.close()
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    assert (np.abs(got - a64 @ b64) <= (k / 8 + 16) * 2.0 ** -24 * (np.abs(a64) @ np.abs(b64))).all()


@pytest.mark.parametrize("shape,ker,stride,pad", [((1, 7, 7, 512), 7, 1, 0), ((2, 9, 8, 36), 4, 2, 1), ((1, 20, 20, 68), 9, 6, 3), ((3, 5, 5, 64), 5, 1, 2)])
@pytest.mark.parametrize("is_max", [False, True])
def test_pooling_of_large_windows(shape, ker, stride, pad, is_max):
    """Taps outside count as 0 (im2col's zeros); a mean within taps x 2^-24 of the mean of magnitudes."""
    rng = np.random.default_rng(ker)
    x = rng.standard_normal(shape).astype(np.float32)
    ctx = S.Context(0)
    try:
        v = (S.max_pool_2d if is_max else S.avg_pool_2d)(ctx.var(x), ker, stride, pad, 1)
        got = v.eval(ctx)
    finally:
        ctx.close()
    big = np.zeros((shape[0], shape[1] + 2 * pad, shape[2] + 2 * pad, shape[3]))
    big[:, pad:pad + shape[1], pad:pad + shape[2]] = x
    oh, ow = (shape[1] + 2 * pad - ker) // stride + 1, (shape[2] + 2 * pad - ker) // stride + 1
    taps = np.stack([big[:, ky:ky + stride * oh:stride, kx:kx + stride * ow:stride][:, :oh, :ow] for ky in range(ker) for kx in range(ker)])
    got = got.reshape(shape[0], oh, ow, shape[3])
    if is_max:
        assert np.array_equal(got, np.maximum(taps.max(0), 0).astype(np.float32))  # (the reference's accumulator starts at 0)
    else:
        assert (np.abs(got - taps.mean(0)) <= ker * ker * 2.0 ** -24 * np.abs(taps).mean(0) + 1e-30).all()
