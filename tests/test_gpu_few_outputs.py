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


@pytest.fixture
def verbose(monkeypatch):
    monkeypatch.setenv("SAGE_VERBOSE_NAMES", "1")  # the launch list tells the kernels apart


@pytest.mark.parametrize("is_max", [False, True])
@pytest.mark.usefixtures("verbose")
def test_pooling_of_what_is_not_finite(is_max):
    """Infinities and nan in one tap each, of their own windows and channels: a sum passes them on, a maximum takes +infinity and passes
    over -infinity and nan (fmaxf), as the ordinary kernel does, which the same windows over more pictures take."""
    rng = np.random.default_rng(8)
    x = rng.standard_normal((1, 7, 7, 128)).astype(np.float32)
    x[0, 1, 2, 3], x[0, 6, 6, 64], x[0, 0, 5, 127], x[0, 3, 3, 9], x[0, 4, 3, 9] = np.inf, -np.inf, np.nan, np.inf, -np.inf
    ctx = S.Context(0)
    try:
        got = []
        for n in (1, 400):
            ctx.trace_begin()
            got.append((S.max_pool_2d if is_max else S.avg_pool_2d)(ctx.var(np.repeat(x, n, 0)), 7, 1, 0, 1).eval(ctx)[0].reshape(128).copy())
            assert ctx.trace()[-1].endswith("[window]") == (n == 1)
            ctx.clear()
    finally:
        ctx.close()
    with np.errstate(invalid="ignore"):
        want = np.fmax(np.fmax.reduce(x.reshape(49, 128), 0), 0) if is_max else x.reshape(49, 128).astype(np.float64).mean(0)
    for g in got:
        if is_max:
            assert np.array_equal(g, want)
        else:
            odd = ~np.isfinite(want)
            assert odd.sum() == 4 and np.array_equal(g[odd], want[odd], equal_nan=True)
            assert (np.abs(g[~odd] - want[~odd]) <= 49 * 2.0 ** -24 * np.abs(x.reshape(49, 128)).mean(0)[~odd]).all()
