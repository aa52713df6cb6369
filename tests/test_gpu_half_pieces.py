"""The product over two half-precision pieces per operand (kernels/gemm_h2_device.inc) at the edges of its tiles, its 64-k
groups and its representation, through the op-level entry point.

Bound, elementwise against float64, with S = |A| |B|: the pieces of both operands are within 2^-23 of an element that lies
within 2^-29 of its group's largest (2 x 2^-23 S), the dropped lo x lo term adds 2^-24 S, a chain of 12 truncating additions
at most 12 x 2^-23 S, and the sum of the K / 64 chains in fp32 (K / 64 + 2) x 2^-24 S.
"""
import ctypes

import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu
L = ctypes.c_int64


@pytest.fixture(scope="module")
def ctx():
    c = S.Context(0)
    yield c
    c.close()


def product(ctx, a, b, ta=False, tb=False):
    """a, b: [batch, rows, cols] as stored."""
    n_b, m, k = a.shape[0], a.shape[2 if ta else 1], a.shape[1 if ta else 2]
    n = b.shape[1 if tb else 2]
    A, B, C = ctx.tensor(a), ctx.tensor(b), ctx.empty((n_b, m, n))
    ctx._ck(S.lib.sage_gemm_strided_batched(ctx.h, int(ta), int(tb), L(m), L(n), L(k), A.buf, L(0), L(a.shape[2]), L(m * k), B.buf, L(0), L(b.shape[2]), L(k * n),
                                            C.buf, L(0), L(n), L(m * n), L(n_b)))
    out = C.numpy()
    for t in (A, B, C):
        t.release()
    return out


def excess(got, a, b, floor=0.0):
    """Largest |got - a b| over its bound; `floor`: an absolute error per unit of the other operand's column sums."""
    a, b = a.astype(np.float64), b.astype(np.float64)
    k = a.shape[-1]
    s = np.abs(a) @ np.abs(b)
    bound = s * (2.0 ** -22 + 2.0 ** -24 + 12 * 2.0 ** -23 + (k / 64 + 2) * 2.0 ** -24) + floor
    return float((np.abs(got - a @ b) / np.maximum(bound, 1e-300)).max())


@pytest.mark.parametrize("m,n,k", [(64, 32, 32), (128, 64, 63), (129, 65, 64), (256, 256, 65), (257, 193, 128), (300, 448, 190), (512, 640, 1000),
                                   (1000, 2050, 257), (2500, 1600, 96), (64, 4096, 130), (320, 64, 6400)])
def test_edges_of_tiles_and_groups(ctx, m, n, k):
    rng = np.random.default_rng(m * 31 + n * 7 + k)
    a, b = rng.standard_normal((1, m, k), dtype=np.float32), rng.standard_normal((1, k, n), dtype=np.float32)
    assert excess(product(ctx, a, b), a, b) <= 1.0
    assert ctx.status_word() == 0


@pytest.mark.parametrize("ta,tb", [(False, True), (True, False), (True, True)])
@pytest.mark.parametrize("batch,m,n,k", [(1, 200, 132, 76), (3, 130, 68, 260), (2, 77, 301, 133)])
def test_transposed_and_batched_operands(ctx, ta, tb, batch, m, n, k):
    rng = np.random.default_rng(900 + m)
    a = rng.standard_normal((batch, k, m) if ta else (batch, m, k), dtype=np.float32)
    b = rng.standard_normal((batch, n, k) if tb else (batch, k, n), dtype=np.float32)
    got = product(ctx, a, b, ta, tb)
    assert excess(got, np.swapaxes(a, 1, 2) if ta else a, np.swapaxes(b, 1, 2) if tb else b) <= 1.0


@pytest.mark.parametrize("ea,eb", [(100, -100), (-90, 90), (120, 0), (0, 120), (-90, 20)])
def test_operands_far_from_one(ctx, ea, eb):
    """Whole operands scaled by powers of two give the scaled product, bit for bit, for rows of A above 2^-96."""
    rng = np.random.default_rng(77)
    a, b = rng.uniform(0.5, 1.0, (1, 192, 200)).astype(np.float32), rng.uniform(0.5, 1.0, (1, 200, 128)).astype(np.float32)
    plain = product(ctx, a, b).astype(np.float64)
    got = product(ctx, np.ldexp(a, ea), np.ldexp(b, eb)).astype(np.float64)
    assert np.isfinite(got).all()
    assert np.array_equal(got, np.ldexp(plain, ea + eb))


def test_wide_range_inside_a_group(ctx):
    """Elements far below their group's largest: relative accuracy down to 2^-29 of it, below that an absolute error of at
    most 2^-50 of it."""
    rng = np.random.default_rng(78)
    m, n, k = 130, 70, 192
    a = rng.standard_normal((1, m, k)).astype(np.float32)
    a *= np.ldexp(1.0, -rng.integers(0, 28, a.shape)).astype(np.float32)
    b = rng.standard_normal((1, k, n)).astype(np.float32)
    assert excess(product(ctx, a, b), a, b) <= 1.0
    a[:, :, 64:128] = np.ldexp(rng.uniform(0.5, 1, (1, m, 64)), -45)
    a[:, :, 64] = 1.0
    b[:, 64, :] = 0.0   # the large elements multiply zeros: only the small ones are left of the middle group
    a[:, :, :64] = 0.0
    a[:, :, 128:] = 0.0
    assert excess(product(ctx, a, b), a, b, floor=2.0 ** -50 * np.abs(b).sum(1, keepdims=True)) <= 1.0


def test_infinities_and_nan_stay_in_their_rows(ctx):
    rng = np.random.default_rng(79)
    a, b = rng.uniform(0.5, 1, (1, 140, 128)).astype(np.float32), rng.uniform(0.5, 1, (1, 128, 96)).astype(np.float32)
    a[0, 3, 70] = np.nan
    a[0, 5, 10] = np.inf
    got = product(ctx, a, b)[0]
    assert np.isnan(got[3]).all() and not np.isfinite(got[5]).any()
    rest = [i for i in range(140) if i not in (3, 5)]
    assert np.isfinite(got[rest]).all()
    assert ctx.status_word() == 0
