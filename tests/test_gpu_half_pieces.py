"""The product over two half-precision pieces per operand (kernels/gemm_h2_device.inc) at the edges of its tiles, its 64-k
groups and its representation, through the op-level entry point.

Bound, elementwise against float64, with S = |A| |B|: the pieces of both operands are within 2^-23 of an element that lies
within 2^-29 of its group's largest (2 x 2^-23 S), the dropped lo x lo term adds 2^-24 S, a chain of 12 truncating additions
at most 12 x 2^-23 S, and the sum of the K / 64 chains in fp32 (K / 64 + 2) x 2^-24 S.
"""
import ctypes
import re

import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu
L = ctypes.c_int64


@pytest.fixture(scope="module")
def ctx():
    """A context whose launch list tells the kernels apart (the plain list has one name for every tensor-core product)."""
    with pytest.MonkeyPatch.context() as m:
        m.setenv("SAGE_VERBOSE_NAMES", "1")
        c = S.Context(0)
    yield c
    c.close()


def evaluated(ctx, y, pattern, count=1, splits=None):
    """The value of y, whose evaluation launched at least `count` kernels of names that `pattern` finds, and `splits` passes that
    only split an operand."""
    ctx.trace_begin()
    ctx.eval(y)
    names = ctx.trace()
    assert sum(bool(re.search(pattern, n)) for n in names) >= count, (pattern, names)
    assert splits is None or names.count("split_h2") == splits, names
    return ctx.read(y)


def product(ctx, a, b, ta=False, tb=False):
    """a, b: [batch, rows, cols] as stored."""
    n_b, m, k = a.shape[0], a.shape[2 if ta else 1], a.shape[1 if ta else 2]
    n = b.shape[1 if tb else 2]
    A, B, C = ctx.tensor(a), ctx.tensor(b), ctx.empty((n_b, m, n))
    ctx.trace_begin()
    ctx._ck(S.lib.sage_gemm_strided_batched(ctx.h, int(ta), int(tb), L(m), L(n), L(k), A.buf, L(0), L(a.shape[2]), L(m * k), B.buf, L(0), L(b.shape[2]), L(k * n),
                                            C.buf, L(0), L(n), L(m * n), L(n_b)))
    names = ctx.trace()
    assert names[:-1] == ["split_h2"] * 2 and names[-1].startswith("gemm_tc_h2["), names
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


# How operand B is read: single elements along K and across it, 16 bytes of one row, of four; one to five tiles of 64 k a CTA, the last
# one cut; K beyond 2^15, where tiles share a factor.  Operand A's blocks of one tile and of several.
@pytest.mark.parametrize("tb,n,k", [(True, 67, 1985), (True, 68, 1984), (False, 67, 1985), (False, 68, 1985), (True, 96, 1028), (False, 132, 520), (True, 33, 2561), (False, 64, 33000),
                                    (True, 64, 33000), (True, 40, 33001)])
@pytest.mark.parametrize("m", [70, 2500])
def test_splits_of_operands(ctx, tb, n, k, m):
    rng = np.random.default_rng(n + k)
    if k > 30000 and m > 70:
        pytest.skip("one size of A is enough for the longest K")
    a, b = rng.standard_normal((1, m, k), dtype=np.float32), rng.standard_normal((1, n, k) if tb else (1, k, n), dtype=np.float32)
    b[0, :: 7 if tb else 1, 1::3] *= 2.0 ** -20   # rows, and tiles of them, of different ranges
    a[0, 1::5] *= 2.0 ** 18
    assert excess(product(ctx, a, b, False, tb), a, np.swapaxes(b, 1, 2) if tb else b) <= 1.0
    assert ctx.status_word() == 0


# Slices of K that meet in a cluster: one task of 8 x 64 sums for eight CTAs, fewer tasks than slices, tasks that the slices do not divide,
# a last task with one row, the last column tile cut; several tiles, a batch.
@pytest.mark.parametrize("m,n,k,batch", [(5, 1000, 4096, 1), (7, 640, 4608, 1), (9, 513, 4096, 1), (24, 192, 2304, 1), (127, 64, 1536, 1), (127, 130, 1536, 1), (128, 512, 2304, 1), (250, 300, 2304, 1),
                                         (65, 64, 1152, 3), (384, 768, 3072, 1), (768, 512, 2304, 1), (400, 512, 2048, 1)])
def test_slices_that_meet_in_a_cluster(ctx, m, n, k, batch):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((batch, m, k), dtype=np.float32), rng.standard_normal((batch, n, k), dtype=np.float32)
    got = product(ctx, a, b, False, True)
    assert ",slices" in ctx.trace()[-1], ctx.trace()
    assert excess(got, a, np.swapaxes(b, 1, 2)) <= 1.0
    assert np.array_equal(got, product(ctx, a, b, False, True))
    assert ctx.status_word() == 0


# Sums sent beside the operands, sent over them (three slices of many K-blocks), and fetched (two slices; four without a residual).
@pytest.mark.parametrize("n,hw,c,residual,how", [(8, 28, 128, True, ",fetched,slices2"), (8, 14, 256, False, ",fetched,slices4"), (8, 14, 256, True, ",over,slices4"), (24, 7, 512, True, ",over,slices3"),
                                                 (6, 28, 128, True, ",slices3"), (3, 28, 128, False, ",slices6"), (8, 7, 512, False, ",over,slices6"), (9, 14, 320, True, ",slices")])
def test_slices_of_convolutions(ctx, n, hw, c, residual, how):
    """3 x 3, bias, residual and relu behind, the result read by a second convolution.  Tolerance as for the other convolutions."""
    rng = np.random.default_rng(n + c)
    x, f = rng.uniform(-1, 1, (n, hw, hw, c)).astype(np.float32), rng.uniform(-1, 1, (3, 3, c, c)).astype(np.float32)
    b = rng.uniform(-1, 1, (c,)).astype(np.float32)
    xv, fv = ctx.var(x), ctx.var(f)
    y = S.conv_2d(xv, fv, 1, 1, 1) + ctx.var(b)
    y = S.relu(y + xv) if residual else S.relu(y)
    want = np.maximum(_conv64(x, f, 1, 1) + b + (x if residual else 0), 0.0)
    got = evaluated(ctx, y, re.escape(how))
    assert _close(got, want)
    ctx.clear()
    assert np.array_equal(got, y.eval(ctx))
    ctx.clear()
    z = S.conv_2d(y, ctx.var(f[:, :, :, :64].copy()), 1, 1, 1)
    assert _close(z.eval(ctx), _conv64(want, f[:, :, :, :64], 1, 1))
    assert ctx.status_word() == 0


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


@pytest.mark.parametrize("m,k,n1,n2", [(129, 128, 64, 70), (300, 192, 192, 64), (2048, 64, 448, 96), (12544, 64, 512, 64), (70, 4096, 128, 33)])
def test_a_product_hands_pieces_to_the_next(ctx, m, k, n1, n2):
    """The first product's result exists only as pieces (with its epilogue applied, K slices summed where it has them); every
    group of it lands in its place, also where the last column tile is cut off.  Tolerance: 1e-5 of max(|b|, rms), as for the
    other products behind an epilogue."""
    rng = np.random.default_rng(m + n1)
    x, w1 = rng.uniform(-1, 1, (m, k)).astype(np.float32), rng.uniform(-1, 1, (k, n1)).astype(np.float32)
    b, w2 = rng.uniform(-1, 1, (n1,)).astype(np.float32), rng.uniform(-1, 1, (n1, n2)).astype(np.float32)
    y = S.matmul(S.relu(S.matmul(ctx.var(x) * 1.0, ctx.var(w1)) + ctx.var(b)), ctx.var(w2))
    got = evaluated(ctx, y, r"^gemm_tc_h2\[", 2, splits=2).astype(np.float64)  # (the weights)
    want = np.maximum(x.astype(np.float64) @ w1 + b, 0.0) @ w2.astype(np.float64)
    assert (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-5
    assert ctx.status_word() == 0


@pytest.mark.parametrize("n,h,c,oc,ker,stride", [(7, 9, 64, 64, 3, 1), (3, 17, 64, 192, 3, 2), (6, 7, 512, 128, 3, 1), (33, 8, 128, 64, 1, 2), (1, 56, 64, 64, 3, 1)])
def test_convolutions_on_pieces(ctx, n, h, c, oc, ker, stride):
    """Two convolutions in a row (windows kept in shared memory, gathered, cut into K slices), the second over the first's pieces."""
    rng = np.random.default_rng(h * c)
    x = rng.uniform(-1, 1, (n, h, h, c)).astype(np.float32)
    f1, f2 = rng.uniform(-1, 1, (ker, ker, c, oc)).astype(np.float32), rng.uniform(-1, 1, (3, 3, oc, 64)).astype(np.float32)
    b = rng.uniform(-1, 1, (oc,)).astype(np.float32)

    def conv(a, f, s):
        k, p = f.shape[0], f.shape[0] // 2
        a = np.pad(a.astype(np.float64), ((0, 0), (p, p), (p, p), (0, 0)))
        o = (a.shape[1] - k) // s + 1
        return sum(a[:, i:i + s * o:s, j:j + s * o:s][:, :o, :o] @ f[i, j].astype(np.float64) for i in range(k) for j in range(k))
    y = S.relu(S.conv_2d(ctx.var(x) * 1.0, ctx.var(f1), stride, ker // 2, 1) + ctx.var(b))
    got = evaluated(ctx, S.conv_2d(y, ctx.var(f2), 1, 1, 1), r"^gemm_tc_h2\[.*,conv", 2, splits=2).astype(np.float64)  # (the filters)
    want = conv(np.maximum(conv(x, f1, stride) + b, 0.0), f2, 1)
    assert got.shape == want.shape
    assert (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-5
    assert ctx.status_word() == 0


def test_epilogue_operands_off_the_16_byte_grid(ctx):
    """A result in pieces behind operands that 16-byte loads cannot read (a slice that starts off the grid; an odd row pitch)."""
    rng = np.random.default_rng(81)
    x, w1 = rng.uniform(-1, 1, (150, 64)).astype(np.float32), rng.uniform(-1, 1, (64, 128)).astype(np.float32)
    r, w2 = rng.uniform(-1, 1, (150, 131)).astype(np.float32), rng.uniform(-1, 1, (128, 64)).astype(np.float32)
    y = S.matmul(S.relu(S.matmul(ctx.var(x) * 1.0, ctx.var(w1)) + ctx.var(r).slice(1, 1, 129)), ctx.var(w2))
    got = evaluated(ctx, y, r"^gemm_tc_h2\[", 2, splits=2).astype(np.float64)
    want = np.maximum(x.astype(np.float64) @ w1 + r[:, 1:129], 0.0) @ w2.astype(np.float64)
    assert (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-5


@pytest.mark.parametrize("n,length,heads,direct", [(3, 77, 4, True), (2, 130, 2, False), (1, 64, 1, True), (2, 257, 3, False)])
def test_attention_hands_pieces_to_the_next(ctx, n, length, heads, direct):
    """Masked attention over any number of keys, its context multiplied by a weight; queries, keys and values straight from
    products or behind a sum.  Tolerance 1e-4, as for the other attention blocks."""
    rng = np.random.default_rng(length)
    e = heads * 64
    x = rng.uniform(-1, 1, (n, length, e)).astype(np.float32)
    w = [(rng.standard_normal((e, e)) / np.sqrt(e)).astype(np.float32) for _ in range(4)]
    mask = (rng.random((n, length)) < 0.8).astype(np.float32)
    mask[:, 0] = 1
    X = ctx.var(x) * 1.0
    q, k, v = [S.matmul(X, ctx.var(w[i])) + (0.0 if direct else X) for i in range(3)]

    def split(t):
        return S.transpose(S.view(t, [n, length, heads, 64]), 2, 1)
    s = S.matmul_batched(split(q), S.transpose(split(k), -1, -2)) / 8.0 + (-(S.view(ctx.var(mask), [n, 1, 1, length])) + 1.0) * -1e5
    y = S.view(S.transpose(S.matmul_batched(S.softmax(s, [3]), split(v)), 2, 1), [n, length, e])
    got = evaluated(ctx, S.matmul(y, ctx.var(w[3])), r"^(attention|gemm)_tc_h2\[", 3, splits=4 if direct else None).astype(np.float64)
    x64 = x.astype(np.float64)
    q, k, v = [(x64 @ w[i] + (0.0 if direct else x64)).reshape(n, length, heads, 64).transpose(0, 2, 1, 3) for i in range(3)]
    s = q @ k.transpose(0, 1, 3, 2) / 8.0 + (1.0 - mask.astype(np.float64))[:, None, None, :] * -1e5
    p = np.exp(s - s.max(-1, keepdims=True))
    want = ((p / p.sum(-1, keepdims=True)) @ v).transpose(0, 2, 1, 3).reshape(n, length, e) @ w[3].astype(np.float64)
    assert (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-4
    assert ctx.status_word() == 0


@pytest.mark.parametrize("shape,ker,stride,pad,is_max", [((13, 11, 13, 64), 3, 2, 1, True), ((17, 9, 9, 128), 2, 2, 0, False), ((11, 20, 20, 64), 5, 3, 2, True), ((5, 12, 12, 192), 3, 1, 1, False)])
def test_pooling_hands_pieces_to_a_convolution(ctx, shape, ker, stride, pad, is_max):
    """Windows of more and fewer taps than are fetched at a time, cut at the image's edge; the convolution behind reads the
    pool's pieces.  Tolerance as for the other convolutions."""
    rng = np.random.default_rng(sum(shape))
    x = rng.uniform(-1, 1, shape).astype(np.float32)
    f = rng.uniform(-1, 1, (3, 3, shape[3], 64)).astype(np.float32)
    pool = S.max_pool_2d if is_max else S.avg_pool_2d
    p = pool(ctx.var(x) * 1.0, ker, stride, pad, 1)
    alone = p.eval(ctx)
    ctx.clear()
    got = evaluated(ctx, S.conv_2d(p, ctx.var(f), 1, 1, 1), r"^gemm_tc_h2\[.*,conv", splits=1).astype(np.float64)  # (the filter)

    def windows(a, k, s, q):
        a = np.pad(a.astype(np.float64), ((0, 0), (q, q), (q, q), (0, 0)))
        oh, ow = (a.shape[1] - k) // s + 1, (a.shape[2] - k) // s + 1
        return [[a[:, i:i + s * oh:s, j:j + s * ow:s][:, :oh, :ow] for j in range(k)] for i in range(k)]
    taps = np.stack([t for r in windows(x, ker, stride, pad) for t in r])
    want = np.maximum(taps.max(0), 0) if is_max else taps.mean(0)
    assert np.abs(alone - want).max() <= 1e-6 * ker * ker
    w = windows(alone, 3, 1, 1)
    want = sum(w[i][j] @ f[i, j].astype(np.float64) for i in range(3) for j in range(3))
    assert (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-5


@pytest.mark.parametrize("n,length,heads,keyed", [(10, 257, 12, True), (75, 200, 2, False), (37, 512, 2, True)])
def test_attention_with_a_thread_per_row(ctx, n, length, heads, keyed):
    """Enough tiles of more than three key blocks for the form with a thread per query row: a last tile of one row, a last block
    of eight keys, tiles that follow one another in a CTA; with and without an operand of the scores.  Tolerance 1e-4, as for the
    other attention blocks."""
    rng = np.random.default_rng(length + n)
    q, k, v = [rng.uniform(-2, 2, (n, heads, length, 64)).astype(np.float32) for _ in range(3)]
    bias = rng.uniform(-3, 3, (n, length)).astype(np.float32)
    s = S.matmul_batched(ctx.var(q), S.transpose(ctx.var(k), -1, -2)) / 8.0
    if keyed:
        s = s + S.view(ctx.var(bias), [n, 1, 1, length])
    got = evaluated(ctx, S.matmul_batched(S.softmax(s, [3]), ctx.var(v)), r"^attention_tc_h2\[.*,rows")
    for i in range(0, n, max(n // 4, 1)):
        s = q[i].astype(np.float64) @ k[i].astype(np.float64).transpose(0, 2, 1) / 8.0 + (bias[i] if keyed else 0.0)
        p = np.exp(s - s.max(-1, keepdims=True))
        want = (p / p.sum(-1, keepdims=True)) @ v[i].astype(np.float64)
        assert (np.abs(got[i] - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-4
    assert ctx.status_word() == 0


@pytest.mark.parametrize("n,heads,length", [(5, 2, 77), (5, 1, 200), (5, 30, 257)])
def test_attention_over_scores_far_below_zero(monkeypatch, n, heads, length):
    """Every score of a sequence shifted by the same amount, as a mask on the whole sequence does: the quotient is unchanged
    whichever maximum is subtracted, also where the reference's reduce starts at 0 (ref_compat = 1) and exp(x - 0) lies far below
    what half-precision pieces of a weight near 1 hold.  Both forms of the kernel.  Per row, relative to the row's rms: 1e-4, as
    for the other attention blocks.  A row whose every exp(x) is 0 in fp32 is 0 / 0 under ref_compat, as in the reference."""
    monkeypatch.setenv("SAGE_VERBOSE_NAMES", "1")
    rng = np.random.default_rng(length)
    q, k, v = [rng.uniform(-1, 1, (n, heads, length, 64)).astype(np.float32) for _ in range(3)]
    shift = np.array([-20, -30, -40, -80, -150], np.float32)
    q64, k64, v64 = [t.astype(np.float64) for t in (q, k, v)]
    s = q64 @ k64.transpose(0, 1, 3, 2) / 8.0
    p = np.exp(s - s.max(-1, keepdims=True))
    want = (p / p.sum(-1, keepdims=True)) @ v64
    for compat in (1, 0):
        c = S.Context(0, ref_compat=compat)
        try:
            sc = S.matmul_batched(c.var(q), S.transpose(c.var(k), -1, -2)) / 8.0 + S.view(c.var(shift), [n, 1, 1, 1])
            got = evaluated(c, S.matmul_batched(S.softmax(sc, [3]), c.var(v)), r"^attention_tc_h2\[.*,rows" if heads == 30 else r"^attention_tc_h2\[[0-9x]*\]").astype(np.float64)
            assert c.status_word() == 0
        finally:
            c.close()
        if compat:
            assert np.isnan(got[4]).all()
        rows = slice(0, 4 if compat else 5)
        err = np.abs(got - want) / np.sqrt((want ** 2).mean(-1, keepdims=True))
        assert np.nanmax(err[rows]) <= 1e-4 and not np.isnan(err[rows]).any(), [float(e.max()) for e in err]


@pytest.mark.parametrize("compat", [1, 0])
def test_attention_whose_first_keys_are_masked_with_infinity(compat):
    """More than one block of keys at -inf before the first finite score: their weights are 0, not exp(-inf + inf)."""
    rng = np.random.default_rng(83)
    n, heads, length = 2, 2, 300
    q, k, v = [rng.uniform(-1, 1, (n, heads, length, 64)).astype(np.float32) for _ in range(3)]
    bias = np.zeros((n, length), np.float32)
    bias[:, :140] = -np.inf
    c = S.Context(0, ref_compat=compat)
    try:
        sc = S.matmul_batched(c.var(q), S.transpose(c.var(k), -1, -2)) / 8.0 + S.view(c.var(bias), [n, 1, 1, length])
        got = S.matmul_batched(S.softmax(sc, [3]), c.var(v)).eval(c).astype(np.float64)
        assert "attention" in c.describe() and c.status_word() == 0
    finally:
        c.close()
    s = q.astype(np.float64) @ k[:, :, 140:].astype(np.float64).transpose(0, 1, 3, 2) / 8.0
    p = np.exp(s - s.max(-1, keepdims=True))
    want = (p / p.sum(-1, keepdims=True)) @ v[:, :, 140:].astype(np.float64)
    assert (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-4


def _conv64(x, f, stride, pad):
    x = np.pad(x.astype(np.float64), ((0, 0), (pad, pad), (pad, pad), (0, 0)))
    k = f.shape[0]
    oh, ow = (x.shape[1] - k) // stride + 1, (x.shape[2] - k) // stride + 1
    return sum(x[:, i:i + stride * (oh - 1) + 1:stride, j:j + stride * (ow - 1) + 1:stride] @ f[i, j].astype(np.float64) for i in range(k) for j in range(k))


def _close(got, want, tol=1e-5):
    return (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= tol


# One picture in one tile (cut into K slices); several pictures a tile, the last tile not full; rows of a picture in tiles, the last
# with fewer; pixels two apart, with and without a window; dilated taps; rows of the longest a tile takes.
@pytest.mark.parametrize("n,h,w,c,oc,ker,stride,dil", [(1, 7, 7, 512, 512, 3, 1, 1), (17, 2, 2, 512, 128, 3, 1, 1), (20, 5, 5, 64, 64, 3, 2, 1), (30, 4, 4, 64, 200, 1, 1, 1),
                                                       (1, 16, 16, 64, 320, 3, 1, 1), (1, 20, 23, 64, 192, 3, 1, 1), (2, 15, 11, 64, 256, 1, 2, 1), (1, 12, 12, 192, 160, 3, 1, 2),
                                                       (1, 3, 128, 64, 136, 3, 1, 1), (70, 2, 2, 64, 64, 1, 2, 1)])
def test_convolutions_of_images_below_128_kib(ctx, n, h, w, c, oc, ker, stride, dil):
    """Small images are read through tiled boxes: bias and relu behind, the result handed to a second convolution.  Tolerance as for
    the other convolutions."""
    rng = np.random.default_rng(h * w + c)
    x, f = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32), rng.uniform(-1, 1, (ker, ker, c, oc)).astype(np.float32)
    b = rng.uniform(-1, 1, (oc,)).astype(np.float32)
    wide = np.zeros((dil * (ker - 1) + 1,) * 2 + f.shape[2:], np.float32)
    wide[::dil, ::dil] = f
    pad = dil * (ker // 2)
    y = S.relu(S.conv_2d(ctx.var(x) * 1.0, ctx.var(f), stride, pad, dil) + ctx.var(b))
    want = np.maximum(_conv64(x, wide, stride, pad) + b, 0.0)
    assert _close(evaluated(ctx, y, r"^gemm_tc_h2\[.*,conv"), want)
    assert "im2col" not in " ".join(ctx.trace())
    if oc % 64 == 0:
        ctx.clear()
        f2 = rng.uniform(-1, 1, (3, 3, oc, 64)).astype(np.float32)
        assert _close(evaluated(ctx, S.conv_2d(y, ctx.var(f2), 1, 1, 1), r"^gemm_tc_h2\[.*,conv", 2, splits=1), _conv64(want, f2, 1, 1))
    assert ctx.status_word() == 0


def _conv_excess(got, x, f, stride, pad):
    """Largest error over the bound at the top of the file, the chains of 16 and 4 fp32 terms of a wide group's 64 k (20 x 2^-24) with it."""
    want, s = _conv64(x, f, stride, pad), _conv64(np.abs(x), np.abs(f), stride, pad)
    bound = s * (2.0 ** -22 + 2.0 ** -24 + 12 * 2.0 ** -23 + (f[..., 0].size / 64 + 22) * 2.0 ** -24)
    return float((np.abs(got - want) / np.maximum(bound, 1e-300)).max())


def _spread(rng, n, span):
    """Powers of two over `span` binades, the ends among them."""
    e = rng.integers(0, span + 1, n)
    e[:2] = 0, span
    return (2.0 ** (span // 2 - rng.permutation(e))).astype(np.float32)


# Slices of K and none; several images a tile; a window, columns two apart, a single tap; channels that end inside a tile of columns;
# a filter whose columns are not loaded four at a time.
@pytest.mark.parametrize("span", [20, 30, 60])
@pytest.mark.parametrize("n,h,w,c,oc,ker,stride", [(1, 7, 7, 512, 512, 3, 1), (9, 5, 5, 64, 130, 3, 2), (1, 20, 23, 64, 192, 3, 1), (3, 6, 6, 192, 33, 1, 1), (1, 16, 16, 64, 64, 2, 1)])
def test_small_images_whose_channels_lie_far_apart(ctx, n, h, w, c, oc, ker, stride, span):
    """Channels of one group of 64 over up to 2^60, and a filter that makes up for it: every product counts, and keeps the bits it has in
    single precision.  As an input, as a map's result, and as views that have to be gathered."""
    rng = np.random.default_rng(span + oc)
    d = _spread(rng, c, span)
    x = (rng.uniform(0.5, 1, (n, h, w, c)) * rng.choice([-1, 0, 1], (n, h, w, c)) * d).astype(np.float32)
    f = (rng.uniform(0.5, 1, (ker, ker, c, oc)) * rng.choice([-1, 1], (ker, ker, c, oc)) / d[:, None]).astype(np.float32)
    pad = ker // 2 if ker % 2 else 0
    xv, fv = ctx.var(x), ctx.var(f)
    label = r"^gemm_tc_h2\[.*,conv,boxes"
    for y in (S.conv_2d(xv, fv, stride, pad, 1), S.conv_2d(xv * 1.0, fv, stride, pad, 1)):
        assert _conv_excess(evaluated(ctx, y, label), x, f, stride, pad) <= 1.0
        ctx.clear()
    flat = np.concatenate([np.ones(7, np.float32), x.ravel()])
    y = S.conv_2d(S.view(ctx.var(flat).slice(0, 7, 7 + x.size), list(x.shape)), fv, stride, pad, 1)
    assert _conv_excess(evaluated(ctx, y, label), x, f, stride, pad) <= 1.0
    assert ctx.status_word() == 0


def test_small_images_with_one_far_operand(ctx):
    """A channel far above the others that no filter uses, and filters that lie far apart between such channels: the small ones count."""
    rng = np.random.default_rng(7)
    x, f = rng.uniform(-1, 1, (2, 9, 9, 128)).astype(np.float32), rng.uniform(-1, 1, (3, 3, 128, 96)).astype(np.float32)
    x[..., 5] *= 2.0 ** 50
    f[:, :, 5] = 0
    assert _conv_excess(evaluated(ctx, S.conv_2d(ctx.var(x), ctx.var(f), 1, 1, 1), r"conv,boxes"), x, f, 1, 1) <= 1.0
    x[..., 5], f[:, :, 5] = 0, 2.0 ** 50
    f[..., 7] *= np.float32(2.0 ** -60)
    assert _conv_excess(evaluated(ctx, S.conv_2d(ctx.var(x), ctx.var(f), 1, 1, 1), r"conv,boxes"), x, f, 1, 1) <= 1.0
    x[0, 0, 0, 0], x[1, 3, 4, 6] = np.inf, np.nan  # ... and what is not finite stays where it belongs
    got = evaluated(ctx, S.conv_2d(ctx.var(x), ctx.var(f), 1, 1, 1), r"conv,boxes")
    want = _conv64(x, f, 1, 1)
    assert np.array_equal(np.isfinite(got), np.isfinite(want)) and not np.isfinite(got[0, 0, 0]).any()
    fin = np.isfinite(want)
    x[0, 0, 0, 0] = x[1, 3, 4, 6] = 0
    assert (np.abs(got - _conv64(x, f, 1, 1)) / np.maximum(2e-6 * _conv64(np.abs(x), np.abs(f), 1, 1), 1e-300))[fin].max() <= 1.0
    assert ctx.status_word() == 0


# The image as another convolution's result, out of slices (512 channels) and not; out of a pool; beside another reader; kept.
@pytest.mark.parametrize("c,hw,oc", [(512, 7, 64), (64, 14, 64), (64, 8, 128)])
def test_small_images_that_a_program_makes(ctx, c, hw, oc):
    """The producers of an image note its wide groups.  The second convolution against float64 of the first one's own result."""
    rng = np.random.default_rng(c + hw)
    d = _spread(rng, c, 44)
    x = rng.uniform(0, 1, (1, 2 * hw, 2 * hw, c)).astype(np.float32)
    f1 = (rng.uniform(-1, 1, (1, 1, c, c)) * d).astype(np.float32)
    f2 = (rng.uniform(-1, 1, (3, 3, c, oc)) / d[:, None]).astype(np.float32)
    xv, b = ctx.var(x), ctx.var((rng.uniform(-1, 1, (c,)) * d).astype(np.float32))
    img = S.max_pool_2d(xv * ctx.var(d), 2, 2, 0, 1)
    first = S.relu(S.conv_2d(S.max_pool_2d(xv, 2, 2, 0, 1), ctx.var(f1), 1, 0, 1) + b)
    for made in (first, img):
        z = S.conv_2d(made, ctx.var(f2), 1, 1, 1)
        alone = evaluated(ctx, z, r"conv,boxes")
        ctx.clear()
        ctx.eval(z, made)
        kept, both = ctx.read(made), ctx.read(z)
        assert _conv_excess(both, kept, f2, 1, 1) <= 1.0
        assert np.array_equal(alone, both)
        ctx.clear()
        other = S.gemm(S.view(made, [hw * hw, c]), ctx.var(f2[0, 0]))  # a reader that takes the same pieces
        ctx.eval(z, other)
        assert np.array_equal(ctx.read(z), alone)
        assert np.isfinite(ctx.read(other)).all()
        ctx.clear()
    assert ctx.status_word() == 0


@pytest.mark.parametrize("off", [0, 1, 4, 32, 64])
@pytest.mark.parametrize("tail", [0, 5])
@pytest.mark.parametrize("ker,stride", [(3, 1), (1, 2)])
def test_convolution_of_an_image_off_the_grid_of_groups(ctx, off, tail, ker, stride):
    """A part of a flat array as the image: its start may lie anywhere and its storage be of any length.  Tolerance as for the
    other convolutions."""
    rng = np.random.default_rng(off + tail)
    shape = (4, 16, 16, 64)
    n = int(np.prod(shape))
    flat = rng.uniform(-1, 1, (off + n + tail,)).astype(np.float32)
    x = flat[off:off + n].reshape(shape)
    f = rng.uniform(-1, 1, (ker, ker, 64, 64)).astype(np.float32)
    v = ctx.var(flat)
    y = S.conv_2d(S.view(v.slice(0, off, off + n), list(shape)), ctx.var(f), stride, ker // 2, 1)
    assert _close(evaluated(ctx, y, r"^gemm_tc_h2\[.*,conv"), _conv64(x, f, stride, ker // 2))
    ctx.set(v, -flat)   # the gathered copy goes with the contents
    ctx.clear()
    assert _close(y.eval(ctx), _conv64(-x, f, stride, ker // 2))
    assert ctx.status_word() == 0


@pytest.mark.parametrize("off,tail", [(4, 0), (32, 0), (0, 3), (64, 0)])
def test_convolution_entry_point_inside_a_larger_buffer(ctx, off, tail):
    rng = np.random.default_rng(84)
    x, f = rng.uniform(-1, 1, (2, 20, 20, 64)).astype(np.float32), rng.uniform(-1, 1, (3, 3, 64, 96)).astype(np.float32)
    flat = np.concatenate([np.full(off, 7, np.float32), x.ravel(), np.full(tail, 7, np.float32)])
    xt, ft, yt = ctx.tensor(flat), ctx.tensor(f), ctx.empty((2, 20, 20, 96))
    cx, cf, cy = ctx.tensor(x), ft.c(), yt.c()
    inner = cx.c()
    inner.buf, inner.offset = xt.c().buf, off
    win = S.window(1, 1, 1, 1)
    ctx._ck(S.lib.sage_conv2d_nhwc(ctx.h, ctypes.byref(inner), ctypes.byref(cf), ctypes.byref(win), ctypes.byref(cy)))
    assert _close(yt.numpy(), _conv64(x, f, 1, 1))
    for t in (xt, ft, yt, cx):
        t.release()


@pytest.mark.parametrize("off", [0, 1, 3, 4])
def test_pooling_of_an_image_off_the_16_byte_grid(ctx, off):
    """The convolution behind reads the pool's pieces where the pool writes them, and splits its result where it does not."""
    rng = np.random.default_rng(85)
    shape = (4, 30, 30, 64)
    n = int(np.prod(shape))
    flat = rng.uniform(-1, 1, (off + n,)).astype(np.float32)
    x, f = flat[off:].reshape(shape), rng.uniform(-1, 1, (3, 3, 64, 64)).astype(np.float32)
    p = S.max_pool_2d(S.view(ctx.var(flat).slice(0, off, off + n), list(shape)), 2, 2, 0, 1)
    got = evaluated(ctx, S.conv_2d(p, ctx.var(f), 1, 1, 1), r"^gemm_tc_h2\[.*,conv", splits=2 if off % 4 else 1)
    m = np.maximum(x.reshape(4, 15, 2, 15, 2, 64).max((2, 4)), 0)
    assert _close(got, _conv64(m, f, 1, 1))
    assert ctx.status_word() == 0


@pytest.mark.parametrize("off", [0, 1, 32])
def test_part_of_a_result_behind_a_reshape(ctx, off):
    """A convolution and a product over a part of another product's result that starts inside a group of 64."""
    rng = np.random.default_rng(86)
    n = 2 * 20 * 20 * 64
    a, w = rng.uniform(-1, 1, (1600, 128)).astype(np.float32), rng.uniform(-1, 1, (128, 64)).astype(np.float32)
    f, w2 = rng.uniform(-1, 1, (3, 3, 64, 64)).astype(np.float32), rng.uniform(-1, 1, (64, 128)).astype(np.float32)

    def part():
        return S.view(S.matmul(ctx.var(a) * 1.0, ctx.var(w)), [2 * n]).slice(0, off, off + n)
    flat = (a.astype(np.float64) @ w).ravel()[off:off + n]
    assert _close(evaluated(ctx, S.conv_2d(S.view(part(), [2, 20, 20, 64]), ctx.var(f), 1, 1, 1), r"^gemm_tc_h2\[", 2), _conv64(flat.reshape(2, 20, 20, 64), f, 1, 1))
    assert _close(evaluated(ctx, S.matmul(S.view(part(), [800, 64]), ctx.var(w2)), r"^gemm_tc_h2\[", 2), flat.reshape(800, 64) @ w2.astype(np.float64))
    assert ctx.status_word() == 0


@pytest.mark.parametrize("stride", [1, 2])
def test_a_filter_that_is_computed_from_a_variable(ctx, stride):
    """The packed filter of a first convolution follows the variable it is computed from, pass after pass."""
    rng = np.random.default_rng(87)
    x, m = rng.uniform(-1, 1, (2, 20, 200, 3)).astype(np.float32), rng.uniform(0.5, 1.5, (32,)).astype(np.float32)
    f = ctx.var(np.zeros((3, 3, 3, 32), np.float32))
    y = S.conv_2d(ctx.var(x), f * ctx.var(m), stride, 1, 1)
    for _ in range(5):
        values = rng.uniform(-1, 1, (3, 3, 3, 32)).astype(np.float32)
        ctx.set(f, values)
        ctx.clear()
        assert _close(evaluated(ctx, y, r"^conv_first_h2\[" if stride == 2 else r"^gemm_tc_3xtf32\[.*,conv"), _conv64(x, values * m, stride, 1))


def test_products_from_two_threads(monkeypatch):
    """Two contexts on two host threads, each launching the same kernels with rings of its own length in shared memory."""
    import threading
    monkeypatch.setenv("SAGE_VERBOSE_NAMES", "1")
    shapes = [[(64, 64, 256), (192, 512, 2048), (70, 128, 512)], [(24, 64, 4096), (192, 512, 320), (40, 96, 8192)]]
    wrong = []

    def work(mine):
        c = S.Context(0)
        try:
            rng = np.random.default_rng(len(mine))
            cases = [(rng.standard_normal((1, m, k), dtype=np.float32), rng.standard_normal((1, k, n), dtype=np.float32)) for m, n, k in mine]
            for _ in range(60):
                wrong.extend((a.shape, b.shape) for a, b in cases if not excess(product(c, a, b), a, b) <= 1.0)
        except Exception as e:
            wrong.append(repr(e))
        finally:
            c.close()
    threads = [threading.Thread(target=work, args=(s,)) for s in shapes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]


@pytest.mark.parametrize("m,n,k,tb", [(200, 130, 512, False), (200, 130, 520, True), (24, 96, 4096, False), (70, 40, 40000, False)])
@pytest.mark.parametrize("span,shift", [(30, 0), (50, 0), (80, 0), (90, -80)])
def test_range_along_the_contraction(ctx, m, n, k, tb, span, shift):
    """Rows of B scaled by 2^e and columns of A by 2^-e, e running over `span` along K: every term of a sum counts the same, and
    both operands keep their bits because their scales follow K in steps of 64.  Inside a group e spans span * 64 / k <= 10."""
    rng = np.random.default_rng(88)
    e = np.round(np.linspace(-span / 2, span / 2, k)).astype(np.int32)
    a = np.ldexp(rng.standard_normal((1, m, k)).astype(np.float32), -e[None, None, :] - shift)
    b = np.ldexp(rng.standard_normal((1, k, n)).astype(np.float32), e[None, :, None] + shift)  # (shift: into the subnormal numbers)
    got = product(ctx, a, np.ascontiguousarray(np.swapaxes(b, 1, 2)) if tb else b, tb=tb)
    assert excess(got, a, b) <= 1.0
    assert ctx.status_word() == 0


def test_range_along_the_contraction_inside_a_program(ctx):
    """The same for products of a program: separate and grouped weights, and a convolution's filter over its channels."""
    rng = np.random.default_rng(89)
    e = np.round(np.linspace(-20, 20, 512)).astype(np.int32)
    a = np.ldexp(rng.standard_normal((150, 512)).astype(np.float32), -e[None, :])
    w = np.ldexp(rng.standard_normal((512, 128)).astype(np.float32), e[:, None])
    got = evaluated(ctx, S.matmul(ctx.var(a) * 1.0, ctx.var(w)), r"^gemm_tc_h2\[")
    assert excess(got[None], a[None], w[None]) <= 1.0
    img = np.ldexp(rng.standard_normal((1, 12, 12, 512)).astype(np.float32), -e)
    f = np.ldexp(rng.standard_normal((3, 3, 512, 64)).astype(np.float32), e[None, None, :, None])
    got = evaluated(ctx, S.conv_2d(ctx.var(img) * 1.0, ctx.var(f), 1, 1, 1), r"^gemm_tc_h2\[.*,conv")
    assert (np.abs(got - _conv64(img, f, 1, 1)) / _conv64(np.abs(img), np.abs(f), 1, 1)).max() <= 3e-6
    scale = np.ldexp(np.ones(512, np.float32), -e)
    x = (rng.standard_normal((1, 64, 512)) * scale).astype(np.float32)
    ws = [np.ldexp(rng.standard_normal((512, 128)).astype(np.float32) / 16, e[:, None]) for _ in range(3)]
    X = ctx.var(x)
    q, k, v = [S.transpose(S.view(S.matmul(X, ctx.var(u)) + ctx.var(np.zeros(128, np.float32)), [1, 64, 2, 64]), 2, 1) for u in ws]
    y = S.matmul_batched(S.softmax(S.matmul_batched(q, S.transpose(k, -1, -2)) / 64.0, [3]), v)
    got = evaluated(ctx, y, r"^gemm_tc_h2\[64x128x512x3").astype(np.float64)
    q, k, v = [(x.astype(np.float64) @ u).reshape(1, 64, 2, 64).transpose(0, 2, 1, 3) for u in ws]
    s = q @ k.transpose(0, 1, 3, 2) / 64.0
    p = np.exp(s - s.max(-1, keepdims=True))
    want = (p / p.sum(-1, keepdims=True)) @ v
    assert (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-4


def _excess_conv(got, x, f, stride, pad):
    """Largest error over the bound: pieces and one chain of 4 KH additions on the tensor cores, or a sum in fp32 over the whole
    window, with S = the convolution of the magnitudes."""
    k = f.shape[0] * f.shape[1] * f.shape[2]
    s = _conv64(np.abs(x), np.abs(f), stride, pad)
    return float((np.abs(got - _conv64(x, f, stride, pad)) / np.maximum(s * max((k + 2) * 2.0 ** -24, 2.0 ** -22 + 2.0 ** -24 + (4 * f.shape[0] + 2) * 2.0 ** -23), 1e-300)).max())


@pytest.mark.parametrize("chan,oc,ker,width", [(3, 64, 7, 224), (3, 72, 7, 224), (4, 64, 3, 180), (1, 32, 8, 160), (2, 128, 5, 315)])
@pytest.mark.parametrize("what", ["plain", "channels", "filter", "dark", "stray", "special"])
def test_range_inside_a_first_convolution(monkeypatch, chan, oc, ker, width, what):
    """Images and filters whose elements are further apart than pieces under one scale hold: channels in different units that the
    filter makes up for, one output channel's filter over a wide range, an image dark but for a spot, one stray tiny pixel; and
    infinities, which stay near where they are.  An image without them beside one with them takes the ordinary way."""
    monkeypatch.setenv("SAGE_VERBOSE_NAMES", "1")
    rng = np.random.default_rng(90 + chan)
    pad = ker // 2
    x = rng.uniform(0.5, 1.0, (3, 30, width, chan)).astype(np.float32) * rng.choice(np.array([-1, 1], np.float32), (3, 30, width, chan))
    f = rng.standard_normal((ker, ker, chan, oc)).astype(np.float32)
    if what == "channels":
        e = np.linspace(-30, 30, chan).astype(np.int32) if chan > 1 else np.zeros(1, np.int32)
        x[1], f = np.ldexp(x[1], -e), np.ldexp(f, e[:, None])
    elif what == "filter":
        f[..., oc // 2] = np.ldexp(f[..., oc // 2], rng.integers(-60, 1, f.shape[:3]))
        x[:, :, :width // 2] = 0.0
    elif what == "dark":
        x[2] = np.ldexp(x[2], -40)
        x[2, 3:5, 7:9] = 1.0
    elif what == "stray":
        x[0, 11, 13, 0] = 1e-30
    elif what == "special":
        x[0, 20, 50, 0], x[1, 5, 60, 0] = np.inf, np.nan
    c = S.Context(0)
    try:
        c.trace_begin()
        got = S.conv_2d(c.var(x), c.var(f), 2, pad, 1).eval(c).astype(np.float64)
        assert any(n.startswith("conv_first_h2") for n in c.trace()) and c.status_word() == 0
    finally:
        c.close()
    if what == "special":
        touched = ~np.isfinite(_conv64(np.where(np.isfinite(x), x, np.nan), f, 2, pad))
        near = np.zeros(got.shape[:3], bool)
        near[0, 10 - ker:10 + ker, 25 - ker:25 + ker] = near[1, :3 + ker, 30 - ker:30 + ker] = True
        assert not np.isfinite(got[touched]).any() and np.isfinite(got[~near]).all()
        return
    assert _excess_conv(got, x, f, 2, pad) <= 1.0
