"""Column reductions over clusters (kernels/reduce.cu: reduce_cols_cluster_kernel) where they can go wrong: rows that no CTA of a
cluster, one or all of them have; a run that ends inside a thread's eight loads; the last column tile cut; both widths of load."""
import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu


# (the lengths of a CTA's run: 64, 65, up to the 1024 rows or 2048 of single columns, and one more, which the other kernel takes)
@pytest.mark.parametrize("rows,cols", [(64, 64), (127, 64), (130, 68), (513, 768), (4096, 768), (4097, 130), (999, 33), (8192, 64), (8193, 64), (16384, 31), (16385, 31), (300, 20000), (65, 2)])
def test_column_reductions(rows, cols):
    """Sums within the bound of a sum of `rows` terms in any order, rows x 2^-24 of the sum of magnitudes; largest elements exactly."""
    rng = np.random.default_rng(rows + cols)
    x = rng.standard_normal((rows, cols), dtype=np.float32)
    ctx = S.Context(0)
    try:
        v = ctx.var(x)
        ctx.trace_begin()
        got = v.sum([0], False).eval(ctx).reshape(-1)
        assert "reduce_cols" in ctx.trace()
        bound = rows * 2.0 ** -24 * np.abs(x).astype(np.float64).sum(0)
        assert (np.abs(got - x.astype(np.float64).sum(0)) <= bound).all()
        big = ctx.var(np.abs(x))
        assert np.array_equal(big.max([0], False).eval(ctx).reshape(-1), np.abs(x).max(0))
        assert ctx.status_word() == 0
    finally:
        ctx.close()


# Kernels of both kinds, and both widths of load; a row pitch above the columns.
@pytest.mark.parametrize("rows,cols", [(300, 68), (2048, 1000), (999, 33), (64, 50000), (1000, 9473), (512, 66000), (9000, 70)])
@pytest.mark.parametrize("pitch", [0, 4, 5])
def test_column_reductions_of_every_kind(rows, cols, pitch):
    """Products, smallest and largest elements with infinities, nan (which both pass over), columns of the type's lowest value and whole
    numbers, in contexts whose accumulators start where they should.  Products: `rows` roundings."""
    rng = np.random.default_rng(rows + pitch)
    x = rng.standard_normal((rows, cols + pitch), dtype=np.float32)
    x[rng.integers(0, rows, 40), rng.integers(0, cols, 40)] = np.nan
    x[rng.integers(0, rows, 40), rng.integers(0, cols, 40)] = np.inf
    x[rng.integers(0, rows, 40), rng.integers(0, cols, 40)] = -np.inf
    x[:, 0], x[:, 1] = -np.finfo(np.float32).max, np.nan
    near = (1 + rng.uniform(-1, 1, (rows, cols + pitch)) / rows).astype(np.float32)
    whole = rng.integers(-2 ** 31, 2 ** 31, (rows, cols + pitch)).astype(np.int32)
    whole[:, 0] = -2 ** 31
    ctx = S.Context(0, ref_compat=0)
    try:
        part = lambda v: v.slice(1, 0, cols) if pitch else v
        ctx.trace_begin()
        v = part(ctx.var(x))
        assert np.array_equal(v.max([0], False).eval(ctx).reshape(-1), np.fmax.reduce(x[:, :cols], 0, initial=-np.inf))
        assert np.array_equal(v.min([0], False).eval(ctx).reshape(-1), np.fmin.reduce(x[:, :cols], 0, initial=np.inf))
        got, want = part(ctx.var(near)).prod([0], False).eval(ctx).reshape(-1), near[:, :cols].astype(np.float64).prod(0)
        assert (np.abs(got - want) <= rows * 2.0 ** -24 * np.abs(want)).all()
        w = part(ctx.var(whole))
        assert np.array_equal(w.max([0], False).eval(ctx).reshape(-1), whole[:, :cols].max(0))
        assert np.array_equal(w.min([0], False).eval(ctx).reshape(-1), whole[:, :cols].min(0))
        assert np.array_equal(w.sum([0], False).eval(ctx).reshape(-1), whole[:, :cols].sum(0, dtype=np.int64).astype(np.int32))
        s = v.sum([0], False).eval(ctx).reshape(-1)
        with np.errstate(invalid="ignore"):
            want = x[:, :cols].astype(np.float64).sum(0)
        assert np.array_equal(np.isnan(s), np.isnan(want)) and np.array_equal(s[np.isinf(want)], want[np.isinf(want)])
        assert ctx.trace().count("reduce_cols") == 7, ctx.trace()
        assert ctx.status_word() == 0
    finally:
        ctx.close()


@pytest.mark.parametrize("rows,cols", [(520, 66560), (600, 60001)])
def test_column_sums_beyond_the_caches(rows, cols):
    """A CTA to a column tile of all rows, the last one cut.  Bound as above."""
    x = np.random.default_rng(cols).standard_normal((rows, cols), dtype=np.float32)
    ctx = S.Context(0)
    try:
        got = ctx.var(x).sum([0], False).eval(ctx).reshape(-1)
        assert (np.abs(got - x.sum(0, dtype=np.float64)) <= rows * 2.0 ** -24 * np.abs(x).sum(0, dtype=np.float64)).all()
        assert ctx.status_word() == 0
    finally:
        ctx.close()
