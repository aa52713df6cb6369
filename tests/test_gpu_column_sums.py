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
