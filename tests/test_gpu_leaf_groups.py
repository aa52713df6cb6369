"""Column sums that nothing of a program reads, in one pass over all of them (kernels/column_sums.cu): rows of one chunk and of many,
columns past one block, both widths of load."""
import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu


def test_column_sums_pass_on_what_is_not_finite():
    rng = np.random.default_rng(5)
    ctx = S.Context(0)
    try:
        xs = [rng.standard_normal((rows, cols)).astype(np.float32) for rows, cols in ((64, 68), (999, 33), (3000, 2052), (5000, 5), (65, 4100), (40000, 2), (7000, 768))]
        for x in xs:
            x[rng.integers(0, len(x), 3), rng.integers(0, x.shape[1], 3)] = (np.nan, np.inf, -np.inf)
        sums = [ctx.var(x).sum([0], False) for x in xs]
        before = ctx.launch_count()[0]
        ctx.eval(*sums)
        assert ctx.launch_count()[0] - before == 2
        for x, s in zip(xs, sums):
            with np.errstate(invalid="ignore"):
                want = x.astype(np.float64).sum(0)
            got = ctx.read(s).reshape(-1)
            assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
            ok = np.isfinite(want)
            assert (np.abs(got[ok] - want[ok]) <= len(x) * 2.0 ** -24 * np.abs(x).astype(np.float64).sum(0)[ok]).all()
        assert ctx.status_word() == 0
    finally:
        ctx.close()
