"""Results that nothing of a program reads, computed together: products in one launch (kernels/gemm_group.cu), column sums in one pass
(kernels/column_sums.cu).  Gradients of s = sum(((X W) + b) * C) over W (X^T C) and b (the column sums of C) for matrices of many
sizes in one program."""
import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu

# (rows, inputs, outputs): K of one chain and of many slices, ragged M, N and K, tiles of every width, single columns (130 + 1), a
# pair's second CTA without rows, rows of one chunk, columns past one block
SIZES = {
    "two": [(64, 64, 32), (4096, 768, 768)],
    "narrow": [(6272, 576, 64), (25088, 49, 64), (6271, 65, 33), (100, 2304, 96), (4100, 300, 160)],
    "wide": [(130, 257, 1001), (2049, 256, 2052), (512, 1152, 260), (96, 4608, 512), (1000, 129, 131)],
    "many": [(64 + 37 * i, 64 + 29 * (i % 7), 32 + 13 * (i % 11)) for i in range(15)],
}


@pytest.mark.parametrize("which", sorted(SIZES))
def test_gradients_of_many_products(which):
    rng = np.random.default_rng(len(which))
    ctx = S.Context(0)
    try:
        ctx_vars, xs, cs, loss = [], [], [], None
        for rows, k, n in SIZES[which]:
            x = (rng.standard_normal((rows, k)) * np.exp2(rng.integers(-12, 12, (1, k)))).astype(np.float32)
            c = (rng.standard_normal((rows, n)) + 0.25).astype(np.float32)
            w, b = ctx.var(np.zeros((k, n), np.float32)), ctx.var(np.zeros((n,), np.float32))
            s = ((ctx.var(x).matmul(w) + b) * ctx.var(c)).sum([0, 1], False)
            loss = s if loss is None else loss + s
            xs.append(x)
            cs.append(c)
            ctx_vars.append((w, b))
        targets = [v.grad(loss) for pair in ctx_vars for v in pair]
        runs = []
        for _ in range(2):
            ctx.clear()
            ctx.eval(*targets)
            runs.append([ctx.read(t).copy() for t in targets])
        assert ctx.status_word() == 0
        for first, second in zip(*runs):  # the first pass and the later ones take the same way
            assert np.array_equal(first, second)
        before = ctx.launch_count()[0]
        ctx.clear()
        ctx.trace_begin()
        ctx.eval(*targets)
        assert len(ctx.trace()) - (ctx.launch_count()[0] - before) >= 2 * (len(xs) - 1)  # launches that did several results' work
        for i, (x, c) in enumerate(zip(xs, cs)):
            dw, db = runs[0][2 * i].reshape(x.shape[1], c.shape[1]), runs[0][2 * i + 1].reshape(-1)
            x64, c64 = x.astype(np.float64), c.astype(np.float64)
            size = np.abs(x64).T @ np.abs(c64)
            # the dropped low x low products, 48 truncating additions of a chain, a rounding for every chain
            bound = (2.0 ** -22 + 48 * 2.0 ** -23 + (x.shape[0] / 128 + 1) * 2.0 ** -24) * size
            assert (np.abs(dw - x64.T @ c64) <= bound).all(), (which, i)
            assert (np.abs(db - c64.sum(0)) <= x.shape[0] * 2.0 ** -24 * np.abs(c64).sum(0)).all(), (which, i)
    finally:
        ctx.close()


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


@pytest.mark.parametrize("shift", [0, 1])
def test_sums_over_whole_tensors(shift):
    """Runs of one block and of many, an end inside a thread's loads, an operand off the 16-byte grid, and operands that exist only for
    their sum, more of them than are kept at once."""
    rng = np.random.default_rng(6)
    ctx = S.Context(0)
    try:
        xs = [rng.standard_normal(n).astype(np.float32) for n in (64, 67, 16384, 16388, 3145728, 5000001)]
        variables = [ctx.var(x) for x in xs]
        if shift:
            variables, xs = [v.slice(0, 1, v.extents[0]) for v in variables], [x[1:] for x in xs]
        big = ctx.var(rng.standard_normal(1 << 23).astype(np.float32))
        sums = [v.sum([0], False) for v in variables] + [(big * (i + 0.5)).sum([0], False) for i in range(10)]
        ctx.eval(*sums)
        big64 = ctx.read(big).astype(np.float64)
        for got, x in zip((ctx.read(s).reshape(-1)[0] for s in sums), [x.astype(np.float64) for x in xs] + [big64 * (i + 0.5) for i in range(10)]):
            assert abs(got - x.sum()) <= 64 * 2.0 ** -24 * np.abs(x).sum()  # fewer than 64 roundings on the way of any element
        assert ctx.status_word() == 0
    finally:
        ctx.close()
