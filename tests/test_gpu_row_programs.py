"""Whole-row programs (graph/rowfuse.cc) over column counts where the block's shape changes."""
import re

import numpy as np
import pytest

import sage_b200 as S

pytestmark = pytest.mark.gpu


# 3000: the two prefetch stages take 48 KiB exactly, and the kernel's own shared memory lies beside them.  From 4096: 32 elements a
# thread where the threads have whole shares (4096, 4100 not, 6140 with an idle vector, 7000, 16384 and one vector less), 16 elsewhere.
@pytest.mark.parametrize("rows,cols", [(37, 3000), (600, 4096), (5, 4092), (37, 4100), (300, 6140), (33, 7000), (5, 8192), (200, 16384), (2, 16380)])
def test_cross_entropy_and_gradient(rows, cols):
    """Loss and gradient of the cross entropy of x y + 3.14 x against float64.  Tolerance: sums of `cols` fp32 terms and a few
    roundings of the exponentials, 1e-5 of the value or of the rms."""
    rng = np.random.default_rng(cols)
    x, y = (rng.standard_normal((rows, cols), dtype=np.float32) for _ in range(2))
    labels = rng.integers(0, cols, (rows, 1)).astype(np.uint32)
    ctx = S.Context(0)
    try:
        xv = ctx.var(x)
        loss = S.softmax_cross_entropy(xv * ctx.var(y) + xv * 3.14, ctx.var(labels))
        gx = xv.grad(loss)
        ctx.eval(loss, gx)
        assert ctx.describe().startswith("row_program[%dx%d" % (rows, cols))
        z = x.astype(np.float64) * y + x * np.float64(np.float32(3.14))
        m = z.max(1, keepdims=True)
        lse = np.log(np.exp(z - m).sum(1, keepdims=True)) + m
        p = np.exp(z - lse)
        p[np.arange(rows), labels[:, 0]] -= 1
        for got, want in ((ctx.read(loss).reshape(-1), (lse - np.take_along_axis(z, labels.astype(np.int64), 1))[:, 0]), (ctx.read(gx), p * (y.astype(np.float64) + np.float32(3.14)))):
            assert (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max() <= 1e-5
        assert ctx.status_word() == 0
    finally:
        ctx.close()


def test_a_program_of_many_reductions():
    """Forty reductions hold 10 KiB of shared memory, and the two prefetch stages of 2560 columns 40 KiB: together more than a kernel
    may have without being allowed it.  Each maximum is one element: the sum of forty of them and a product, 42 roundings."""
    rng = np.random.default_rng(40)
    rows, cols = 24, 2560
    x, y = (rng.standard_normal((rows, cols), dtype=np.float32) for _ in range(2))
    ctx = S.Context(0, ref_compat=0)
    try:
        xv, yv = ctx.var(x), ctx.var(y)
        total = sum(((xv * float(i) + yv).max([1], True) for i in range(1, 40)), (xv + yv).max([1], True))
        out = xv * S.expand(total, [rows, cols])
        got = out.eval(ctx)
        assert re.match(r"row_program\[24x2560; 160 threads x 16\]\{\d+ maps, 40 reductions", ctx.describe()), ctx.describe()
        sums = [(x * np.float32(i) + y).max(1, keepdims=True).astype(np.float64) for i in range(1, 40)] + [(x + y).max(1, keepdims=True).astype(np.float64)]
        assert (np.abs(got - x * sum(sums)) <= 45 * 2.0 ** -24 * np.abs(x) * sum(map(np.abs, sums))).all()
        assert ctx.status_word() == 0
    finally:
        ctx.close()
