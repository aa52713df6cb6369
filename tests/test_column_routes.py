"""Which kernel a column reduction takes (kernels/reduce.cu: launch_reduce_cols): clusters where all their CTAs run at once."""
import numpy as np
import pytest

import sage_b200 as S


@pytest.fixture(scope="module")
def ctx():
    with pytest.MonkeyPatch.context() as m:
        m.setenv("SAGE_VERBOSE_NAMES", "1")
        c = S.Context(-1)
    yield c
    c.close()


@pytest.mark.parametrize("rows,cols,cluster", [(64, 4096, True), (64, 50000, False), (64, 524288, False), (128, 12288, False), (128, 262144, False), (256, 6000, False), (384, 4096, True),
                                               (1000, 768, True), (1000, 4096, False), (1000, 9473, False), (1000, 31, True), (2048, 1001, False), (4096, 768, True), (4096, 64, False),
                                               (8192, 2, False), (1024, 32768, True), (1000, 30011, False), (1000, 50000, False), (1000, 50001, True), (512, 65536, True), (512, 65540, False)])
def test_route(ctx, rows, cols, cluster):
    y = ctx.var(np.zeros((rows, cols), np.float32))
    ctx.trace_begin()
    ctx.eval(y.sum([0], False))
    assert ctx.trace() == ["reduce_cols_cluster" if cluster else "reduce_cols"]
    ctx.clear()
    ctx.drop_programs()
