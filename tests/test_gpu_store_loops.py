"""Products whose store loops over its sub-tiles (kernels/gemm_h2_device.inc, SAGE_H2_ROLL): one tile a CTA, and expressions that call long
functions, at the edges of tiles and sub-tiles, stored as fp32, as pieces for a following product, and both."""
import numpy as np
import pytest
import torch

import sage_b200 as S

pytestmark = pytest.mark.gpu


# rows, k, columns: one tile cut in both directions; no whole 16 bytes in a row; whole groups of 64 (pieces); several tiles a CTA
@pytest.mark.parametrize("m,k,n", [(129, 256, 192), (200, 320, 97), (462, 768, 3072), (4096, 512, 2048), (130, 64, 130), (5000, 256, 1000)])
@pytest.mark.parametrize("long", [False, True])
def test_epilogues(m, k, n, long):
    """Against float64: the product within 2^-19 of |x| |w| (its bound, tests of the half-precision products), through a function whose
    slope is at most 1.13, and the second product, of 64 columns, likewise."""
    rng = np.random.default_rng(m + n)
    x, w, b = rng.standard_normal((m, k)).astype(np.float32), (rng.standard_normal((k, n)) / np.sqrt(k)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    w2 = (rng.standard_normal((n, 64)) / np.sqrt(n)).astype(np.float32)
    ctx = S.Context(0)
    try:
        h = ctx.var(x).matmul(ctx.var(w)) + ctx.var(b)
        y = h * 0.5 * ((h * 0.70710678).erf() + 1.0) if long else S.relu(h)
        z = y.matmul(ctx.var(w2))
        got_y = y.eval(ctx).copy()
        ctx.clear()
        got_z = z.eval(ctx).copy()
        ctx.clear()
        ctx.eval(y, z)
        both = ctx.read(y).copy(), ctx.read(z).copy()
        assert ctx.status_word() == 0
    finally:
        ctx.close()
    x64, w64 = torch.from_numpy(x).double(), torch.from_numpy(w).double()
    h64 = x64 @ w64 + torch.from_numpy(b).double()
    size = x64.abs() @ w64.abs() + torch.from_numpy(b).double().abs()
    y64 = h64 * 0.5 * (torch.erf(h64 * np.float64(np.float32(0.70710678))) + 1) if long else h64.clamp(min=0)
    y_bound = 2.0 ** -19 * size
    w2_64 = torch.from_numpy(w2).double()
    z_bound = y_bound @ w2_64.abs() + 2.0 ** -19 * (y64.abs() @ w2_64.abs())
    for a in (got_y, both[0]):
        assert ((torch.from_numpy(a).double() - y64).abs() <= y_bound).all()
    for a in (got_z, both[1]):
        assert ((torch.from_numpy(a).double() - y64 @ w2_64).abs() <= z_bound).all()


# a residual through the operand ring: tiles of every width, one cut in both directions, rows longer than the result's, one tile and
# several to a CTA, a single K-block, an operand off the 16-byte grid (which the store fetches itself)
@pytest.mark.parametrize("m,k,n", [(129, 64, 64), (200, 320, 100), (300, 256, 128), (4096, 768, 768), (1536, 128, 192), (2000, 200, 516), (6000, 128, 1024), (130, 96, 260)])
@pytest.mark.parametrize("wider,shift", [(0, 0), (8, 4), (8, 1)])
def test_residuals(m, k, n, wider, shift):
    """Against float64, within 2^-19 of |x| |w| + |r|."""
    rng = np.random.default_rng(m + n + wider)
    x, w, b = rng.standard_normal((m, k)).astype(np.float32), (rng.standard_normal((k, n)) / np.sqrt(k)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    r = rng.standard_normal((m, n + wider)).astype(np.float32)
    ctx = S.Context(0)
    try:
        rv = ctx.var(r)
        if wider:
            rv = rv.slice(1, shift, shift + n)
        y = ctx.var(x).matmul(ctx.var(w)) + ctx.var(b) + rv
        for _ in range(2):
            ctx.clear()
            got = y.eval(ctx).copy()
        assert ctx.status_word() == 0
    finally:
        ctx.close()
    x64, w64 = x.astype(np.float64), w.astype(np.float64)
    r64 = r[:, shift:shift + n].astype(np.float64)
    assert (np.abs(got - (x64 @ w64 + b + r64)) <= 2.0 ** -19 * (np.abs(x64) @ np.abs(w64) + np.abs(b) + np.abs(r64))).all()


# wider tiles through the ring, a CTA alone, several tiles to a CTA
@pytest.mark.parametrize("m,k,n", [(1100, 200, 1000), (1100, 64, 1024), (4096, 200, 1000), (3000, 96, 1000), (120, 96, 260)])
@pytest.mark.parametrize("wider,shift", [(0, 0), (8, 4), (8, 1)])
def test_residuals_of_other_tiles(m, k, n, wider, shift):
    test_residuals(m, k, n, wider, shift)
