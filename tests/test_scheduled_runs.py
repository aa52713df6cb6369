"""Evaluation of a program in the order worked out for it.  The order must survive memory getting tight, in the first run or later (the
run then goes on by eviction and recomputation), and values that other evaluations left behind."""
import numpy as np
import pytest

import sage_b200 as S

MIB = 1 << 20


def graph(c, x):
    n = x.size
    a = [x * float(i + 2) + 1.0 for i in range(12)]          # twelve 4 MiB states, each needed early and again late
    s = [v.sum([0], True) for v in a]
    z = s[0]
    for v in s[1:]:
        z = z + v
    t = [(v * z.expand([n])).sum([0], True) for v in a]
    out = s[0] * 0.0
    for v, w in zip(t, s):
        out = out + v + v * 2.0 + w
    return s[3], out


def passes(c, x):
    """Launch counts of four passes (the third with most of the memory taken by somebody else) and their results."""
    mid, out = graph(c, x)
    counts, values, held = [], [], []
    for i in range(4):
        c.clear()
        if i == 2:
            held = [c.alloc(4 * MIB) for _ in range(10)]
        c.trace_begin()
        c.eval(out)
        counts.append(len(c.trace()))
        if c.device >= 0:
            values.append(c.read(out))
        for b in held:
            c.free(b)
        held = []
    c.clear()
    c.eval(mid)                      # an intermediate evaluated on its own becomes an input of the next program
    c.eval(out)
    if c.device >= 0:
        values.append(c.read(out))
    return counts, values


def test_a_scheduled_run_goes_on_when_memory_gets_tight():
    c = S.Context(-1, mem_capacity_bytes=84 * MIB)
    counts, _ = passes(c, c.var(np.zeros((MIB,), np.float32)))
    assert counts[0] == counts[1] == counts[3] and counts[2] > counts[0]
    assert c.mem_stats()["mem_peak"] <= 84 * MIB
    c.close()


@pytest.mark.gpu
def test_scheduled_runs_give_the_first_runs_values():
    x = np.random.default_rng(77).standard_normal(MIB).astype(np.float32) * np.float32(1e-3)
    c = S.Context(0, mem_capacity_bytes=84 * MIB)
    try:
        counts, values = passes(c, c.var(x))
        assert counts[0] == counts[1] == counts[3] and counts[2] > counts[0]
        for v in values[1:]:
            assert np.array_equal(v, values[0]) and np.isfinite(v).all()
        assert c.status_word() == 0
    finally:
        c.close()


def products(c, n, k, x, w):
    """k maps whose tf32 planes two products each read, early and late: with a value (4 n^2 bytes) come planes of twice its size."""
    x, w = c.var(x), c.var(w)
    a = [x * (0.25 * (i + 1)) + 1.0 for i in range(k)]
    s = [v.matmul(w).sum([0], True) for v in a]
    z = s[0]
    for v in s[1:]:
        z = z + v
    z = (z * 1e-3).expand([n, 64])
    t = [v.matmul(z).sum([0], True) for v in a]
    out = s[0] * 0.0
    for v, u in zip(t, s):
        out = out + v + v * 2.0 + u
    return out


def under(device, capacity, n, k, x, w):
    """Launches of maps, and the value, of a first run (every tensor a buffer of its own); None where memory does not suffice."""
    c = S.Context(device, use_cache=0, **({"mem_capacity_bytes": capacity} if capacity else {}))
    try:
        out = products(c, n, k, x, w)
        c.trace_begin()
        try:
            c.eval(out)
        except S.SageError:
            return None
        maps = c.trace().count("sage_map")
        value = c.read(out) if device >= 0 else None
        assert c.status_word() == 0
        return maps, value, c.mem_stats()["mem_peak"]
    finally:
        c.close()


def test_a_step_that_ran_out_of_memory_is_run_again():
    """Six values of 4 MiB with 8 of planes each: below the unrestricted peak, less the scratch of a product's K slices (which does without),
    one of them at least has to go and come back."""
    n, k = 1024, 6
    x, w = np.zeros((n, n), np.float32), np.zeros((n, 64), np.float32)
    maps, _, peak = under(-1, 0, n, k, x, w)
    runs = [under(-1, peak - MIB * d, n, k, x, w) for d in range(4, 20)]
    assert all(r is not None and r[0] > maps for r in runs), "%d %s" % (maps, [r and r[0] for r in runs])


@pytest.mark.gpu
def test_first_runs_under_a_limit_give_the_unrestricted_values():
    n, k = 1024, 6
    rng = np.random.default_rng(78)
    x, w = rng.standard_normal((n, n)).astype(np.float32), rng.standard_normal((n, 64)).astype(np.float32)
    _, want, peak = under(0, 0, n, k, x, w)
    evicted = 0
    for d in list(range(4, 24, 2)) + [30, 40, 50]:
        run = under(0, peak - MIB * d, n, k, x, w)
        if run:
            evicted += 1
            # (the sum over a product's K slices has no room at some limits: one pass over K instead, 2^-20 of the terms' magnitudes)
            assert np.allclose(run[1], want, rtol=0, atol=2.0 ** -14 * np.abs(want).max()), d
    assert evicted >= 8


def independent_products(c, k, x, y):
    """(x a)^T (y b): products that nothing reads, each with operands of its own, which are put off to run together."""
    x, y = c.var(x), c.var(y)
    return [S.transpose(x * float(i + 2), 1, 0).matmul(y * (float(i) - 2.5)) for i in range(k)]


def test_products_put_off_keep_little_alive_and_run_once():
    """Operands of 16 MiB, 32 of planes each: 96 MiB a product, of which 128 and the product's at hand are kept."""
    x = np.zeros((4096, 1024), np.float32)
    peaks = {}
    for k, limits in ((24, (0,)), (8, (0, 168, 184, 232, 264, 312, 328))):
        for limit in limits:
            c = S.Context(-1, **({"mem_capacity_bytes": limit * MIB} if limit else {}))
            out = independent_products(c, k, x, x)
            for _ in range(2):
                c.clear()
                c.trace_begin()
                c.eval(*out)
                assert sum("gemm" in t for t in c.trace()) == k, (k, limit)  # out of memory or not, none is worked out again
            if not limit:
                peaks[k] = c.mem_stats()["mem_peak"]
            c.close()
    assert peaks[24] - peaks[8] == 16 * 4 * MIB  # the results
    assert peaks[8] <= (32 + 2 * 96 + 32 + 8 * 4 + 3 * 20) * MIB  # x and y, two products' operands, values before their planes, results, segments


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [0, 168, 200, 264, 328])
def test_products_put_off_under_a_limit(limit):
    """Against float64, within (2^-22 + 48 x 2^-23 + (rows / 128 + 1) 2^-24) |x|^T |y|, as grouped products by themselves."""
    rng = np.random.default_rng(79)
    x, y = rng.standard_normal((4096, 1024)).astype(np.float32), rng.standard_normal((4096, 1024)).astype(np.float32)
    c = S.Context(0, **({"mem_capacity_bytes": limit * MIB} if limit else {}))
    try:
        out = independent_products(c, 8, x, y)
        for _ in range(2):
            c.clear()
            c.eval(*out)
        got = [c.read(t).copy() for t in out]
        assert c.status_word() == 0
    finally:
        c.close()
    xy, size = x.astype(np.float64).T @ y, np.abs(x).astype(np.float64).T @ np.abs(y)
    bound = (2.0 ** -22 + 48 * 2.0 ** -23 + (4096 / 128 + 1) * 2.0 ** -24 + 2.0 ** -23) * size  # (and the two maps' roundings)
    for i, g in enumerate(got):
        a = (i + 2) * (i - 2.5)
        assert (np.abs(g - a * xy) <= abs(a) * bound).all(), i
