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
