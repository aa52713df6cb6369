"""Repeated evaluation of one program: from the second run on the evaluator follows the order of the first.  The order must
survive memory getting tight later (the run then goes on by eviction and recomputation) and values that other evaluations
left behind."""
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
