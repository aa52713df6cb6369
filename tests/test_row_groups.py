"""States that may share a generated row kernel but not with one another's readers between them."""
import numpy as np
import pytest

import sage_b200 as S


def crossed(c, seed=0):
    """Two chains in row spaces of their own, each of whose second halves reads a product of the other's first half."""
    rng = np.random.default_rng(seed)
    x, y, w, v = (rng.standard_normal(s).astype(np.float32) for s in ((64, 96), (64, 48), (48, 96), (96, 48)))
    a, b = S.softmax(c.var(x) * 2.0, [1]), S.softmax(c.var(y) * 2.0, [1])
    p, q = b.matmul(c.var(w)), a.matmul(c.var(v))

    def softmax(t):
        e = np.exp(t - t.max(1, keepdims=True))
        return e / e.sum(1, keepdims=True)
    x, y, w, v = (t.astype(np.float64) for t in (x, y, w, v))
    a64, b64 = softmax(2 * x), softmax(2 * y)
    return [S.softmax(a * 3.0 + p, [1]), S.softmax(b * 3.0 + q, [1]), p, q], [softmax(3 * a64 + b64 @ w), softmax(3 * b64 + a64 @ v), b64 @ w, a64 @ v]


def test_no_two_groups_read_one_another():
    """Both chains as row kernels would wait for one another: one of them is, and the program ends."""
    c = S.Context(-1)
    targets, _ = crossed(c)
    c.eval(*targets)
    assert c.describe().count("row") >= 1
    c.clear()
    c.trace_begin()
    c.eval(*targets)
    assert c.trace().count("sage_row_program") == 1
    c.close()


@pytest.mark.gpu
def test_values_of_crossed_chains():
    """Products within 2^-19 of |b| |w|, at most 4 here; a softmax's values follow its argument's difference, e^d - 1 ~ d, and 2^-20 of its own."""
    c = S.Context(0)
    try:
        targets, want = crossed(c)
        for _ in range(2):
            c.clear()
            c.eval(*targets)
        for t, ref in zip(targets, want):
            assert np.abs(c.read(t) - ref).max() <= 2.0 ** -16
        assert c.status_word() == 0
    finally:
        c.close()
