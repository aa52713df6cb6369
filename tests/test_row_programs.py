"""Which whole-row programs hold 32 elements a thread (graph/rowfuse.cc), and that those have the registers for it."""
import os
import re
import subprocess

import numpy as np
import pytest

import sage_b200 as S


@pytest.fixture(scope="module")
def ctx():
    c = S.Context(-1)
    yield c
    c.close()


def graphs(ctx, cols):
    """name -> (targets, elements a thread)"""
    rows = 64
    x, y = ctx.var(np.zeros((rows, cols), np.float32)), ctx.var(np.zeros((rows, cols), np.float32))
    labels = ctx.var(np.zeros((rows, 1), np.uint32))
    ex = lambda v: S.expand(v, [rows, cols])

    def entropy(z, grad=True):
        loss = S.softmax_cross_entropy(z, labels)
        return [loss, x.grad(loss)] if grad else [loss]

    def alive(k):  # k values of the row are needed again once all of them have been summed
        u = [f(x) for f in (lambda v: v * 1.5, S.exp, S.tanh, lambda v: v * v, S.sin, S.cos)[:k]]
        total, out = ex(sum((v.sum([1], True) for v in u[1:]), u[0].sum([1], True))), None
        for v in u:
            out = v / (total + 3.0) if out is None else out * (v / (total + 3.0))
        return [out]

    def softmax(z):
        e = (z - ex(z.max([1], True))).exp()
        return e / ex(e.sum([1], True))

    return {"entropy": (entropy(x * y + x * 3.14), 32), "entropy of x": (entropy(x), 32), "loss": (entropy(x * y, False), 32),
            "five alive": (entropy(x.tanh() * y.exp() + x.sin()), 16), "many alive": (entropy((x * y).tanh() * x.sin() + x.exp() * y), 16),
            "softmax": ([softmax(x * y) * 2.0], 16), "one": (alive(1), 16), "three": (alive(3), 16), "six": (alive(6), 16)}


@pytest.mark.parametrize("cols", [4096, 6144])
def test_elements_a_thread(ctx, cols, tmp_path, monkeypatch):
    """Programs that keep many rows alive, or that pick nothing from the row, keep 16; those with 32 compile without spills."""
    dump = tmp_path / "program.cu"
    monkeypatch.setenv("SAGE_ROW_PROGRAM_DUMP", str(dump))
    for name, (targets, elements) in graphs(ctx, cols).items():
        ctx.clear()
        ctx.drop_programs()
        ctx.eval(*targets)
        got = re.match(r"row_program\[64x%d; \d+ threads x (\d+)\]" % cols, ctx.describe())
        assert got and int(got.group(1)) == elements, (name, ctx.describe())
        if elements == 32:
            out = subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-Xptxas", "-v", "-cubin",
                                  "-o", str(tmp_path / "program.cubin"), str(dump)], capture_output=True, text=True)
            assert out.returncode == 0 and "0 bytes spill stores" in out.stderr, (name, out.stderr)
