"""Rules of the device sources that no run shows when they are broken: the sources are read instead."""
import os
import re

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sage_b200", "csrc", "kernels")
PRODUCT = open(os.path.join(KERNELS, "gemm_h2_device.inc")).read()


def test_rows_of_epilogue_operands_are_prefetched_inside_the_result():
    """An L2 prefetch faults on nothing and returns nothing, so an address behind the operand passes every run.  The guard of the row
    operands' prefetch, evaluated for tiles of every width over results that do not fill the last one."""
    guard = re.search(r"What the store will take from the rows.*?\n\s*if \((.*?)\) \{", PRODUCT, re.S).group(1)
    guard = re.sub(r"!SLICED", "True", guard).replace("&&", "and")
    for n in (64, 65, 130, 136, 192, 200, 300, 768):
        for width in (64, 128, 192, 256):
            for n0 in range(0, n, width):
                parts = [part for part in range(4) if eval(guard, {"part": part, "width": width, "n0": n0, "n_end": min(n, n0 + width)})]
                assert parts == [part for part in range(width // 64) if n0 + part * 64 < n], (n, width, n0, guard)


def test_aligned_cluster_barriers_follow_a_reconvergence():
    """barrier.cluster.*.aligned is undefined for a warp whose lanes have gone different ways.  In front of each (or of the
    arrival directly before a wait) stands a barrier of the warp or the block."""
    text = re.sub(r"//[^\n]*", "", PRODUCT)
    body = text[text.index("void gemm_h2_body"):]
    found = 0
    for m in re.finditer(r"barrier\.cluster\.(arrive|wait)\.\w+\.aligned", body):
        found += 1
        before = body[: m.start()].rstrip()
        before = re.sub(r"(if \(!?S\w+\)( \{)?\s*)?asm volatile\(\"$", "", before).rstrip()
        # the statement in front; conditions of the whole block (SLICED, SEND, PAIR, the role of a warp) do not separate lanes
        before = re.sub(r"if (constexpr )?\(!?(SLICED|SEND|PAIR)\)( \{|[^;\n]*;)$", "", before).rstrip()
        assert before.endswith(("__syncwarp();", "__syncthreads();")), before[-200:]
    assert found >= 5
