"""Hand-overs between the CTAs of a pair, as the device sources state them.  A missing release is a race that no run can be trusted to
show, so the sources are read instead."""
import os
import re

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sage_b200", "csrc", "kernels")


def test_what_is_written_to_shared_memory_is_released_to_the_cluster():
    """The tiles that a CTA has split in place are read by matrix instructions of the pair's other CTA: the arrival that
    announces them has to release at cluster scope.  Only tmem_empty, which hands over no memory, may do with less."""
    text = open(os.path.join(KERNELS, "gemm_tc_device.inc")).read()
    helpers = dict(re.findall(r"void (mbar_arrive_remote\w*)\(unsigned cluster_addr\) \{\s*asm volatile\(\"([^\"]*)", text))
    assert helpers
    arrivals = 0
    for name in sorted(os.listdir(KERNELS)):
        if not name.endswith(".inc"):
            continue
        for helper, bar in re.findall(r"(mbar_arrive_remote\w*)\(peer_addr\(smem_u32\(&(\w+)", open(os.path.join(KERNELS, name)).read()):
            arrivals += 1
            assert ".release.cluster." in helpers[helper] or bar == "tmem_empty", (name, helper, bar)
    assert arrivals >= 3
