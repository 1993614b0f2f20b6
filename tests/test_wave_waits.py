"""The bounded waits of the wavefront kernels are a warp's decision: the lanes'
own looks at the error flag may differ, and a lane that left alone would leave
the others in a warp vote.  (The device side of the same is
messi_selftest_bounded_wait, tests/test_gpu_wave_waits.py.)"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "messi_gb300", "csrc")


def test_every_wait_of_a_warp_gives_up_as_one():
    with open(os.path.join(CSRC, "scfg.cu")) as f:
        src = f.read()
    assert len(re.findall(r"\bwarp_keep_waiting\(", src)) >= 4
    assert not re.findall(r"\bkeep_waiting\(", src)
