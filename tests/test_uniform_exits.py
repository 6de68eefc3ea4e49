"""A kernel that gives up because a wait ran out must take its whole CTA along.  Threads that each read the error flag
from global memory can see it differently, and those that go on then meet warp votes and barriers that the others
never reach.  The decision has to come from shared memory behind a barrier, or from a vote of the block.  (Such an
exit cannot be forced on a GPU without a wait that runs out; the sources are read instead.)"""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bsr_b200", "csrc")
# "if (flag) return" or "return flag == 0" on a volatile read of a global error flag, outside a vote
LONE = re.compile(r"if \(\*\(volatile int \*\)(?:a\.)?err\)\s*return|return \*(?:\(volatile int \*\)(?:a\.)?err|verr) [!=]= 0")


def test_no_thread_leaves_alone():
    files = glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))
    assert len(files) > 15
    found = {os.path.basename(f): LONE.findall(open(f).read()) for f in files}
    assert not {f: m for f, m in found.items() if m}


def test_the_pattern_finds_them():
    for line in ("        if (*(volatile int *)a.err) return;", "    return *(volatile int *)err == 0;", "    return *verr == 0;"):
        assert LONE.search(line)
    assert not LONE.search("    return __syncthreads_or(*(volatile int *)err) == 0;")
