"""The traffic figure of the bench line belongs to the kernel sources it was captured
from: every file the profiled sweep is compiled from is in its digest."""
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ouranos_gb300", "csrc")


def _includes(name, seen):
    if name in seen:
        return seen
    seen.add(name)
    with open(os.path.join(CSRC, name)) as f:
        for inc in re.findall(r'#include "([\w.]+)"', f.read()):
            if os.path.exists(os.path.join(CSRC, inc)):
                _includes(inc, seen)
    return seen


def test_digest_covers_the_profiled_kernels_sources():
    sys.path.insert(0, ROOT)
    import bench
    used = _includes("sweep_lane_df64.cu", set())
    # (internal.h holds the whole library's host declarations)
    assert used - {"internal.h"} <= set(bench.SWEEP_SOURCES)
