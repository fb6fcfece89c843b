"""Programmatic launches (csrc/launch.cuh): what a kernel reads before its own wait was written two kernels ago, which holds only if no kernel in between lets its successor
start before its own wait is over.  The first trigger in a CTA counts for the whole CTA, so no thread may trigger that has not waited.  Read from the sources, since the race shows on no input."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "maple_runtime_b200", "csrc")
FILES = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def source(name):
    s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    return re.sub(r"__launch_bounds__\([^)]*\)", "", re.sub(r"/\*.*?\*/", "", s, flags=re.S))


def triggers(s):
    """(kernel, does the triggering thread wait right before) for every trigger"""
    out = []
    for m in re.finditer(r"pdl_trigger\(\);", s):
        front = s[:m.start()].rstrip()
        waited = front.endswith("pdl_wait();") and front[:-len("pdl_wait();")].rstrip()[-1] in ";{}"      # a statement of its own, not the body of an if
        out.append((re.findall(r"\bvoid\s+(\w+)\(", front)[-1], waited))
    return out


@pytest.mark.parametrize("name", [f for f in FILES if "pdl_trigger();" in source(f)])
def test_who_triggers_has_waited(name):
    s = source(name)
    for kernel, waited in triggers(s):
        if not waited:      # only where everything before the kernel is complete when it starts: launched plainly
            assert re.search(r"launch_k\(%s\b" % kernel, s) and not re.search(r"launch_(pdl|clusters?)\(%s\b" % kernel, s), kernel


def test_the_check_sees_a_trigger_without_a_wait():
    assert triggers("__global__ void k(int n) { if (n) pdl_wait(); pdl_trigger(); }") == [("k", False)]
    assert triggers("__global__ void k(int n) { if (n) { pdl_wait(); pdl_trigger(); } }") == [("k", True)]
