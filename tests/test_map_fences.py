"""Tensor maps in global memory (csrc/k_expert_umma.cu): what reads through them acquires them first, and the kernel that writes some releases them.
Read from the sources, since a missing fence shows on no input."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "maple_runtime_b200", "csrc")


def source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


@pytest.mark.parametrize("field", ["gate", "up", "down"])
def test_every_map_in_global_memory_is_acquired(field):
    s = source("k_expert_umma.cu")
    acquired = s.index("acquire(&e->%s)" % field)
    used = [m.start() for m in re.finditer(r"(tma_load_\dd\([^;]*|tma_prefetch_map\()&e\w->%s\b" % field, s)]
    assert len(used) >= 2
    assert acquired < s.index("__syncthreads()", acquired) < min(used)       # by any thread of the CTA, then a barrier, then the use
    assert "fence.proxy.tensormap::generic.acquire" in source("umma.cuh")


def test_the_tables_kernel_releases_its_maps():
    s = source("k_tables.cu")
    body = s[s.index("tables_kernel"):s.index('extern "C" void k_tables')]
    assert body.rindex("tma_release_maps()") > body.rindex("dst[i] = src[i]")
    assert "fence.proxy.tensormap::generic.release" in source("umma.cuh")
