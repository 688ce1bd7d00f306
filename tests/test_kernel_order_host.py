"""Rules of the kernels' control flow that no run can show to hold, read off their sources: what orders an allocation of tensor
memory against the kernels behind it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rivoli_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def code(path):
    s = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
    return re.sub(r"(?m)^#pragma[^\n]*$", "", s)


def closing(s, i):
    """Index behind the bracket that closes the one at ``i``."""
    depth = 0
    for j in range(i, len(s)):
        depth += s[j] in "([{"
        depth -= s[j] in ")]}"
        if depth == 0:
            return j + 1
    raise AssertionError("unbalanced")


def kernels(s):
    return [body(s, m.end()) for m in re.finditer(r"__global__", s)]


def body(s, i):
    i = s.index("{", closing(s, s.index("(", s.index("_kernel", i))))
    return s[i:closing(s, i)]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_dependents_start_behind_the_allocation(path):
    """An allocation of tensor memory waits without a limit for columns that other CTAs of the SM hold. A dependent that is let
    in before it could take them and then wait for this grid: no CTA may let its dependents start before it has its own."""
    for k in kernels(code(path)):
        alloc, trigger = k.find("tmem_alloc"), k.find("rv_grid_dep_trigger")
        if alloc >= 0 and trigger >= 0:
            between = k.find("__syncthreads()", alloc)
            assert alloc < between < trigger
