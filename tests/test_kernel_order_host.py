"""Rules of the kernels' control flow that no run can show to hold, read off their sources: what orders an allocation of tensor
memory against the kernels behind it, and what keeps the threads of a group together at their barriers."""
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


def statement(s, i):
    """End of the statement that begins at or behind ``i``."""
    while s[i].isspace():
        i += 1
    if s[i] == "{":
        return closing(s, i)
    m = re.compile(r"(?:for|if|while)\s*\(").match(s, i)
    if m:
        return statement(s, closing(s, m.end() - 1))
    while s[i] != ";":
        i = closing(s, i) if s[i] in "([{" else i + 1
    return i + 1


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


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_a_kernel_that_gave_up_lets_its_copies_land(path):
    """Copies into shared memory and MMAs that are still on their way would land in whatever CTA comes next."""
    for k in kernels(code(path)):
        for at in (m.start() for m in re.finditer("tmem_dealloc", k)):
            assert re.search(r"settle\([^)]*\);\s*tc::$", k[:at])


BARRIER = re.compile(r"__syncthreads|named_barrier|barrier_any|give_up|bar\.red|bar\.sync")
LOOP = re.compile(r"\b(?:for|while)\s*\(")


def loops(s):
    for m in LOOP.finditer(s):
        head = closing(s, m.end() - 1)
        yield s[m.end():head - 1], s[head:statement(s, head)]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_a_wait_that_gave_up_does_not_leave_a_loop_with_barriers(path):
    """Warps can differ on whether a bounded wait gave up. In a loop whose threads meet at a barrier they go on, or call the
    others, until the group has agreed to leave (``barrier_any``); a warp that just left would let the others wait for good."""
    for head, inside in loops(code(path)):
        if not BARRIER.search(inside):
            continue
        assert not re.search(r"\bok\b", head), head
        own = inside
        for h, nested in loops(inside):
            own = own.replace(nested, ";")
        assert not re.search(r"!\s*ok\s*\)\s*(?:\{\s*)?(?:break|return|continue)", own), own[:400]


@pytest.mark.parametrize("name", ["kv_append_paged_kernel", "step_dense_kernel", "step_prologue_kernel", "index_q_prepare_kernel", "index_score_mma_kernel"])
def test_a_kernel_whose_dependents_read_ahead_waits_first(name):
    """The kernels behind these read what is older than them before their own wait: the attention its q, its row list and counts and
    all pool rows but the step's new ones, the selection everything but the scores. It is complete only if the kernel between them lets
    its dependents in behind its own wait."""
    found = [body(s, m.start()) for s in map(code, SOURCES) for m in re.finditer(r"__global__[^;{]*?\b" + name + r"\s*\(", s)]
    assert len(found) == 1
    k = found[0]
    assert k.count("rv_grid_dep_wait()") == 1 and k.count("rv_grid_dep_trigger()") == 1
    assert k.index("rv_grid_dep_wait()") < k.index("rv_grid_dep_trigger()")
