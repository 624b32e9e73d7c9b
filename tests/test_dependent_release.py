"""A kernel that lets its dependents start early (releaseDependent) and uses
tensor memory must hold its own columns first: a dependent block that allocates
on the same SM would otherwise take them, wait for this kernel's end, and be
waited for.  Read from the sources, since a run that shows the fault hangs."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "digholo_b200", "csrc")


def kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
        depth, start = 0, text.index("{", m.end())
        for i in range(start, len(text)):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            if depth == 0:
                yield m.group(1), re.sub(r"//[^\n]*", "", text[start:i])
                break


@pytest.mark.parametrize("file", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_release_follows_the_allocation(file):
    for name, body in kernels(open(os.path.join(CSRC, file)).read()):
        release, alloc = body.find("releaseDependent("), body.find("tcgen05.alloc")
        if release < 0 or alloc < 0:
            continue
        assert alloc < release, "%s releases its dependents before it has its tensor memory" % name
        assert "__syncthreads()" in body[alloc:release], "%s: the block's threads release before the allocating warp is done" % name
