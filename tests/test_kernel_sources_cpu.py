"""Rules of the CUDA programming model that no run can show to be kept, checked on the sources."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xmvb-cpp_b200", "csrc")


def _kernels(text):
    """(line, body) of every __global__ function of a source."""
    for m in re.finditer(r"__global__", text):
        start = text.index("{", m.end())
        depth, end = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield text.count("\n", 0, m.start()) + 1, text[start:end]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_distributed_shared_memory_starts_and_ends_with_a_cluster_barrier(path):
    """A block's shared memory may be addressed by its cluster only while the block runs: a barrier of the
    cluster stands before the first remote address and after the last one."""
    with open(path) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for line, body in _kernels(text):
        first, last = body.find("map_shared_rank"), body.rfind("map_shared_rank")
        if first < 0:
            continue
        barriers = [m.start() for m in re.finditer(r"cluster\.sync\(\)", body)]
        assert barriers and barriers[0] < first, line
        assert barriers[-1] > last, line
