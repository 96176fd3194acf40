"""Kernels that reach into another block's shared memory: every block of the
cluster arrives at the cluster barrier before, and waits for the others right
ahead of, the first such access.  Without the wait the access is ordered by
luck alone, which no output shows, so the order is checked in the source."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vortexstark_b200", "csrc")


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


SOURCES = [p for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))) if "map_shared_rank" in _code(p)]


def test_there_is_such_a_kernel():
    assert SOURCES


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_remote_access_follows_the_start_barrier(path):
    code = _code(path)
    kernels = re.split(r"__global__", code)[1:]
    for k in (k for k in kernels if "map_shared_rank" in k):
        head = k[: k.index("map_shared_rank")]
        whole = head.find(".sync()")  # arrive and wait in one
        if whole < 0:
            assert 0 <= head.find("barrier_arrive()") < head.find("barrier_wait()")
