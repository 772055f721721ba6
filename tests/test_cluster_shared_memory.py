"""Kernels that reach the shared memory of another CTA of their cluster, read as source: a peer's shared memory may be
touched only between two cluster barriers, the first of which shows that every CTA has started and the last that none
has left."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "taurus_vap_gb300", "csrc")
BARRIER = re.compile(r"\bcluster\.(?:sync|barrier_wait)\(")


def kernels():
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", src):
            start = src.index("{", m.end())
            depth, end = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
                if depth == 0:
                    break
            body = src[start:end]
            if "map_shared_rank(" in body:
                name = re.findall(r"(\w+)\s*\(", src[m.end():start])
                out.append(pytest.param(body, id=next(k for k in name if k.endswith("_kernel"))))
    return out


def test_there_are_such_kernels():
    assert len(kernels()) >= 4


@pytest.mark.parametrize("body", kernels())
def test_remote_shared_memory_lies_between_cluster_barriers(body):
    remote = [m.start() for m in re.finditer(r"map_shared_rank\(", body)]
    barriers = [m.start() for m in BARRIER.finditer(body)]
    assert barriers and barriers[0] < remote[0]
    assert barriers[-1] > remote[-1]
    if "barrier_wait(" in body:  # every wait has its arrival before it
        assert body.count("barrier_wait(") == body.count("barrier_arrive(")
        assert body.index("barrier_arrive(") < body.index("barrier_wait(")
