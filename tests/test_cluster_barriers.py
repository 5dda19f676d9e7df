"""Distributed shared memory may be accessed only once every thread block of the
cluster has started, which a cluster barrier ensures: in each device function
that maps another block's shared memory, a barrier comes first."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nihu_gb300", "csrc")
BARRIER = re.compile(r"\b\w+\.sync\(\)|\bbarrier_wait\(")


def functions(text):
    """The bodies of the file's kernels (everything from one __global__ to the next)."""
    text = re.sub(r"//[^\n]*", "", text)
    starts = [m.start() for m in re.finditer(r"^[^\n/]*__global__", text, re.M)] + [len(text)]
    return [text[a:b] for a, b in zip(starts, starts[1:])]


MAPPING = [(os.path.basename(f), i, body) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))
           for i, body in enumerate(functions(open(f).read())) if "map_shared_rank" in body]


def test_kernels_are_found():
    assert {f for f, _, _ in MAPPING} == {"lu32.cu", "solve_persistent.cu"} and len(MAPPING) >= 3


@pytest.mark.parametrize("name,i,body", MAPPING, ids=[f"{f}-{i}" for f, i, _ in MAPPING])
def test_barrier_before_the_first_remote_access(name, i, body):
    barrier = BARRIER.search(body)
    assert barrier and barrier.start() < body.index("map_shared_rank")
