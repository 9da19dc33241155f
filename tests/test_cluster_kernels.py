"""Kernels whose blocks write to one another's shared memory (csrc/*.cu): a
block of a cluster may be running before another has started, so the first
access to remote shared memory must come after a cluster barrier.  A missing
one shows on a device only by chance, so the order is checked in the source."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "parallellocallyoptimalapproximatesparsematrixinverses_b200" / "csrc"
REMOTE = re.compile(r"map_shared_rank\(|RemoteAddress\(")
BARRIER = re.compile(r"cluster\.sync\(\)|barrier\.cluster\.wait")


def _kernels():
    """(name, body) of every kernel that takes its cluster's handle."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for part in text.split("__global__")[1:]:
            body = part.split("\n}\n", 1)[0]
            if "this_cluster()" in body:
                yield re.search(r"(\w+Kernel)\(", body).group(1), body


def test_cluster_kernels_are_found():
    assert {name for name, _ in _kernels()} >= {"OrderedSumClusterKernel", "PcgSolveKernel"}


@pytest.mark.parametrize("name,body", [pytest.param(n, b, id=n) for n, b in _kernels()])
def test_a_barrier_precedes_the_first_remote_access(name, body):
    remote = REMOTE.search(body)
    barrier = BARRIER.search(body)
    assert remote is not None and barrier is not None
    assert barrier.start() < remote.start(), f"{name} reaches another block's shared memory before any cluster barrier"
