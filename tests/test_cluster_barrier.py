"""Distributed shared memory on the CPU: a block of a cluster may touch another
block's shared memory only once that block has started, which only a barrier of
the cluster establishes; and a block may leave only after the others' last
access to its own.  Read from the sources: every kernel that maps another
block's shared memory passes a cluster barrier before the first such access,
outside any loop, and one after the last.  (A kernel without the barrier is
not run: the access would be a fault.)"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "4d-image-segmentation-algorithm_gb300", "csrc")


def kernels():
    """(file, name, body) of every kernel that maps another block's shared memory"""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void[^;{]*?(\w+)\s*\(Geo[^{;]*\{", src):
            end, depth = m.end(), 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
            body = src[m.end():end]
            if "map_shared_rank" in body:
                yield os.path.basename(path), m.group(1), body


FOUND = list(kernels())


def test_the_rescale_is_found():
    assert ("ss4d_kernels_ref.cu", "k_rescale_balls") in [(f, n) for f, n, _ in FOUND]


@pytest.mark.parametrize("file,name,body", FOUND, ids=[n for _, n, _ in FOUND])
def test_cluster_barrier_before_and_after_remote_access(file, name, body):
    first, last = body.index("map_shared_rank"), body.rindex("map_shared_rank")
    before = body[:first].rfind("cluster.sync()")
    assert before >= 0, f"{file}: {name} reaches another block before a cluster barrier"
    # at the kernel's top level: every block passes it, once, before any loop
    assert body[:before].count("{") == body[:before].count("}")
    assert "cluster.sync()" in body[last:]
