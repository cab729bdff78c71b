"""A block of a cluster may write another block's shared memory only once that
block is known to have started, that is after a barrier of the whole cluster
(CUDA C++ Programming Guide, distributed shared memory).  Checked on the source:
a missing barrier shows on no GPU run that happens to start the blocks together."""
import glob
import os
import re

from tests.util import ROOT

BARRIER = r"team_barrier<TEAM_CLUSTER>\s*\(|cluster_sync\s*\("
REMOTE = r"cluster_put\s*\("


def _kernels():
    for path in sorted(glob.glob(os.path.join(ROOT, "schrodingersem_gb300", "csrc", "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", src):
            start = src.index("{", m.end())
            depth, end = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
            yield os.path.basename(path), src[start:end]


def test_kernels_synchronise_the_cluster_before_remote_stores():
    seen = 0
    for name, body in _kernels():
        store = re.search(REMOTE, body)
        if not store:
            continue
        seen += 1
        barrier = re.search(BARRIER, body)
        assert barrier and barrier.start() < store.start(), name
    assert seen >= 1
