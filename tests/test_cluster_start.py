"""Every kernel that touches the shared memory of another CTA of its cluster waits on a cluster barrier first: the CTAs of a
cluster are scheduled together but do not begin together, and a peer's shared memory may be accessed only once the peer
runs.  A missing barrier shows in no result, so this reads the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ac4k_kernel_b200", "csrc")
# helpers that write to, or signal in, the shared memory of a CTA of the cluster
REMOTE = r"\b(st_shared_cluster_\w+|bulk_copy_to_cluster|mbar_arrive_cluster\w*|tma_load_\w*pair\w*|tc_commit_pair\w*)\("
BARRIER = r"\b(cluster_sync(_relaxed)?|cluster_wait)\("


def _kernels():
    """(file, name, body) of the kernels, comments taken out; a body reaches to the next kernel or host function"""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for part in re.split(r"(?=__global__)", text)[1:]:
            name = re.search(r"(\w+_kernel)\(", part).group(1)
            yield os.path.basename(path), name, re.split(r"\n}\n", part, maxsplit=1)[0]


@pytest.mark.parametrize("file,name,body", [k for k in _kernels() if re.search(REMOTE, k[2])], ids=lambda v: v if len(v) < 60 else "")
def test_barrier_before_a_peers_shared_memory(file, name, body):
    first = re.search(REMOTE, body).start()
    barrier = re.search(BARRIER, body)
    assert barrier and barrier.start() < first, f"{file}: {name} reaches a peer's shared memory before any cluster barrier"


def test_kernels_with_peers_are_found():
    assert {n for _, n, b in _kernels() if re.search(REMOTE, b)} >= {
        "nvfp4_quantize_flat_kernel", "linear_nvfp4_skinny_kernel", "linear_nvfp4_2cta_kernel"}
