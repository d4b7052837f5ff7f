"""Shared memory of another CTA may be accessed only once every CTA of the
cluster is known to have started: each kernel that maps a peer's shared memory
waits on the cluster's barrier before it does so first."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _kernels():
    for path in sorted(glob.glob(os.path.join(ROOT, "rustscan_b200", "csrc", "*.cu"))):
        with open(path) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"__global__", text):
            body = text[text.index("{", m.end()):]
            yield os.path.basename(path), body[:body.index("\n}\n")]


def test_cluster_barrier_precedes_peer_access():
    users = [(path, body) for path, body in _kernels() if "map_shared_rank" in body]
    assert users
    for path, body in users:
        wait = re.search(r"cluster\.(sync|barrier_wait)\(\)", body)
        assert wait and wait.start() < body.index("map_shared_rank"), path
