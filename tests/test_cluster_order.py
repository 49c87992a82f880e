"""Distributed shared memory: a CTA may write another's shared memory only after
a cluster barrier has shown that it runs.  A missing barrier cannot be seen in
results (the others nearly always have started), so the order is read from the
source: in every cluster kernel a barrier is waited for before the first remote
access, and another one before the kernel ends."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ursa_b200", "csrc")
WAIT = r"cluster\.(?:barrier_wait|sync)\(\)"


def _bodies(text):
    """The body of each kernel with a compile-time cluster, comments taken out."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__ void __cluster_dims__", text):
        start = text.index("{", m.end())
        depth, i = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield text[start:i]


def test_cluster_barrier_before_remote_shared_memory():
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        for body in _bodies(open(os.path.join(CSRC, name)).read()):
            remote = [m.start() for m in re.finditer(r"map_shared_rank|\bpublish\(", body)]
            if not remote:
                continue
            seen += 1
            waits = [m.start() for m in re.finditer(WAIT, body)]
            assert waits and waits[0] < remote[0], f"{name}: remote write before a cluster barrier"
            assert waits[-1] > remote[-1], f"{name}: no barrier after the last remote write"
    assert seen
