"""Closeness and many-source distances where the grid is cut into groups:
source counts on both sides of a batch of 256, fewer and more batches than
groups, a last batch of one source, and graphs with rows long enough to be
scanned in chunks.  Exact (integer folds, one division)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n, seed, hub=0):
    rng = np.random.default_rng(seed)
    s, d = rng.integers(0, n, (2, 5 * n))
    if hub:
        s = np.r_[s, rng.integers(0, n, hub)]
        d = np.r_[d, np.full(hub, n // 3)]
    return s.astype(np.uint32), d.astype(np.uint32)


@pytest.mark.parametrize("n, hub", [(1, 0), (255, 0), (256, 0), (257, 200), (512, 0), (513, 3000), (4097, 5000), (9000, 65)])
def test_closeness_and_distances(orc, n, hub):
    from ursa_b200 import Topology, algo

    s, d = _graph(n, n + hub, hub)
    g, o = Topology.build(n, s, d), orc.Topology(n, s, d)
    assert np.array_equal(algo.closeness(g), orc.closeness(o))
    sources = np.random.default_rng(1).integers(0, n, min(n, 600))
    rows = algo.bfs_distances_multi(g, sources, "both")
    for i in {0, len(sources) // 2, len(sources) - 1}:
        assert np.array_equal(rows[i], algo.bfs_distances(g, int(sources[i]), "both"))
