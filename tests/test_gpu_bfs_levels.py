"""bfs_distances across the ways a level can go: searches that end inside and
past the first run of enqueued levels, hubs of many frontier entries, a core
that is pulled followed by a thin tail (the scan level), with rows that the
tail's block walks together and more of them than it lists.  Exact, every
direction."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _path(n):
    return n, np.arange(n - 1), np.arange(1, n), 0


def _core_and_tail(hubs, width, seed):
    """A dense core of 3,000 nodes, a few doors to `hubs` nodes of `width`
    out-edges each, whose ends continue as a path."""
    rng = np.random.default_rng(seed)
    core = 3_000
    s, d = rng.integers(0, core, (2, 20 * core))
    hub = core + np.arange(hubs)
    door = rng.integers(0, core, hubs)
    first = core + hubs
    leaves = first + rng.integers(0, 2 * width, hubs * width)
    n = first + 2 * width + 40
    tail = np.arange(n - 41, n - 1)
    src = np.r_[s, door, np.repeat(hub, width), leaves[:5], tail]
    dst = np.r_[d, hub, leaves, np.full(5, n - 41), tail + 1]
    return n, src, dst, int(s[0])


CASES = {
    **{f"path_{n}": _path(n) for n in (1, 2, 8, 9, 10, 25, 26, 300)},
    "star": (70_001, np.zeros(70_000, int), np.arange(1, 70_001), 0),
    "star_in": (70_001, np.arange(1, 70_001), np.zeros(70_000, int), 12),
    "hub_of_span": (600, np.r_[np.zeros(511, int), np.arange(1, 512)], np.r_[np.arange(1, 512), np.full(511, 599)], 0),
    "tail_few_hubs": _core_and_tail(3, 1025, 1),
    "tail_many_hubs": _core_and_tail(100, 1500, 2),
    "tail_short_rows": _core_and_tail(50, 40, 3),
    "source_without_edges": (50, [1, 2], [2, 3], 0),
    "self_loops": (5, [0, 0, 1, 2, 2], [0, 1, 1, 2, 3], 0),
}


@pytest.mark.parametrize("direction", ["out", "in", "both"])
@pytest.mark.parametrize("name", CASES)
def test_against_oracle(orc, name, direction):
    from ursa_b200 import Topology, algo

    n, s, d, source = CASES[name]
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    got = algo.bfs_distances(Topology.build(n, s, d), source, direction)
    assert np.array_equal(got, orc.bfs_distances(orc.Topology(n, s, d), source, direction))
