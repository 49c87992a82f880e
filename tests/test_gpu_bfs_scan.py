"""bfs_distances through the scan level with rows that a block walks together:
the first top-down level after pulling is made of hubs, as many as a block
lists and more.  The rule that picks each level's way is replayed from the
distances, so that the test says itself that such a level occurs.  Exact."""

import numpy as np
import pytest

ALPHA, BETA, LONG_ROW, LONG_LIST, BLOCK = 14.0, 24.0, 1024, 64, 256
LIST, PULL, SCAN = "list", "pull", "scan"


def _levels(n, m, dist, deg):
    """(way, frontier) of every level."""
    front = np.flatnonzero(dist == 0)
    T = int(deg[front].sum())
    way = PULL if T > m / ALPHA else LIST
    left = m - (0 if way == PULL else T)
    out, level = [], 0
    while front.size and T:
        out.append((way, front))
        nxt = np.flatnonzero(dist == level + 1)
        T = int(deg[nxt].sum())
        pull = way == PULL and not (nxt.size < n / BETA and nxt.size < front.size)
        pull = pull or T > left / ALPHA
        way = PULL if pull else SCAN if way == PULL else LIST
        left -= 0 if pull else min(left, T)
        front, level = nxt, level + 1
    return out


def _case(orc, hubs, width, seed):
    """A random core, `hubs` nodes of `width` out-edges behind its last full
    level, with consecutive ids from the start of a block on, and a part that
    the search never meets, whose edges keep the hubs' below the limit."""
    rng = np.random.default_rng(seed)
    core, first = 20_000, 20_224
    s, d = rng.integers(0, core, (2, 20 * core)).astype(np.uint32)
    dist = orc.bfs_distances(orc.Topology(core, s, d), 0, "out")
    sizes = np.bincount(dist[dist >= 0])
    door = np.flatnonzero(dist == int(np.flatnonzero(sizes > 1_000)[-1]))
    assert first % BLOCK == 0 and door.size > 2 * hubs
    hub = first + np.arange(hubs)
    leaf0 = first + hubs
    leaves = leaf0 + rng.integers(0, 3_000, hubs * width)
    apart = leaf0 + 3_000
    m2 = int(ALPHA * hubs * width * 1.2)
    s2, d2 = apart + rng.integers(0, 5_000, (2, m2))
    return (apart + 5_000, np.r_[s, door[:hubs], np.repeat(hub, width), s2].astype(np.uint32),
            np.r_[d, hub, leaves, d2].astype(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("hubs, width", [(3, 1025), (64, 1100), (100, 1100), (100, 1300)])
def test_hubs_after_pulling(orc, hubs, width):
    from ursa_b200 import Topology, algo

    n, s, d = _case(orc, hubs, width, hubs + width)
    ref = orc.bfs_distances(orc.Topology(n, s, d), 0, "out")
    deg = np.bincount(s, minlength=n)
    scans = [f for way, f in _levels(n, s.size, ref, deg) if way == SCAN]
    long = [f[deg[f] > LONG_ROW] for f in scans]
    assert any(x.size == hubs and np.bincount(x // BLOCK).max() == hubs for x in long)
    assert np.array_equal(algo.bfs_distances(Topology.build(n, s, d), 0, "out"), ref)
    assert np.array_equal(algo.bfs_distances(Topology.build(n, d, s), 0, "in"), ref)
