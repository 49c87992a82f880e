"""Weak components where the first link's trees are chains that blocks collapse
tile by tile (256 nodes): paths up and down the ids, strides around a tile,
rings, trees, node counts around a tile's end; and both sides of the edge counts
from which the passes are sampled.  Exact (minimum member ids)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TILE, SAMPLED = 256, 1 << 18


def _stride(n, k, down):
    a, b = np.arange(n - k), np.arange(k, n)
    return (n, b, a) if down else (n, a, b)


def _ring(n, k):
    s = np.repeat(np.arange(n), k)
    return n, s, (s + np.tile(np.arange(1, k + 1), n)) % n


def _random(n, m, seed):
    rng = np.random.default_rng(seed)
    return n, rng.integers(0, n, m), rng.integers(0, n, m)


def _tree(n, down):
    a, b = np.arange(1, n), (np.arange(1, n) - 1) // 2
    return (n, a, b) if down else (n, b, a)


def _pieces(n, length):
    """Paths of `length` nodes, from high ids to low ones."""
    v = np.arange(n)
    v = v[v % length != 0]
    return n, v, v - 1


N = 2 * SAMPLED
CASES = {
    **{f"stride_{k}_{'down' if d else 'up'}": _stride(N + 1, k, d) for k in (1, 2, 255, 256, 257) for d in (0, 1)},
    **{f"path_tile_{x:+d}": _stride(SAMPLED + TILE + x, 1, True) for x in (-1, 0, 1, 2)},
    "ring_1": _ring(N, 1),
    "ring_8": _ring(100_003, 8),
    "tree_up": _tree(N, True),
    "tree_down": _tree(N, False),
    "pieces_300": _pieces(N, 300),
    "pieces_256": _pieces(N, 256),
    **{f"sparse_{x:+d}": _random(400_000, 300_000 + x, x + 9) for x in (-1, 0, 1)},
    **{f"few_edges_{x:+d}": _random(100_000, SAMPLED + x, x + 5) for x in (-1, 0)},
    "two_per_node": _random(300_000, 600_000, 3),
}


@pytest.mark.parametrize("name", CASES)
def test_against_oracle(orc, name):
    from ursa_b200 import Topology, algo

    n, s, d = CASES[name]
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    got = algo.connected_components_weak(Topology.build(n, s, d))
    ref = orc.connected_components_weak(orc.Topology(n, s, d))
    low = np.full(n, n, np.int64)
    np.minimum.at(low, ref, np.arange(n))
    assert np.array_equal(got, low[ref])
