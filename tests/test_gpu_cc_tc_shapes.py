"""Shapes at the edges of the components and triangle kernels' rules: graphs
on both sides of the edge count from which components are sampled, with and
without a component that holds most edges, long chains, long rows outside the
largest component; cliques whose oriented lists end on either side of every
table size.  Exact."""

import numpy as np
import pytest

from cases import canon

pytestmark = pytest.mark.gpu


def _grid(n, w):
    i = np.arange(n - 1)
    j = np.arange(n - w)
    return np.r_[i, j], np.r_[i + 1, j + w]


def _two_stars(n, copies):
    """Two stars (the smaller one's hub row is longer than a warp takes)."""
    m = 3 * n // 4
    s = np.r_[np.zeros(m - 1, np.int64), np.full(n - m - 1, m)]
    d = np.r_[np.arange(1, m), np.arange(m + 1, n)]
    return np.tile(s, copies), np.tile(d, copies)


def _graphs():
    rng = np.random.default_rng(3)
    n = 300_000
    up = np.arange(n - 1)
    a = rng.integers(0, n, 2 * n)
    block = np.minimum(n - 1, a // 50 * 50 + rng.integers(0, 50, 2 * n))
    big = rng.integers(0, n // 2, (2, n))  # one giant, the rest in pairs and singles
    pairs = np.arange(n // 2, n - 1, 3)
    yield "path_up", n, up, up + 1
    yield "path_down", n, up + 1, up
    yield "path_262143", 262_144, np.arange(262_143), np.arange(262_143) + 1  # below the sampled size
    yield "path_262144", 262_145, np.arange(262_144), np.arange(262_144) + 1  # the first sampled one
    yield "grid", n, *_grid(n, 512)
    yield "no_giant", n, a, block
    yield "giant_and_pairs", n, np.r_[big[0], pairs], np.r_[big[1], pairs + 1]
    yield "two_stars", 40_000, *_two_stars(40_000, 8)
    yield "in_stars", 40_000, *_two_stars(40_000, 8)[::-1]
    yield "self_loops", 100_000, np.arange(400_000) % 100_000, np.arange(400_000) % 100_000


@pytest.mark.parametrize("graph", list(_graphs()), ids=lambda g: g[0])
def test_components(orc, graph):
    from ursa_b200 import Topology, algo

    _, n, s, d = graph
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    ref = canon(orc.connected_components_weak(orc.Topology(n, s, d)))
    assert np.array_equal(algo.connected_components_weak(Topology.build(n, s, d)), ref)


@pytest.mark.parametrize("sizes", [(24, 25, 26, 27), (256, 257, 258), (1025, 1026), (1027, 40, 3)], ids=str)
def test_cliques_around_table_sizes(sizes):
    """A k-clique's oriented lists have 0..k-1 elements; every vertex closes
    C(k-1, 2) triangles.  Repeated until the graph takes the ranked path."""
    from ursa_b200 import Topology, algo

    rng = np.random.default_rng(sum(sizes))
    src, dst, want = [], [], []
    at = 0
    while at == 0 or sum(x.size for x in src) < 140_000:
        for k in sizes:
            a, b = np.triu_indices(k, 1)
            src.append(a + at)
            dst.append(b + at)
            want.append(np.full(k, (k - 1) * (k - 2) // 2))
            at += k
    perm = rng.permutation(at)
    s = perm[np.concatenate(src)].astype(np.uint32)
    d = perm[np.concatenate(dst)].astype(np.uint32)
    expect = np.empty(at, np.uint32)
    expect[perm] = np.concatenate(want)
    assert np.array_equal(algo.triangle_count(Topology.build(at, s, d)), expect)
