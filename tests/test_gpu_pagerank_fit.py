"""Which kernel takes an unweighted PageRank of a skewed graph: one cluster where
every CTA keeps its long rows' sources in shared memory, the large kernel (which
builds a plan on the topology) elsewhere.  The rule is replayed here on the
in-degrees, and both sides are compared with the f64 oracle; f32 shares carry a
relative rounding of 2^-24 each, which damping bounds by 1 / (1 - 0.85): 2e-6."""

import numpy as np
import pytest

SMEM, CTAS, DIRECT, PIECE = 224 * 1024, 8, 64, 128


def _bytes(n, rows, longs, pieces):
    return (8 * n + 18 * rows + 4 + 7) // 8 * 8 + 10 * pieces + 10 * (longs + 1) + 2 * (PIECE + 2) * pieces


def _exact(indeg):
    n, m = indeg.size, int(indeg.sum())
    cost = max(1, -(-m // n))
    key = np.r_[0, np.cumsum(indeg)][:-1] + np.arange(n) * cost
    cut = [int(np.searchsorted(key, c * (n * cost + m) // CTAS)) for c in range(CTAS)] + [n]
    for a, b in zip(cut, cut[1:]):
        long = indeg[a:b][indeg[a:b] > DIRECT]
        if _bytes(n, b - a, long.size, int((-(-long // PIECE)).sum())) > SMEM:
            return False
    return True


def _any_fits(n, m):
    longs = m // (DIRECT + 1)
    return _bytes(n, n // 4 + 2, longs, longs + m // PIECE) <= SMEM


def _one_cluster(indeg):
    n, m = indeg.size, int(indeg.sum())
    return n <= 14_336 and m <= 1 << 18 and (_any_fits(n, m) or _exact(indeg))


def test_bound_implies_fit():
    """The sizes that are not looked at fit whatever the in-degrees."""
    rng = np.random.default_rng(1)
    for _ in range(400):
        n = int(rng.integers(1, 14_337))
        m = int(rng.integers(1, 1 << 18))
        if not _any_fits(n, m):
            continue
        shapes = [np.full(m // 65, 65), np.full(m // 129, 129), np.array([m])]
        for s in shapes:
            indeg = np.zeros(n, np.int64)
            indeg[: min(n, s.size)] = s[:n]
            assert _exact(indeg)


def _hubs(n, hub_rows, hub_edges, others):
    rng = np.random.default_rng(n + hub_edges)
    d = np.r_[rng.choice(hub_rows, hub_edges), rng.integers(0, n, others)]
    return n, rng.integers(0, n, d.size), rng.permutation(d)


CASES = {
    "hub_fits": _hubs(4_000, [7], 70_000, 20_000),
    "hub_does_not": _hubs(4_000, [7], 100_000, 20_000),
    "two_hubs_one_cta": _hubs(14_000, [0, 1], 200_000, 60_000),
    "hubs_over_ctas": _hubs(14_000, np.arange(10) * 1_400, 200_000, 60_000),
    "hubs_over_ctas_fit": _hubs(8_000, np.arange(16) * 500, 150_000, 60_000),
    "eight_rows": _hubs(8, np.arange(8), 200_000, 60_000),
    "rows_of_66": (12_000, np.arange(66 * 3_900) % 12_000, np.repeat(np.arange(3_900) * 3, 66)),
    "short_and_long": _hubs(9_000, np.arange(0, 9_000, 40), 30_000, 100_000),
    "last_rows_long": _hubs(5_000, np.arange(4_980, 5_000), 90_000, 10_000),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_route_and_ranks(orc, name):
    from ursa_b200 import PageRankStats, Topology, _lib, algo

    n, s, d = CASES[name]
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    g = Topology.build(n, s, d)
    before = _lib.load().ursa_gpu_topo_device_bytes(g.handle)
    st = PageRankStats()
    got = algo.pagerank(g, max_iter=25, tol=0.0, stats=st)
    planned = _lib.load().ursa_gpu_topo_device_bytes(g.handle) != before
    assert planned != _one_cluster(np.bincount(d, minlength=n))
    ref = orc.pagerank(orc.Topology(n, s, d), 0.85, 25, 0.0)
    assert st.iterations == 25 and np.max(np.abs(got - ref) / ref) <= 2e-6
    assert np.array_equal(algo.pagerank(g, max_iter=25, tol=0.0), got)
