"""PageRank around the limits of the one-cluster kernel: node and edge counts
on both sides of them, rows on both sides of every length class (64 and 128
in-edges, 32 pieces), fewer nodes than CTAs, no iterations.  Against the f64
oracle; f32 shares carry a relative rounding of 2^-24 each, which a pull
iteration averages and damping bounds by 1 / (1 - 0.85): 2e-6.  Runs to a tolerance use the default one: the
shares' rounding (about 1e-8 in the residual) must stay well below it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MAX_NODES, MAX_EDGES = 14_336, 1 << 18
rng = np.random.default_rng(17)


def _random(n, m):
    return n, rng.integers(0, n, m), rng.integers(0, n, m)


def _rows(n, lengths):
    """A row of every given in-degree, sources cycling over all nodes."""
    dst = np.repeat(np.arange(len(lengths)) * (n // len(lengths)), lengths)
    return n, np.arange(dst.size) * 7 % n, dst


CASES = {
    "one_node": (1, [0], [0]),
    "five_nodes": (5, [0, 1, 2, 3], [1, 2, 3, 0]),
    "seven_isolated": (7, [], []),
    "max_nodes": _random(MAX_NODES, 100_000),
    "above_max_nodes": _random(MAX_NODES + 1, 100_000),
    "max_edges": _random(9_000, MAX_EDGES),
    "above_max_edges": _random(9_000, MAX_EDGES + 1),
    "lengths": _rows(10_000, [8, 9, 63, 64, 65, 127, 128, 129, 256, 257, 4095, 4096, 4097, 4224, 12_289]),
    "max_nodes_one_hub": _rows(MAX_NODES, [MAX_EDGES]),
    "long_rows": _rows(4_000, [65] * 2_000),
    "dangling": (6_000, rng.integers(0, 3_000, 20_000), rng.integers(0, 6_000, 20_000)),
}


@pytest.mark.parametrize("max_iter, tol", [(0, 1e-6), (1, 0.0), (25, 0.0), (100, 1e-6)])
@pytest.mark.parametrize("name", CASES)
def test_against_oracle(orc, name, max_iter, tol):
    from ursa_b200 import PageRankStats, Topology, algo

    n, s, d = CASES[name]
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    st = PageRankStats()
    g = Topology.build(n, s, d)
    got = algo.pagerank(g, max_iter=max_iter, tol=tol, stats=st)
    ref, iters = orc.pagerank(orc.Topology(n, s, d), 0.85, max_iter, tol, return_iters=True)
    assert st.iterations == iters or (tol > 0 and abs(int(st.iterations) - iters) == 1)
    assert np.max(np.abs(got - ref) / ref) <= 2e-6
    assert np.array_equal(algo.pagerank(g, max_iter=max_iter, tol=tol), got)  # without statistics, and repeatable
