"""Batch PageRank on both sides of the node count up to which a graph's rows are
taken without loading ahead: rows of every class (0, 1, 2, ... 32 lanes), fewer
rows than warps, more units than warps, in one batch.  f32 shares against the f64
oracle: 2^-24 each, which damping bounds by 1 / (1 - 0.85): 2e-6."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NEAR = 1024


def _graph(n, seed):
    rng = np.random.default_rng(seed)
    lengths = rng.choice([0, 1, 2, 3, 5, 9, 17, 40, 200, 600], n, p=[.2, .2, .1, .1, .1, .1, .1, .08, .015, .005])
    d = np.repeat(np.arange(n), lengths)
    return n, rng.integers(0, n, d.size), d


def test_against_oracle(orc):
    from ursa_b200.batch import GraphBatch

    sizes = [1, 2, 31, 33, 500, NEAR - 1, NEAR, NEAR + 1, 2_000, 5_000]
    graphs = [_graph(n, n) for n in sizes] + [(NEAR, np.zeros(0, int), np.zeros(0, int))]
    b = GraphBatch.from_graphs(graphs)
    for _ in range(2):
        b.run(max_iter=20, tol=0.0)
        res = b.results()
        for i, (n, s, d) in enumerate(graphs):
            ref = orc.pagerank(orc.Topology(n, np.asarray(s, np.uint32), np.asarray(d, np.uint32)), 0.85, 20, 0.0)
            got = res.graph(i)
            assert got["iterations"] == 20
            assert np.max(np.abs(got["pagerank"] - ref) / ref) <= 2e-6, n
    b.close()
