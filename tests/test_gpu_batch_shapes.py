"""Batched graphs at the edges of the batch kernels' loops: edge counts around
a span of a components pass (four slots per thread), rows on both sides of
every in-degree class, lists longer than a warp, graphs without triangles,
edges or nodes.  Components and triangle counts exact, ranks within the bar of
the batch tests (max relative error 2e-6 at a fixed iteration count)."""

import numpy as np
import pytest

from cases import canon

pytestmark = pytest.mark.gpu


def _graphs():
    rng = np.random.default_rng(9)
    for m in (1023, 1024, 1025, 2047, 2049, 4095, 4097):
        yield m + 1, np.arange(m), np.arange(1, m + 1)  # paths: m oriented edges
    for k in (3, 32, 33, 34, 65):
        a, b = np.triu_indices(k, 1)
        yield k, a, b
    deg = [0, 1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 200]
    yield 300, rng.integers(13, 300, sum(deg)), np.repeat(np.arange(13), deg)  # a row of each class
    yield 5000, np.zeros(4999, int), np.arange(1, 5000)
    yield 20_000, *rng.integers(0, 20_000, (2, 60_000))
    yield 7, np.empty(0, int), np.empty(0, int)
    yield 0, np.empty(0, int), np.empty(0, int)


@pytest.mark.parametrize("config", [([4096, 16384, 57344], [256, 512, 1024], 32, 256), ([57344], [128], 5, 128)], ids=str)
def test_against_oracle(orc, config):
    from ursa_b200.batch import GraphBatch

    graphs = [(n, np.asarray(s, np.uint32), np.asarray(d, np.uint32)) for n, s, d in _graphs()]
    batch = GraphBatch.from_graphs(graphs)
    batch.set_config(*config)
    batch.run(max_iter=20, tol=0.0)
    res = batch.results()
    for g, (n, s, d) in enumerate(graphs):
        if n == 0:
            continue
        r, o = res.graph(g), orc.Topology(n, s, d)
        ref = orc.pagerank(o, 0.85, 20, 0.0)
        assert np.max(np.abs(r["pagerank"] - ref) / ref) <= 2e-6, g
        assert np.array_equal(r["components"], canon(orc.connected_components_weak(o))), g
        assert np.array_equal(r["triangles"], orc.triangle_count(o)), g
