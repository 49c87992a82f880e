"""dijkstra_distances across the device-driven rounds: graphs on both sides of
the edge count from which distances are reached in steps, weights that make
the steps many (log-normal over six decades), few (equal), none (zero, or an
infinite or NaN mean), ties at a step's end, long chains, hubs of many frontier
entries, every direction.  Bit-exact."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EDGES = 1 << 20


def _weights(kind, m, rng):
    if kind == "uniform":
        return rng.uniform(1.0, 10.0, m).astype(np.float32).astype(np.float64)
    if kind == "lognormal":
        return np.exp(rng.normal(0.0, 3.0, m))
    if kind == "ones":
        return np.ones(m)
    if kind == "zeros":
        return np.zeros(m)
    if kind == "tiny":
        return rng.uniform(1.0, 2.0, m) * 5e-324 * 1000
    w = rng.uniform(0.0, 1.0, m)
    w[rng.integers(0, m, m // 50 + 1)] = np.inf if kind == "with_inf" else np.nan
    return w


@pytest.mark.parametrize("kind", ["uniform", "lognormal", "ones", "zeros", "tiny", "with_inf"])
@pytest.mark.parametrize("m", [EDGES - 1, EDGES])
def test_random(orc, m, kind):
    from ursa_b200 import Topology, algo

    rng = np.random.default_rng(m)
    n = 50_000
    s, d = rng.integers(0, n, (2, m)).astype(np.uint32)
    d[: m // 8] = 7  # a hub
    s[m // 8 : m // 4] = 11
    w = _weights(kind, m, rng)
    g, o = Topology.build(n, s, d), orc.Topology(n, s, d)
    for direction in ("out", "in", "both"):
        got = algo.dijkstra_distances(g, w, 3, direction)
        ref = orc.dijkstra_distances(o, w, 3, direction)
        assert np.array_equal(got.view(np.uint64), ref.view(np.uint64)), direction


def test_nan_weights_reach_nothing_and_end():
    from ursa_b200 import Topology, algo

    rng = np.random.default_rng(1)
    n, m = 40_000, EDGES
    s, d = rng.integers(0, n, (2, m)).astype(np.uint32)
    w = np.full(m, np.nan)
    got = algo.dijkstra_distances(Topology.build(n, s, d), w, 5)
    assert got[5] == 0.0 and np.isinf(np.delete(got, 5)).all()


@pytest.mark.parametrize("n", [1, 2, 17, 40, 3000])
def test_chain(orc, n):
    from ursa_b200 import Topology, algo

    s, d = np.arange(n - 1, dtype=np.uint32), np.arange(1, n, dtype=np.uint32)
    w = np.random.default_rng(n).uniform(0.1, 5.0, n - 1)
    got = algo.dijkstra_distances(Topology.build(n, s, d), w, 0)
    assert np.array_equal(got, orc.dijkstra_distances(orc.Topology(n, s, d), w, 0))
