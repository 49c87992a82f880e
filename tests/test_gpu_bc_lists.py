"""Betweenness where one block of the level kernels meets more rows of over
1,024 edges than it lists (32), so that the rest are left to their warps: long
in-rows on the way forward, long out-rows on the way back.  A warp takes the
nodes a grid's worth of warps apart, so the hubs' ids are 0..7 modulo that.
Sums in another order than the oracle's: relative error <= 1e-9, as for the
other betweenness tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
WARPS = 148 * 4 * 8
N = 40_000


def _hubs():
    v = np.arange(N)
    return v[v % WARPS < 8]


def _case(kind):
    rng = np.random.default_rng(7)
    hub = _hubs()
    assert hub.size > 2 * 32
    a, b = rng.integers(0, N, (2, 2 * N))
    row, other = np.repeat(hub, 1_100), rng.integers(0, N, hub.size * 1_100)
    if kind == "in":
        return np.r_[other, a], np.r_[row, b]
    # every node reaches every hub in two steps, by way of node 100: all of them
    # are on one level of every search
    to, fro = np.arange(N), np.full(N, 100)
    return np.r_[row, a, to, np.full(hub.size, 100)], np.r_[other, b, fro, hub]


@pytest.mark.parametrize("kind", ["in", "out"])
def test_against_oracle(orc, kind):
    from ursa_b200 import Topology, algo

    s, d = (np.asarray(x, np.uint32) for x in _case(kind))
    got = algo.betweenness(Topology.build(N, s, d), 3 / N, 11)
    ref = orc.betweenness(orc.Topology(N, s, d), 3 / N, 11)
    assert np.any(ref > 0)
    assert np.all(np.abs(got - ref) <= 1e-9 * np.maximum(np.abs(ref), 1e-300))
