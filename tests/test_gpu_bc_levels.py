"""Betweenness where its level kernels change course: searches deeper than
the levels kept (paths around 32 levels, a cycle of 120), rows around the length
that a whole block walks, more such rows than a block lists, batches of 1 to
65 sources, parallel edges and self-loops.  Sums in another order than the
oracle's: relative error <= 1e-9, as for the other betweenness tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _path(n):
    return n, np.arange(n - 1), np.arange(1, n)


def _hubs(lengths, n, seed, into):
    """Rows of the given lengths at the lowest ids (out- or in-rows) on a sparse random graph."""
    rng = np.random.default_rng(seed)
    hub = np.repeat(np.arange(len(lengths)), lengths)
    far = rng.integers(0, n, hub.size)
    s, d = (far, hub) if into else (hub, far)
    a, b = rng.integers(0, n, (2, 2 * n))
    return n, np.r_[s, a], np.r_[d, b]


CASES = {
    **{f"path_{n}": (*_path(n), None) for n in (30, 31, 32, 33, 34, 130)},
    "cycle_120": (120, np.arange(120), (np.arange(120) + 1) % 120, None),
    "deep_65_sources": (*_path(300), 0.2),
    "long_in_rows": (*_hubs([1023, 1024, 1025, 1026, 3000], 2_000, 1, True), 0.03),
    "long_out_rows": (*_hubs([1023, 1024, 1025, 1026, 3000], 2_000, 2, False), 0.03),
    "all_rows_long": (*_hubs([1100] * 300, 300, 3, True), 0.2),
    "parallel_and_loops": (40, np.tile(np.arange(40), 6), np.r_[np.arange(40), np.tile((np.arange(40) * 3 + 1) % 40, 5)], None),
    "one_source": (500, *np.random.default_rng(4).integers(0, 500, (2, 3000)), 0.001),
    "65_sources": (650, *np.random.default_rng(5).integers(0, 650, (2, 4000)), 0.1),
}


@pytest.mark.parametrize("name", CASES)
def test_against_oracle(orc, name):
    from ursa_b200 import Topology, algo

    n, s, d, sample = CASES[name]
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    got = algo.betweenness(Topology.build(n, s, d), sample, 7)
    ref = orc.betweenness(orc.Topology(n, s, d), sample, 7)
    assert np.all(np.abs(got - ref) <= 1e-9 * np.maximum(np.abs(ref), 1e-300))
