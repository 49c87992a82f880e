"""Sampled betweenness on graphs large enough that the source shuffle runs on the
device, around the number of steps from which it does: another source set, or
another order of it, would give other values.  The graphs have few edges, so
that the searches are short.  Relative error <= 1e-9, as for the other betweenness
tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 1 << 15  # steps past the sample from which the device takes them


@pytest.mark.parametrize("n, k, seed", [(STEPS, 1, 0), (STEPS + 1, 1, 0), (STEPS + 2, 1, 1), (STEPS + 64, 64, 7),
                                        (STEPS + 64, 65, 7), (STEPS + 4000, 4000, 2**64 - 1), (100_003, 300, None)])
def test_sources_against_oracle(orc, n, k, seed):
    from ursa_b200 import Topology, algo

    s, d = np.random.default_rng(n + k).integers(0, n, (2, 2 * n), dtype=np.uint32)
    sample = (k - 0.5) / n
    assert int(np.ceil(n * sample)) == k
    got = algo.betweenness(Topology.build(n, s, d), sample, seed)
    ref = orc.betweenness(orc.Topology(n, s, d), sample, seed)
    assert np.all(np.abs(got - ref) <= 1e-9 * np.maximum(np.abs(ref), 1e-300))
