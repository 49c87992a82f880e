"""dijkstra_distances where the distances lie in clusters with wide gaps, so
that a refill finds nothing below the threshold and jumps: gaps of many means,
gaps past which adding a step no longer moves the threshold, several clusters,
far nodes that fall meanwhile.  Bit-exact."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EDGES = 1 << 20

KINDS = {
    "two_levels": lambda r, m: np.where(r.random(m) < 0.995, 1e-12, 1.0),
    "huge_gap": lambda r, m: np.where(r.random(m) < 0.8, 1e-290, 1e290),
    "three_levels": lambda r, m: 10.0 ** (-12.0 * r.integers(0, 3, m)),
    "rare_in_the_sample": lambda r, m: np.where(np.arange(m) % 1024 == 1, 1e9, r.uniform(1e-9, 2e-9, m)),
    "zero_or_one": lambda r, m: (r.random(m) < 0.7).astype(np.float64),
}


@pytest.mark.parametrize("n", [30_000, 600_000])
@pytest.mark.parametrize("kind", KINDS)
def test_against_oracle(orc, kind, n):
    from ursa_b200 import Topology, algo

    rng = np.random.default_rng(n)
    s, d = rng.integers(0, n, (2, EDGES + 5)).astype(np.uint32)
    w = KINDS[kind](rng, s.size)
    g, o = Topology.build(n, s, d), orc.Topology(n, s, d)
    for source, direction in ((3, "out"), (int(s[9]), "both")):
        got = algo.dijkstra_distances(g, w, source, direction)
        ref = orc.dijkstra_distances(o, w, source, direction)
        assert np.array_equal(got.view(np.uint64), ref.view(np.uint64)), direction
