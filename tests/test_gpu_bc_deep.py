"""Betweenness of searches that outgrow the mask levels: the batch that meets
the limit goes on from there, later ones start without masks.  Layered graphs
with several shortest paths per pair (and parallel edges), batches of sources
spread over the layers, grids, a deep part beside a shallow one.  Sums in
another order than the oracle's: relative error <= 1e-9, as for the other
betweenness tests."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layers(width, depth, degree, seed):
    rng = np.random.default_rng(seed)
    s = np.repeat(np.arange(width * (depth - 1)), degree)
    d = (s // width + 1) * width + rng.integers(0, width, s.size)
    p = rng.permutation(width * depth)
    return width * depth, p[s], p[d]


def _grid(w, h):
    i = np.arange(w * h).reshape(h, w)
    s = np.r_[i[:, :-1].ravel(), i[:-1].ravel()]
    d = np.r_[i[:, 1:].ravel(), i[1:].ravel()]
    return w * h, np.r_[s, d], np.r_[d, s]


def _beside(a, b):
    return a[0] + b[0], np.r_[a[1], b[1] + a[0]], np.r_[a[2], b[2] + a[0]]


CASES = {
    "layers_33": (*_layers(8, 33, 5, 1), None),
    "layers_40_one_batch": (*_layers(30, 40, 3, 2), 0.05),
    "layers_70_two_batches": (*_layers(20, 70, 4, 3), 0.08),
    "grid_25": (*_grid(25, 25), None),
    "deep_beside_shallow": (*_beside(_layers(12, 50, 3, 4), _layers(300, 3, 8, 5)), 0.2),
}


@pytest.mark.parametrize("name", CASES)
def test_against_oracle(orc, name):
    from ursa_b200 import Topology, algo

    n, s, d, sample = CASES[name]
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    got = algo.betweenness(Topology.build(n, s, d), sample, 7)
    ref = orc.betweenness(orc.Topology(n, s, d), sample, 7)
    assert np.all(np.abs(got - ref) <= 1e-9 * np.maximum(np.abs(ref), 1e-300))
