"""The residual and the dangling mass are exact sums (fixed point), rounded
once: on a graph without edges every node is dangling and every rank is the
base, so both follow from n equal terms in plain arithmetic.  Bit for bit, over
the sizes of the one-cluster kernel."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fx_sum(terms):
    """Terms truncated to multiples of 2^-96 and added as integers, the total
    rounded as its two 64-bit words are."""
    total = sum(int(float(t).as_integer_ratio()[0] * 2**96 // float(t).as_integer_ratio()[1]) * k for t, k in terms)
    hi, lo = total >> 64, total & (2**64 - 1)
    return (float(hi) * 2.0**64 + float(lo)) * 2.0**-96


@pytest.mark.parametrize("n", [3, 7, 49, 1_000, 3_001, 9_973, 14_336])
def test_edgeless_graph(n):
    from ursa_b200 import PageRankStats, Topology, algo

    damping, first = 0.85, 1.0 / n
    rank = first
    g = Topology.build(n, np.zeros(0, np.uint32), np.zeros(0, np.uint32))
    for iters in (1, 2, 3):
        new = (1.0 - damping) / n + damping * _fx_sum([(rank, n)]) / n
        delta = _fx_sum([(abs(new - rank), n)])
        rank = new
        st = PageRankStats()
        got = algo.pagerank(g, damping=damping, max_iter=iters, tol=0.0, stats=st)
        assert np.all(got == rank)
        assert st.iterations == iters and st.last_delta == delta
