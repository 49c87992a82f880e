"""CSR builds around the row count from which the sorted column travels with
the keys, with one to three radix passes, a last tile of one row, and out of
range ids: both CSRs against a stable argsort.  Exact."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
M = 3 << 24


@pytest.mark.parametrize("n, m", [(200, M), (3_000, M - 1), (70_001, M + 4097)])
def test_against_argsort(n, m):
    from ursa_b200 import Topology

    rng = np.random.default_rng(n)
    src = (n * rng.random(m, np.float32) ** 2).astype(np.uint32)  # skewed: long and short runs
    dst = rng.integers(0, n, m, dtype=np.uint32)
    src[src >= n] = n - 1
    g = Topology.build(n, src, dst)
    for key, other, adj in ((src, dst, g.out()), (dst, src, g.incoming())):
        order = np.argsort(key, kind="stable")
        assert np.array_equal(adj.edge_ids, order.astype(np.uint32))
        assert np.array_equal(adj.targets, other[order])
        assert np.array_equal(adj.offsets, np.concatenate([[0], np.cumsum(np.bincount(key, minlength=n))]).astype(np.uint64))


def test_out_of_range_id_is_refused():
    from ursa_b200 import Topology, UrsaGpuError

    src = np.zeros(M, np.uint32)
    dst = np.zeros(M, np.uint32)
    dst[M // 3] = 70_000
    with pytest.raises(UrsaGpuError):
        Topology.build(70_000, src, dst)
