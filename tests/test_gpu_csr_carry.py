"""CSR builds whose sorts carry the other column, in both directions: endpoints
already on the device (a column that still arrives is gathered), one, two and
three radix passes, last tiles of one row, a part and all of a tile, and the
row count below which nothing is carried.  Exact, against a stable sort."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
M = 3 << 24
TILE = 4096


@pytest.mark.parametrize("n, m", [(200, M + 1), (257, M), (3_000, M), (65_536, M + 1_537), (65_537, M + TILE),
                                  (3_000, M - 1)])
@pytest.mark.parametrize("on_device", [True, False])
def test_against_stable_sort(n, m, on_device):
    import torch

    from ursa_b200 import Topology

    g = torch.Generator(device="cuda").manual_seed(n)
    src = (n * torch.rand(m, device="cuda", generator=g) ** 2).int().clamp_(max=n - 1)  # skewed: long and short runs
    dst = torch.randint(0, n, (m,), device="cuda", generator=g, dtype=torch.int32)
    if on_device:
        torch.cuda.synchronize()
        t = Topology.build_device(n, src, dst)
    else:
        t = Topology.build(n, src.cpu().numpy().view(np.uint32), dst.cpu().numpy().view(np.uint32))
    for key, other, adj in ((src, dst, t.out()), (dst, src, t.incoming())):
        order = torch.sort(key, stable=True).indices
        assert np.array_equal(adj.edge_ids, order.cpu().numpy().astype(np.uint32))
        assert np.array_equal(adj.targets, other[order].cpu().numpy().view(np.uint32))
        off = torch.cumsum(torch.bincount(key, minlength=n), 0).cpu().numpy()
        assert np.array_equal(adj.offsets, np.r_[0, off].astype(np.uint64))


def test_out_of_range_id_on_the_device_is_refused():
    import torch

    from ursa_b200 import Topology, UrsaGpuError

    src = torch.zeros(M, dtype=torch.int32, device="cuda")
    dst = torch.zeros(M, dtype=torch.int32, device="cuda")
    src[M // 5] = 3_000
    torch.cuda.synchronize()
    with pytest.raises(UrsaGpuError):
        Topology.build_device(3_000, src, dst)
