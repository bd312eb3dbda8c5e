"""Self maps whose hash table exceeds the L2, which go over the occupancy index, against the general builder (which the
oracle covers): dimensions, tensor strides, offsets inside and beyond the reach of the index, negative coordinates, clouds
dense enough for the index and clouds that overflow it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,n,extent,kernel,dilation,stride", [
    (3, 1_970_000, 110, 3, 1, 1), (3, 2_000_001, 5000, 3, 1, 1), (3, 1_970_000, 110, 5, 1, 1), (3, 1_970_000, 100, 3, 3, 1),
    (3, 1_980_000, 100, 3, 1, 4), (3, 1_980_000, 100, 3, 2, 6), (2, 1_970_000, 1100, 3, 1, 2), (4, 2_100_003, 36, 3, 1, 1),
    (5, 1_970_000, 16, 3, 1, 2), (1, 1_970_000, 1_500_000, 9, 1, 1),
])
def test_large_self_map_equals_general_builder(D, n, extent, kernel, dilation, stride):
    from riemannengine_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(D * 1000 + n)
    c = torch.cat([torch.randint(0, 3, (3 * n, 1), generator=g, device="cuda"),
                   torch.randint(-extent // 2, extent - extent // 2, (3 * n, D), generator=g, device="cuda") * stride], 1)
    c = torch.unique(c, dim=0)
    c = c[torch.randperm(c.size(0), generator=g, device="cuda")][:n].int().contiguous()
    assert c.size(0) == n
    table = ops.table_build(c)
    off = ops.region_offsets(0, [kernel] * D, [dilation] * D, [stride] * D)
    a = ops.kmap_build(table, table.coords, off)
    b = ops.kmap_build(table, table.coords, off, self_map=True)
    assert torch.equal(a.nbr, b.nbr) and torch.equal(a.offset_ptr, b.offset_ptr)
    if kernel > 3 or D > 4:
        return
    (pa, xa, ya), (pb, xb, yb) = a.pairs(), b.pairs()
    assert torch.equal(torch.as_tensor(pa), torch.as_tensor(pb)) and xa.numel() == xb.numel() == int(a.offset_ptr[-1])
    for k in (0, off.shape[0] // 2, off.shape[0] - 1):
        lo, hi = int(a.offset_ptr[k]), int(a.offset_ptr[k + 1])
        order_a, order_b = ya[lo:hi].argsort(), yb[lo:hi].argsort()
        assert torch.equal(xa[lo:hi][order_a], xb[lo:hi][order_b]) and torch.equal(ya[lo:hi][order_a], yb[lo:hi][order_b])
