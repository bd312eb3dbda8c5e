"""Self maps whose hash table takes most of the L2, which may go over the occupancy index, against the general builder
(which the oracle covers): dimensions, tensor strides, offsets inside and beyond the reach of the index, negative coordinates,
clouds dense enough for the index and too thin for it, rows in random and in spatial order - and which way they went."""
import pytest
import torch

pytestmark = pytest.mark.gpu


IN_USE, NOT_CHOSEN, FULL = -1, 0, 1


def _index_state(kmap):
    """The word of the build's workspace that says what became of the index (csrc/rmn_kmap_blocks.cuh)."""
    n, K = kmap.n_query, kmap.K
    counts = ((K * ((n + 255) // 256) + K + 64) * 4 + 255) // 256 * 256
    at = counts + (n // 8 + 64) * 32 + 4
    return kmap.workspace[at:at + 4].cpu().view(torch.int32).item()


# (a stride that is no power of two leaves the blocks thin; order: "random", or "sorted" by coordinates; index: what
# becomes of it, None below three dimensions, where there is none)
@pytest.mark.parametrize("D,n,extent,kernel,dilation,stride,order,index", [
    (3, 1_970_000, 110, 3, 1, 1, "random", IN_USE), (3, 2_000_001, 5000, 3, 1, 1, "random", NOT_CHOSEN),
    (3, 1_970_000, 110, 5, 1, 1, "random", IN_USE), (3, 1_970_000, 100, 3, 3, 1, "random", IN_USE),
    (3, 1_980_000, 100, 3, 1, 4, "random", IN_USE), (3, 1_980_000, 100, 3, 2, 6, "random", NOT_CHOSEN),
    (2, 1_970_000, 1100, 3, 1, 2, "random", None), (4, 2_100_003, 36, 3, 1, 1, "random", IN_USE),
    (5, 1_970_000, 16, 3, 1, 2, "random", IN_USE), (1, 1_970_000, 1_500_000, 9, 1, 1, "random", None),
    (3, 2_600_001, 110, 3, 1, 1, "sorted", NOT_CHOSEN), (3, 1_970_003, 250, 3, 1, 1, "random", NOT_CHOSEN),
])
def test_large_self_map_equals_general_builder(D, n, extent, kernel, dilation, stride, order, index):
    from riemannengine_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(D * 1000 + n)
    c = torch.cat([torch.randint(0, 3, (3 * n, 1), generator=g, device="cuda"),
                   torch.randint(-extent // 2, extent - extent // 2, (3 * n, D), generator=g, device="cuda") * stride], 1)
    c = torch.unique(c, dim=0)
    c = c[torch.randperm(c.size(0), generator=g, device="cuda")][:n]
    c = (torch.unique(c, dim=0) if order == "sorted" else c).int().contiguous()
    assert c.size(0) == n
    table = ops.table_build(c)
    off = ops.region_offsets(0, [kernel] * D, [dilation] * D, [stride] * D)
    a = ops.kmap_build(table, table.coords, off)
    b = ops.kmap_build(table, table.coords, off, self_map=True)
    assert torch.equal(a.nbr, b.nbr) and torch.equal(a.offset_ptr, b.offset_ptr)
    assert index is None or _index_state(b) == index
    if kernel > 3 or D > 4:
        return
    (pa, xa, ya), (pb, xb, yb) = a.pairs(), b.pairs()
    assert torch.equal(torch.as_tensor(pa), torch.as_tensor(pb)) and xa.numel() == xb.numel() == int(a.offset_ptr[-1])
    for k in (0, off.shape[0] // 2, off.shape[0] - 1):
        lo, hi = int(a.offset_ptr[k]), int(a.offset_ptr[k + 1])
        order_a, order_b = ya[lo:hi].argsort(), yb[lo:hi].argsort()
        assert torch.equal(xa[lo:hi][order_a], xb[lo:hi][order_b]) and torch.equal(ya[lo:hi][order_a], yb[lo:hi][order_b])


def test_index_that_turns_out_too_small_gives_way_to_the_table():
    """Rows that the choice samples lie in full blocks, all others thinly: chosen, then full."""
    from riemannengine_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    n = 2_000_003
    thin = torch.randint(16, 4000, (n + 200_000, 3), generator=g, device="cuda")
    thin = torch.unique(thin, dim=0)
    c = thin[torch.randperm(thin.size(0), generator=g, device="cuda")][:n]
    dense = torch.cartesian_prod(*[torch.arange(16, device="cuda")] * 3)   # 64 blocks of 64 voxels
    by_block = dense[((dense // 4) * torch.tensor([16, 4, 1], device="cuda")).sum(1).argsort(stable=True)]
    at = torch.arange(64, device="cuda") * n // 64                         # one voxel of every block where the choice looks
    c[at] = by_block[::64]
    rest = torch.ones(4096, dtype=torch.bool, device="cuda")
    rest[::64] = False
    free = torch.arange(n, device="cuda")[~torch.isin(torch.arange(n, device="cuda"), at)]
    c[free[torch.randperm(free.numel(), generator=g, device="cuda")[:4032]]] = by_block[rest]
    coords = torch.cat([torch.zeros((n, 1), dtype=torch.long, device="cuda"), c], 1).int().contiguous()
    table = ops.table_build(coords)
    assert table.n_unique == n
    off = ops.region_offsets(0, [3] * 3, [1] * 3, [1] * 3)
    a, b = ops.kmap_build(table, table.coords, off), ops.kmap_build(table, table.coords, off, self_map=True)
    assert _index_state(b) == FULL
    assert torch.equal(a.nbr, b.nbr) and torch.equal(a.offset_ptr, b.offset_ptr)


def _cloud(D, n, extent, stride, order, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.cat([torch.randint(0, 3, (3 * n, 1), generator=g, device="cuda"),
                   torch.randint(-extent // 2, extent - extent // 2, (3 * n, D), generator=g, device="cuda") * stride], 1)
    c = torch.unique(c, dim=0)
    c = c[torch.randperm(c.size(0), generator=g, device="cuda")][:n]
    return (torch.unique(c, dim=0) if order == "sorted" else c).int().contiguous()


# the index used and (thin clouds) not used, rows in spatial order, further offsets, one voxel of key bits and many
@pytest.mark.parametrize("D,n,extent,kernel,dilation,stride,order,in_use", [
    (3, 1_970_000, 110, 3, 1, 1, "random", True), (3, 2_000_001, 5000, 3, 1, 1, "random", False),
    (3, 1_970_001, 100, 3, 3, 4, "sorted", True), (4, 2_100_003, 36, 3, 1, 1, "random", True),
    (5, 1_970_000, 16, 3, 1, 2, "random", True),
])
def test_ordered_map_is_the_self_map_in_another_order(D, n, extent, kernel, dilation, stride, order, in_use):
    from riemannengine_b200 import capi, ops
    c = _cloud(D, n, extent, stride, order, D * 1000 + n)
    table = ops.table_build(c)
    off = ops.region_offsets(0, [kernel] * D, [dilation] * D, [stride] * D)
    K = off.shape[0]
    want = ops.kmap_build(table, table.coords, off).nbr
    lib = capi.lib()
    size = lib.rmn_kmap_ordered_workspace_bytes(n, D + 1, K)
    assert size > 0 and lib.rmn_kmap_ordered_workspace_bytes(1_900_000, D + 1, K) == 0
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    rows, nbr = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty((K, n), dtype=torch.int32, device="cuda")
    offsets = torch.as_tensor(off, dtype=torch.int32, device="cuda").contiguous()
    capi.check(lib.rmn_kmap_build_ordered(ops._ptr(table.buffer), ops._ptr(table.coords), n, D + 1, ops._ptr(offsets), K,
                                          ops._ptr(rows), ops._ptr(nbr), ops._ptr(scratch), size, ops._stream()), "ordered")
    identity = torch.arange(n, dtype=torch.int32, device="cuda")
    assert torch.equal(rows.sort().values, identity) and torch.equal(rows, identity) == (not in_use)
    for k in range(K):
        assert torch.equal(nbr[k], want[k][rows.long()])


def test_layers_that_only_run_forward_give_the_same_rows_over_an_ordered_map():
    """The C++ host takes an ordered map where no gradient is wanted, the public map otherwise: same bits, bias, residual and
    padded channels included; pair lists asked for afterwards are those of the public map."""
    from riemannengine_b200 import cpp
    C = cpp.load()
    n = 1_980_000
    c = _cloud(3, n, 110, 1, "random", 7)
    g = torch.Generator(device="cuda").manual_seed(8)
    for c_in, c_out in ((32, 32), (4, 20)):
        layer = C.RiemannConvolution(c_in, c_out, kernel_size=3, stride=1, bias=True, dimension=3)
        layer.to("cuda:0")
        layer.to(torch.bfloat16)
        feats = torch.randn((n, c_in), generator=g, device="cuda").bfloat16()
        want = layer(C.SparseTensor(feats, c)).F.detach()
        with torch.no_grad():
            x = C.SparseTensor(feats, c)
            got, again = layer(x), layer(x)
        assert torch.equal(got.F, want) and torch.equal(again.F, want)
    key = x.coordinate_map_key
    pairs = x.coordinate_manager.kernel_map_pairs(key, got.coordinate_map_key, [3] * 3, [1] * 3, [1] * 3)
    y = C.SparseTensor(feats, c)
    public = y.coordinate_manager.kernel_map_pairs(y.coordinate_map_key, y.coordinate_map_key, [3] * 3, [1] * 3, [1] * 3)
    assert all(torch.equal(torch.as_tensor(a), torch.as_tensor(b)) for a, b in zip(pairs, public))


# up to 4096 counts (offsets x blocks of 256 rows) the last block of the probing kernel adds them up, beyond a kernel of its own
@pytest.mark.parametrize("n,self_map,kernel", [(1, True, 3), (300, True, 1), (5000, True, 3), (74_752, True, 3), (74_753, True, 3),
                                               (300, False, 2), (131_072, False, 2), (131_073, False, 2)])
def test_offset_pointers_and_pair_lists_of_small_maps(n, self_map, kernel):
    from riemannengine_b200 import ops
    c = _cloud(3, n, 60, 1, "random", n)
    table = ops.table_build(c)
    off = ops.region_offsets(0, [kernel] * 3, [1] * 3, [1] * 3)
    m = ops.kmap_build(table, table.coords, off, self_map=self_map)
    counts = (m.nbr >= 0).sum(1)
    assert torch.equal(m.offset_ptr[1:], counts.cumsum(0)) and int(m.offset_ptr[0]) == 0
    ptr, a, q = m.pairs()
    for k in range(off.shape[0]):
        lo, hi = int(m.offset_ptr[k]), int(m.offset_ptr[k + 1])
        want = (m.nbr[k] >= 0).nonzero().flatten()
        order = q[lo:hi].argsort()
        assert torch.equal(q[lo:hi][order].long(), want) and torch.equal(a[lo:hi][order], m.nbr[k][want])


def test_fused_layers_over_an_ordered_map_give_the_rows_of_the_public_one():
    """Convolution, batch norm and ReLU as one kernel, over the map that a layer without gradients takes and over the public one,
    which a request for pair lists leaves in the manager: the same bits."""
    from riemannengine_b200 import cpp
    C = cpp.load()
    n = 1_980_000
    c = _cloud(3, n, 110, 1, "random", 9)
    g = torch.Generator(device="cuda").manual_seed(9)
    for c_in, c_out in ((32, 64), (64, 20)):
        layer = C.RiemannConvolution(c_in, c_out, kernel_size=3, stride=1, bias=True, dimension=3)
        layer.to("cuda:0")
        layer.to(torch.bfloat16)
        feats = torch.randn((n, c_in), generator=g, device="cuda").bfloat16()
        stats = [torch.rand(c_out, generator=g, device="cuda") + 0.5 for _ in range(4)]
        ordered, public = C.SparseTensor(feats, c), C.SparseTensor(feats, c)
        key = public.coordinate_map_key
        public.coordinate_manager.kernel_map_pairs(key, key, [3] * 3, [1] * 3, [1] * 3)
        got, want = (C.fused_conv_bn_relu(x, layer, *stats, 1e-5, True).F for x in (ordered, public))
        assert torch.equal(got, want) and float(got.max()) > 0


# rows around a block of 256 and around the four of them that a CUDA block takes; the index used and not used
@pytest.mark.parametrize("D,n,extent,kernel,order", [(3, 1_970_000, 110, 3, "random"), (3, 1_970_177, 5000, 3, "random"),
                                                     (3, 1_970_945, 100, 3, "sorted"), (4, 1_980_161, 36, 3, "random")])
def test_public_map_made_from_an_ordered_one(D, n, extent, kernel, order):
    """The same table, counts and pair lists as a build of its own, bit for bit."""
    from riemannengine_b200 import capi, ops
    c = _cloud(D, n, extent, 1, order, n)
    table = ops.table_build(c)
    off = ops.region_offsets(0, [kernel] * D, [1] * D, [1] * D)
    K = off.shape[0]
    want = ops.kmap_build(table, table.coords, off, self_map=True)
    lib = capi.lib()
    scratch = torch.empty(lib.rmn_kmap_ordered_workspace_bytes(n, D + 1, K), dtype=torch.uint8, device="cuda")
    rows, ordered = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty((K, n), dtype=torch.int32, device="cuda")
    offsets = torch.as_tensor(off, dtype=torch.int32, device="cuda").contiguous()
    capi.check(lib.rmn_kmap_build_ordered(ops._ptr(table.buffer), ops._ptr(table.coords), n, D + 1, ops._ptr(offsets), K,
                                          ops._ptr(rows), ops._ptr(ordered), ops._ptr(scratch), scratch.numel(), ops._stream()),
               "rmn_kmap_build_ordered")
    del scratch
    size = lib.rmn_kmap_workspace_bytes(n, K)
    workspace = torch.full((size + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    nbr = torch.full((K, n), -2, dtype=torch.int32, device="cuda")
    offset_ptr = torch.full((K + 1,), -1, dtype=torch.int64, device="cuda")
    on_host = torch.full((K + 1,), -1, dtype=torch.int64).pin_memory()
    args = [ops._ptr(rows), ops._ptr(ordered), n, K, ops._ptr(nbr), ops._ptr(offset_ptr), on_host.data_ptr(), ops._ptr(workspace)]
    assert lib.rmn_kmap_build_from_ordered(*args, size - 1, ops._stream()) != 0
    capi.check(lib.rmn_kmap_build_from_ordered(*args, size, ops._stream()), "rmn_kmap_build_from_ordered")
    torch.cuda.synchronize()
    assert bool((workspace[size:] == 0xA5).all())
    for k in range(K):
        assert torch.equal(nbr[k], want.nbr[k])
    assert torch.equal(offset_ptr, want.offset_ptr) and torch.equal(on_host, want.offset_ptr.cpu())
    got = ops.NeighbourTable(nbr, offset_ptr, workspace[:size], n, K, n)
    for a, b in zip(got.pairs(), want.pairs()):
        assert torch.equal(torch.as_tensor(a), torch.as_tensor(b))


def test_a_layer_without_gradients_leaves_no_second_build_behind():
    """Pair lists and training passes behind a layer that only ran forward: results, gradients and lists of a manager in which it
    did not, and no two maps held."""
    from riemannengine_b200 import cpp
    C = cpp.load()
    n = 1_980_000
    c = _cloud(3, n, 110, 1, "random", 11)
    g = torch.Generator(device="cuda").manual_seed(11)
    layer = C.RiemannConvolution(32, 32, kernel_size=3, stride=1, bias=True, dimension=3)
    layer.to("cuda:0")
    layer.to(torch.bfloat16)
    feats, grad = (torch.randn((n, 32), generator=g, device="cuda").bfloat16() for _ in range(2))

    def both_passes(forward_first):
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        f = feats.clone().requires_grad_(True)
        x = C.SparseTensor(f, c)
        with torch.no_grad():
            first = layer(x if forward_first else C.SparseTensor(feats, c)).F
        layer.zero_grad()
        out = layer(x).F
        out.backward(grad)
        key = x.coordinate_map_key
        pairs = x.coordinate_manager.kernel_map_pairs(key, key, [3] * 3, [1] * 3, [1] * 3)
        with torch.no_grad():
            after = layer(x).F
        results = [first, out.detach(), f.grad, layer.kernel.grad.clone(), after] + [torch.as_tensor(p) for p in pairs]
        return results, torch.cuda.memory_allocated() - before

    both_passes(False)   # (what is allocated once)
    (want, held), (got, held_after) = both_passes(False), both_passes(True)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert held_after <= held + 27 * n * 2   # (a second table would be 27 n x 4)
