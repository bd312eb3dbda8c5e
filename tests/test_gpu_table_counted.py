"""rmn_table_build_counted (counts stored by the build itself) and rmn_kmap_build_host against the calls without them: row
counts around the one-block build and around 256-row blocks, with and without duplicates, the hint either way, a packing
overflow; row counts at which the offsets of a map are split over blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _coords(n, D, extent, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.randint(-extent, extent, (n, D), generator=g, device="cuda")
    return torch.cat([torch.randint(0, 2, (n, 1), generator=g, device="cuda"), c], 1).int().contiguous()


def _counted(coords, hint):
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    n, W = coords.shape
    new = lambda size, dtype: torch.empty(size, dtype=dtype, device="cuda")  # noqa: E731
    table, ws = new(lib.rmn_table_bytes(n), torch.uint8), new(lib.rmn_table_build_workspace_bytes(n), torch.uint8)
    mapping, inverse, unique = new(n, torch.int64), new(n, torch.int64), new((n, W), torch.int32)
    info = torch.zeros(4, dtype=torch.int32)
    rc = lib.rmn_table_build_counted(ops._ptr(coords), n, W, ops._ptr(table), table.numel(), ops._ptr(mapping),
                                     ops._ptr(inverse), ops._ptr(unique), ops._ptr(ws), ws.numel(), hint, info.data_ptr(),
                                     ops._stream())
    return rc, info, mapping, inverse, unique, table


@pytest.mark.parametrize("hint", [0, 1])
@pytest.mark.parametrize("D", [1, 3, 4])
@pytest.mark.parametrize("n,extent", [(1, 5), (1023, 4), (1025, 10_000), (2048, 9), (2048, 10_000), (2049, 9), (4097, 10_000),
                                      (300_001, 30)])
def test_counted_build_matches_torch(n, D, extent, hint):
    c = _coords(n, D, extent, n + D)
    rc, info, mapping, inverse, unique, table = _counted(c, hint)
    assert rc == 0
    rows, inv = torch.unique(c, dim=0, return_inverse=True)
    first = torch.full((rows.size(0),), n, dtype=torch.int64, device="cuda").scatter_reduce(
        0, inv, torch.arange(n, device="cuda"), "amin")
    order = first.argsort()
    m = rows.size(0)
    assert info.tolist()[0] == m and info.tolist()[3] == n
    assert torch.equal(mapping[:m], first[order])
    assert torch.equal(unique[:m], rows[order])
    assert torch.equal(inverse, order.argsort()[inv])
    from riemannengine_b200 import capi, ops
    found = torch.empty(n, dtype=torch.int32, device="cuda")
    capi.check(capi.lib().rmn_table_find(ops._ptr(table), ops._ptr(c), n, c.size(1), ops._ptr(found), ops._stream()), "find")
    assert torch.equal(found.long(), inverse)


@pytest.mark.parametrize("n", [3, 3000])
def test_counted_build_reports_a_range_that_does_not_pack(n):
    from riemannengine_b200 import capi
    c = _coords(n, 3, 2 ** 30, 1)
    c[0, 1:], c[1, 1:] = -2 ** 31, 2 ** 31 - 1
    rc, info, *_ = _counted(c, 0)
    assert rc != capi.OK and info.tolist()[1] == rc


@pytest.mark.parametrize("n", [1, 255, 900, 20_000, 60_000])
def test_split_offsets_and_host_pointers(n):
    from riemannengine_b200 import capi, ops
    c = torch.unique(_coords(n, 3, max(3, int(n ** (1 / 3))), n), dim=0).contiguous()
    table = ops.table_build(c)
    off = ops.region_offsets(0, [3] * 3, [1] * 3, [1] * 3)
    d_off = torch.from_numpy(off).int().cuda()
    m, K = c.size(0), off.shape[0]
    want = torch.full((K, m), -1, dtype=torch.int32, device="cuda")
    for k in range(K):
        q = c.clone()
        q[:, 1:] += d_off[k]
        capi.check(capi.lib().rmn_table_find(ops._ptr(table.buffer), ops._ptr(q), m, 4, ops._ptr(want[k]), ops._stream()), "find")
    for self_map in (0, 1):
        nbr = torch.empty((K, m), dtype=torch.int32, device="cuda")
        ptr, ws = torch.empty(K + 1, dtype=torch.int64, device="cuda"), torch.empty(
            capi.lib().rmn_kmap_workspace_bytes(m, K), dtype=torch.uint8, device="cuda")
        host = torch.zeros(K + 1, dtype=torch.int64).pin_memory()
        capi.check(capi.lib().rmn_kmap_build_host(ops._ptr(table.buffer), ops._ptr(table.coords), m, 4, ops._ptr(d_off), K,
                                                  self_map, ops._ptr(nbr), ops._ptr(ptr), host.data_ptr(), ops._ptr(ws),
                                                  ws.numel(), ops._stream()), "kmap")
        torch.cuda.synchronize()
        assert torch.equal(nbr, want)
        assert host.tolist() == ptr.tolist() == [0] + (want >= 0).sum(1).cumsum(0).tolist()


@pytest.mark.parametrize("n,channels,extent,mean", [(1, 1, 3, 1), (5000, 4, 8, 1), (5000, 3, 1000, 1), (70_001, 16, 20, 0),
                                                    (4096, 4, 2, 0)])
def test_segment_reduce_matches_float64(n, channels, extent, mean):
    from riemannengine_b200 import capi, ops
    c = _coords(n, 3, extent, n)
    _, info, mapping, inverse, _, _ = _counted(c, 0)
    m = info.tolist()[0]
    x = torch.randn((n, channels), device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    out, counts = torch.empty((m, channels), device="cuda"), torch.empty(m, dtype=torch.int32, device="cuda")
    capi.check(capi.lib().rmn_segment_reduce(ops._ptr(x), n, channels, ops._ptr(inverse), ops._ptr(mapping), m, mean,
                                             ops._ptr(out), ops._ptr(counts), ops._stream()), "segment")
    want = torch.zeros((m, channels), dtype=torch.float64, device="cuda").index_add_(0, inverse, x.double())
    per = torch.bincount(inverse, minlength=m).double().unsqueeze(1)
    if mean:
        want /= per
    assert float((out.double() - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max()))
    assert n == m or torch.equal(counts.double(), per[:, 0])


def test_voxel_averages_are_fixed_where_determinism_is_asked_for():
    """With torch.use_deterministic_algorithms every sum has torch's fixed order; without it the order is the atomics'."""
    from riemannengine_b200 import cpp
    C = cpp.load()
    n = 200_000
    points = _coords(n, 3, 6, 9).float()
    x = torch.randn((n, 5), device="cuda", generator=torch.Generator(device="cuda").manual_seed(9)) * 1e3
    voxels, inverse = torch.unique(points, dim=0, return_inverse=True)
    torch.use_deterministic_algorithms(True)
    try:
        want = torch.zeros((voxels.size(0), 5), device="cuda").index_add_(0, inverse, x)
        want /= torch.zeros(voxels.size(0), device="cuda").index_add_(0, inverse, torch.ones(n, device="cuda"))[:, None]
        for _ in range(3):
            y = C.TensorField(x, points).sparse()
            row = (y.C.float()[:, None] == voxels[None]).all(2).int().argmax(1)
            assert torch.equal(y.F, want[row])
    finally:
        torch.use_deterministic_algorithms(False)


def test_voxel_averages_hand_forward_derivatives_on():
    import torch.autograd.forward_ad as fwd
    from riemannengine_b200 import cpp
    C = cpp.load()
    points = _coords(500, 3, 3, 2).float()
    with fwd.dual_level():
        x = fwd.make_dual(torch.randn((500, 4), device="cuda"), torch.full((500, 4), 3.0, device="cuda"))
        tangent = fwd.unpack_dual(C.TensorField(x, points).sparse().F).tangent
    assert tangent is not None and torch.allclose(tangent, torch.full_like(tangent, 3.0))
