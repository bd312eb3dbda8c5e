"""bf16 convolution on prepared weights (gathered operand in tensor memory) against a float64 reference: every channel
pair, row counts around one 128-row tile and around those that fill the SMs, even and odd numbers of offsets, transposed and
reversed weights, epilogue and channel statistics."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(32, 32), (32, 64), (64, 32), (64, 64), (64, 128), (128, 64), (128, 128), (128, 256), (256, 128), (256, 256)]


def _reference(feats, w, nbr):
    out = torch.zeros((nbr.size(1), w.size(2)), dtype=torch.float64, device=feats.device)
    for k in range(w.size(0)):
        hit = nbr[k] >= 0
        out[hit] += feats[nbr[k][hit].long()].double() @ w[k].double()
    return out


def _close(got, want):
    assert got.shape == want.shape
    assert float((got.double() - want).abs().max()) <= 6e-3 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("c_in,c_out", SHAPES)
@pytest.mark.parametrize("n,K,fill", [(1, 1, 1.0), (127, 2, 0.5), (129, 27, 0.4), (513, 8, 1.0), (1030, 5, 0.01),
                                      (75_775, 2, 0.5), (100_003, 3, 0.5), (150_001, 3, 0.5)])
def test_image_passes_match_float64(c_in, c_out, n, K, fill):
    from riemannengine_b200 import capi, ops
    assert capi.lib().rmn_conv_weight_image_bytes(K, c_in, c_out, capi.BF16) > 0
    g = torch.Generator(device="cuda").manual_seed(n + c_in + 3 * c_out)
    n_src = n + 7
    nbr = torch.randint(0, n_src, (K, n), generator=g, dtype=torch.int32, device="cuda")
    nbr[torch.rand((K, n), generator=g, device="cuda") >= fill] = -1
    feats = torch.randn((n_src, c_in), generator=g, device="cuda").bfloat16()
    w = (torch.randn((K, c_in, c_out), generator=g, device="cuda") / c_in ** 0.5).bfloat16()
    shift, scale = (torch.randn(c_out, generator=g, device="cuda") for _ in range(2))
    want = _reference(feats, w, nbr)
    _close(ops.conv_forward(feats, w, nbr), want)
    _close(ops.conv_forward(feats, w, nbr, scale=scale, shift=shift, relu=True),
           torch.relu(want * scale.double() + shift.double()))
    _close(ops.conv_backward_input(feats, w.transpose(1, 2).contiguous(), nbr), want)
    # the reversed image stands for the weights in the opposite order of their offsets
    image = ops._weight_image(w.flip(0).contiguous(), False, feats, reverse=True)
    out = torch.empty((n, c_out), dtype=torch.bfloat16, device="cuda")
    capi.check(capi.lib().rmn_conv_forward_image(ops._ptr(feats), n_src, c_in, ops._ptr(image), K, c_out, ops._ptr(nbr),
                                                 None, n, ops._ptr(out), None, None, None, 0, ops._stream()), "image")
    assert torch.equal(out, ops.conv_forward(feats, w, nbr))
    got, stats = ops.conv_forward_stats(feats, w, nbr, shift=shift)
    _close(got, want + shift.double())
    stored = got.double()
    want_stats = torch.stack([stored.sum(0), (stored * stored).sum(0)])
    assert float((stats - want_stats).abs().max()) <= 1e-4 * max(1.0, float((stored * stored).sum(0).max()))


@pytest.mark.parametrize("n", [100, 150_001])   # single 64-column blocks / super-tiles of all columns
@pytest.mark.parametrize("c_in,c_out", [(64, 48), (64, 16), (64, 96), (32, 128), (32, 256), (256, 64), (256, 32), (48, 64), (512, 512)])
def test_image_calls_refuse_pairs_without_a_kernel(n, c_in, c_out):
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    assert lib.rmn_conv_weight_image_bytes(1, c_in, c_out, capi.BF16) == 0
    feats, out = (torch.full((n, c), 3.0, dtype=torch.bfloat16, device="cuda") for c in (c_in, c_out))
    image = torch.zeros(4 * 512 * 512, dtype=torch.uint8, device="cuda")
    nbr = torch.arange(n, dtype=torch.int32, device="cuda")[None].contiguous()
    args = (ops._ptr(feats), n, c_in, ops._ptr(image), 1, c_out, ops._ptr(nbr), None, n, ops._ptr(out), None, None)
    assert lib.rmn_conv_forward_image(*args, None, 0, ops._stream()) == capi.ERR_UNSUPPORTED
    stats = torch.zeros((2, c_out), dtype=torch.float64, device="cuda")
    size = lib.rmn_channel_stats_workspace_bytes(c_out)
    work = torch.empty(size, dtype=torch.uint8, device="cuda")
    assert lib.rmn_conv_forward_image_stats(*args, 0, ops._ptr(stats), ops._ptr(work), size,
                                            ops._stream()) == capi.ERR_UNSUPPORTED
    torch.cuda.synchronize()
    assert bool((out == 3.0).all())


@pytest.mark.parametrize("n,c_in,c_out", [(1, 4, 20), (1000, 20, 96), (4099, 33, 64)])
def test_padded_layer_with_bias_matches_float64(n, c_in, c_out):
    """Channel counts without a kernel of their own: padded features, weights and gradients, the bias gradient."""
    from riemannengine_b200 import cpp, ops
    C = cpp.load()
    g = torch.Generator(device="cuda").manual_seed(n)
    c = torch.unique(torch.randint(0, 40, (2 * n, 3), generator=g, device="cuda"), dim=0)[:n]
    coords = torch.cat([torch.zeros_like(c[:, :1]), c], 1).int().contiguous()
    layer = C.RiemannConvolution(c_in, c_out, kernel_size=3, stride=1, bias=True, dimension=3)
    layer.to("cuda:0")
    layer.to(torch.bfloat16)
    feats = torch.randn((coords.size(0), c_in), generator=g, device="cuda").bfloat16().requires_grad_(True)
    grad = torch.randn((coords.size(0), c_out), generator=g, device="cuda").bfloat16()
    y = layer(C.SparseTensor(feats, coords))
    y.F.backward(grad)
    table = ops.table_build(coords)
    nbr = ops.kmap_build(table, table.coords, ops.region_offsets(0, [3] * 3, [1] * 3, [1] * 3), self_map=True).nbr
    w, b = layer.kernel.detach(), layer.bias.detach()
    _close(y.F.detach(), _reference(feats.detach(), w, nbr) + b.double())
    _close(feats.grad, _reference(grad, w.flip(0).transpose(1, 2), nbr))
    _close(layer.bias.grad, grad.double().sum(0, keepdim=True))
    want = torch.stack([feats.detach()[nbr[k][nbr[k] >= 0].long()].double().t() @ grad[nbr[k] >= 0].double() for k in range(27)])
    _close(layer.kernel.grad, want)


def test_network_in_evaluation_mode_matches_its_layers():
    """Without gradients conv, batch norm, residual and ReLU run as one kernel; with them, layer by layer."""
    from riemannengine_b200 import cpp
    C = cpp.load()
    torch.manual_seed(5)
    g = torch.Generator(device="cuda").manual_seed(5)
    c = torch.unique(torch.randint(0, 24, (3000, 3), generator=g, device="cuda"), dim=0)
    coords = torch.cat([torch.zeros_like(c[:, :1]), c], 1).int().contiguous()
    net = C.MinkUNet(4, 20, width=32, dimension=3)
    net.to("cuda:0")
    net.to(torch.bfloat16)
    feats = torch.randn((coords.size(0), 4), generator=g, device="cuda").bfloat16()
    for _ in range(3):   # running statistics that are not the identity
        net(C.SparseTensor(feats, coords))
    net.train(False)
    want = net(C.SparseTensor(feats, coords)).F.detach().double()
    with torch.no_grad():
        got = net(C.SparseTensor(feats, coords)).F.double()
    assert float((got - want).norm()) <= 2e-2 * float(want.norm())


@pytest.mark.parametrize("c_src,ld,c_dst,skip", [(4, 4, 32, 0), (20, 32, 20, 0), (32, 64, 32, 32), (33, 70, 33, 3), (7, 9, 40, 1)])
def test_pad_channels_copies_strided_rows(c_src, ld, c_dst, skip):
    from riemannengine_b200 import capi, ops
    n = 1027
    x = torch.randn((n, ld + skip), device="cuda").bfloat16()
    out = torch.full((n, c_dst), 7.0, device="cuda", dtype=torch.bfloat16)
    capi.check(capi.lib().rmn_pad_channels(x.data_ptr() + 2 * skip, n, c_src, ld + skip, ops._ptr(out), c_dst, ops._stream()), "pad")
    assert torch.equal(out, torch.nn.functional.pad(x[:, skip:skip + c_src], (0, c_dst - c_src)))


def test_channel_cat_splits_its_gradient():
    from riemannengine_b200 import cpp
    C = cpp.load()
    coords = torch.tensor([[0, i, 0, 0] for i in range(300)], dtype=torch.int32, device="cuda")
    for dtype in (torch.float32, torch.bfloat16):
        a, b = (torch.randn((300, c), device="cuda").to(dtype).requires_grad_(True) for c in (32, 20))
        x = C.SparseTensor(a, coords)
        y = C.cat([x, C.SparseTensor(b, x.coordinate_map_key, x.coordinate_manager)])
        g = torch.randn((300, 52), device="cuda").to(dtype)
        y.F.backward(g)
        assert torch.equal(y.F, torch.cat([a, b], 1))
        assert torch.equal(a.grad, g[:, :32]) and torch.equal(b.grad, g[:, 32:])


def _cat_inputs():
    from riemannengine_b200 import cpp
    C = cpp.load()
    coords = torch.tensor([[0, i, 0, 0] for i in range(40)], dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b, w = (torch.randn((40, c), generator=g, device="cuda") for c in (12, 8, 20))
    base = C.SparseTensor(a, coords)
    on_map = lambda t: C.SparseTensor(t, base.coordinate_map_key, base.coordinate_manager)  # noqa: E731
    return a, b, w, lambda x, y: C.cat([on_map(x), on_map(y)]).F


def test_channel_cat_is_twice_differentiable():
    a, b, w, cat = _cat_inputs()
    second = []
    for join in (cat, lambda x, y: torch.cat([x, y], 1)):
        x, y = a.clone().requires_grad_(True), b.clone().requires_grad_(True)
        first = torch.autograd.grad((join(x, y) ** 3 * w).sum(), (x, y), create_graph=True)
        second.append(torch.autograd.grad(sum((f ** 2).sum() for f in first), (x, y)))
    for got, want in zip(*second):
        assert torch.equal(got, want)


def test_channel_cat_takes_forward_mode_batched_gradients_and_function_transforms():
    import torch.autograd.forward_ad as fwd
    a, b, w, cat = _cat_inputs()
    with fwd.dual_level():
        x = fwd.make_dual(a.clone().requires_grad_(True), torch.ones_like(a))
        y = fwd.make_dual(b.clone().requires_grad_(True), 2 * torch.ones_like(b))
        tangent = fwd.unpack_dual(cat(x, y)).tangent
    assert torch.equal(tangent, torch.cat([torch.ones_like(a), 2 * torch.ones_like(b)], 1))
    x, y = a.clone().requires_grad_(True), b.clone().requires_grad_(True)
    seeds = torch.stack([w, 2 * w, -w])
    ga, gb = torch.autograd.grad(cat(x, y), (x, y), seeds, is_grads_batched=True)
    assert torch.equal(ga, seeds[:, :, :12]) and torch.equal(gb, seeds[:, :, 12:])
    ga, gb = torch.func.grad(lambda x, y: (cat(x, y) * w).sum(), argnums=(0, 1))(a, b)
    assert torch.equal(ga, w[:, :12]) and torch.equal(gb, w[:, 12:])
