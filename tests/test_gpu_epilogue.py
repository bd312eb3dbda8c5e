"""What the kernels do behind the sum: ReLU, residual and folded batch norm of the convolutions and the affine pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _room(n, seed, extent=24):
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = torch.unique(torch.randint(0, extent, (n, 3), generator=g, device="cuda"), dim=0)
    return torch.cat([torch.zeros_like(c[:, :1]), c], 1).int().contiguous(), g


# (channels, type, whether the plain entry point is called): k_conv_ta, k_conv_tc, the two fp32 kernels, the generic bf16 one
@pytest.mark.parametrize("c_in,c_out,dtype,plain", [(32, 64, torch.bfloat16, False), (32, 64, torch.bfloat16, True),
                                                    (32, 64, torch.float32, True), (5, 7, torch.float32, True),
                                                    (5, 7, torch.bfloat16, True)])
def test_relu_epilogue_keeps_nan(c_in, c_out, dtype, plain):
    from riemannengine_b200 import capi, ops
    n = 300
    g = torch.Generator(device="cuda").manual_seed(3)
    nbr = torch.arange(n, device="cuda", dtype=torch.int32)[None].contiguous()
    feats = torch.randn((n, c_in), generator=g, device="cuda").to(dtype)
    feats[17, 2] = float("nan")
    w = torch.randn((1, c_in, c_out), generator=g, device="cuda").to(dtype)
    if plain:
        out = torch.empty((n, c_out), dtype=dtype, device="cuda")
        capi.check(capi.lib().rmn_conv_forward_fused(
            ops._ptr(feats), n, c_in, ops._ptr(w), 1, c_out, ops._ptr(nbr), n, ops._ptr(out),
            capi.F32 if dtype == torch.float32 else capi.BF16, None, None, 1, ops._stream()), "rmn_conv_forward_fused")
    else:
        out = ops.conv_forward(feats, w, nbr, relu=True)
    want = torch.relu(feats.double() @ w[0].double())
    assert torch.equal(out.isnan(), want.isnan()) and bool(out[17].isnan().all())
    rest = torch.arange(n, device="cuda") != 17
    assert torch.allclose(out[rest].double(), want[rest], rtol=1e-2, atol=5e-2)
    assert float(out[rest].min()) == 0.0


@pytest.mark.parametrize("channels,dtype", [(64, torch.bfloat16), (7, torch.bfloat16), (12, torch.float32)])
def test_affine_relu_keeps_nan(channels, dtype):
    from riemannengine_b200 import ops
    x = torch.randn((100, channels), device="cuda").to(dtype)
    x[3, 1] = float("nan")
    ones = torch.ones(channels, device="cuda")
    assert torch.equal(ops.affine_act(x, ones, None, relu=True).isnan(), x.isnan())


def test_network_shows_a_nan_in_its_input_with_and_without_gradients():
    from riemannengine_b200 import cpp
    C = cpp.load()
    coords, g = _room(2000, 1)
    torch.manual_seed(1)
    net = C.MinkUNet(4, 20, width=32, dimension=3)
    net.to("cuda:0")
    net.to(torch.bfloat16)
    net.train(False)
    feats = torch.randn((coords.size(0), 4), generator=g, device="cuda").bfloat16()
    feats[11, 0] = float("nan")
    want = net(C.SparseTensor(feats, coords)).F.isnan()
    with torch.no_grad():
        got = net(C.SparseTensor(feats, coords)).F.isnan()
    assert bool(want.any()) and torch.equal(got, want)
