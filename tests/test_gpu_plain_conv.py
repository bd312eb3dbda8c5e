"""The plain convolution entry points of the C ABI (weights as they are, no prepared image), which neither host calls where the
prepared weights cover a layer: every tensor-core pair with and without a plan, the gather4 producers, statistics, fp32 input
gradients, and the hosts' fallback to them - against a float64 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu

PAIRS = [(32, 32), (32, 64), (64, 32), (64, 64), (64, 128), (128, 64), (128, 128), (128, 256), (256, 128), (256, 256)]


def _reference(feats, w, nbr):
    out = torch.zeros((nbr.size(1), w.size(2)), dtype=torch.float64, device=feats.device)
    for k in range(w.size(0)):
        hit = nbr[k] >= 0
        out[hit] += feats[nbr[k][hit].long()].double() @ w[k].double()
    return out


def _close(got, want, tol=6e-3):   # fp32 sums rounded to bf16: half a unit of 2^-8 of the largest value, and some
    assert float((got.double() - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))


def _cloud(n, K, fill, n_src, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nbr = torch.randint(0, n_src, (K, n), generator=g, dtype=torch.int32, device="cuda")
    nbr[torch.rand((K, n), generator=g, device="cuda") >= fill] = -1
    return nbr, g


def _forward(feats, w, nbr, dtype, plan=None, scale=None, shift=None, relu=0):
    from riemannengine_b200 import capi, ops
    K, c_in, c_out = w.shape
    out = torch.empty((nbr.size(1), c_out), dtype=feats.dtype, device="cuda")
    capi.check(capi.lib().rmn_conv_forward_planned(
        ops._ptr(feats), feats.size(0), c_in, ops._ptr(w), K, c_out, ops._ptr(nbr), ops._ptr(plan), nbr.size(1), ops._ptr(out),
        dtype, ops._ptr(scale), ops._ptr(shift), relu, ops._stream()), "rmn_conv_forward_planned")
    return out


def _input_gradient(grad, w, nbr_t, dtype, plan=None):
    from riemannengine_b200 import capi, ops
    K, c_in, c_out = w.shape
    out = torch.empty((nbr_t.size(1), c_in), dtype=grad.dtype, device="cuda")
    capi.check(capi.lib().rmn_conv_backward_input_planned(
        ops._ptr(grad), grad.size(0), c_out, ops._ptr(w), K, c_in, ops._ptr(nbr_t), ops._ptr(plan), nbr_t.size(1), ops._ptr(out),
        dtype, ops._stream()), "rmn_conv_backward_input_planned")
    return out


@pytest.mark.parametrize("n", [127, 5003])   # below one row tile; ragged over many
@pytest.mark.parametrize("c_in,c_out", PAIRS)
def test_bf16_passes_with_and_without_a_plan(c_in, c_out, n, monkeypatch):
    from riemannengine_b200 import capi, ops
    K, n_src = 27, n + 9
    nbr, g = _cloud(n, K, 0.3, n_src, n + c_in + 3 * c_out)
    nbr[:, n // 2:n // 2 + 60] = -1                       # rows without any neighbour
    feats = torch.randn((n_src, c_in), generator=g, device="cuda").bfloat16()
    w = (torch.randn((K, c_in, c_out), generator=g, device="cuda") / c_in ** 0.5).bfloat16()
    wt = w.transpose(1, 2).contiguous()
    scale, shift = (torch.randn(c_out, generator=g, device="cuda") for _ in range(2))
    offsets = ops.region_offsets(0, [3] * 3, [1] * 3, [1] * 3)
    want = _reference(feats, w, nbr)
    plan = ops.conv_plan_build(nbr, offsets)
    other = nbr.clone()
    other[:14] = -1                                       # (a plan holds its own table: whether it is used shows)
    for p, expect in ((None, want), (plan, want), (ops.conv_plan_build(other, offsets), _reference(feats, w, other))):
        _close(_forward(feats, w, nbr, capi.BF16, p), expect)
        _close(_input_gradient(feats, wt, nbr, capi.BF16, p), expect)
        _close(_forward(feats, w, nbr, capi.BF16, p, scale, shift, 1), torch.relu(expect * scale.double() + shift.double()))
    plain = _forward(feats, w, nbr, capi.BF16)
    assert torch.equal(plain, _forward(feats, w, nbr, capi.BF16, plan))
    # gather4 producers: the same sums in the same order
    monkeypatch.setenv("RMN_B200_CONV_TMA", "1")
    assert torch.equal(plain, _forward(feats, w, nbr, capi.BF16))
    assert torch.equal(_input_gradient(feats, wt, nbr, capi.BF16), _input_gradient(feats, wt, nbr, capi.BF16, plan))
    monkeypatch.delenv("RMN_B200_CONV_TMA")
    # channel statistics of the stored values
    lib, size = capi.lib(), capi.lib().rmn_channel_stats_workspace_bytes(c_out)
    for p in (None, plan):
        out, stats = torch.empty((n, c_out), dtype=torch.bfloat16, device="cuda"), torch.empty(
            (2, c_out), dtype=torch.float64, device="cuda")
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        capi.check(lib.rmn_conv_forward_stats_planned(
            ops._ptr(feats), n_src, c_in, ops._ptr(w), K, c_out, ops._ptr(nbr), ops._ptr(p), n, ops._ptr(out), capi.BF16, None,
            None, 0, ops._ptr(stats), ops._ptr(ws), size, ops._stream()), "rmn_conv_forward_stats_planned")
        assert torch.equal(out, plain)
        sums = torch.stack([plain.double().sum(0), (plain.double() ** 2).sum(0)])
        assert float((stats - sums).abs().max()) <= 1e-4 * max(1.0, float(sums.abs().max()))
    assert lib.rmn_device_status(None) == capi.OK


@pytest.mark.parametrize("n,c_in,c_out,K", [(1, 4, 8, 1), (70, 5, 7, 27), (1030, 32, 64, 27), (3000, 64, 36, 8)])
def test_fp32_input_gradient(n, c_in, c_out, K):
    from riemannengine_b200 import capi
    nbr_t, g = _cloud(n, K, 0.6, n + 3, n)
    grad = torch.randn((n + 3, c_out), generator=g, device="cuda")
    w = torch.randn((K, c_in, c_out), generator=g, device="cuda")
    _close(_input_gradient(grad, w, nbr_t, capi.F32), _reference(grad, w.transpose(1, 2), nbr_t), 1e-5)


def test_hosts_take_features_that_are_not_32_byte_aligned():
    from riemannengine_b200 import cpp, engine as E
    C = cpp.load()
    g = torch.Generator(device="cuda").manual_seed(4)
    c = torch.unique(torch.randint(0, 20, (4000, 3), generator=g, device="cuda"), dim=0)
    coords = torch.cat([torch.zeros_like(c[:, :1]), c], 1).int().contiguous()
    n = coords.size(0)

    def misaligned(*shape):
        t = torch.empty(shape[0] * shape[1] + 8, dtype=torch.bfloat16, device="cuda")[8:].view(shape)
        assert t.data_ptr() % 32 == 16
        return t.copy_(torch.randn(shape, generator=g, device="cuda"))

    x, grad = misaligned(n, 64), misaligned(n, 64)
    weights = (torch.randn((27, 64, 64), generator=g, device="cuda") / 30).bfloat16()
    results = []
    for feats, gy in ((x, grad), (x.clone(), grad.clone())):
        for make in ("cpp", "python"):
            feats_ = feats.detach().requires_grad_(True)
            if make == "cpp":
                layer = C.RiemannConvolution(64, 64, kernel_size=3, stride=1, dimension=3)
                layer.to("cuda:0")
                layer.to(torch.bfloat16)
                s = C.SparseTensor(feats_, coords)
            else:
                layer = E.RiemannConvolution(64, 64, kernel_size=3, dimension=3).cuda().bfloat16()
                s = E.SparseTensor(feats_, coords)
            with torch.no_grad():
                layer.kernel.copy_(weights)
            y = layer(s).F
            y.backward(gy)
            results.append((y.detach(), feats_.grad, layer.kernel.grad))
    for other in results[:-1]:
        for got, want in zip(other, results[-1]):
            assert float((got.double() - want.double()).norm()) <= 2e-3 * float(want.double().norm())
