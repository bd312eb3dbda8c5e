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
                                                 None, n, ops._ptr(out), None, None, 0, ops._stream()), "image")
    assert torch.equal(out, ops.conv_forward(feats, w, nbr))
    got, stats = ops.conv_forward_stats(feats, w, nbr, shift=shift)
    _close(got, want + shift.double())
    stored = got.double()
    want_stats = torch.stack([stored.sum(0), (stored * stored).sum(0)])
    assert float((stats - want_stats).abs().max()) <= 1e-4 * max(1.0, float((stored * stored).sum(0).max()))
