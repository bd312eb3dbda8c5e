"""fp32 convolution kernels (compacted rows) against a float64 reference, at the edges of their tiles: row counts
around the 32 rows of a warp and the batches, channel counts that are multiples of four but not of a tile, fills from
one neighbour to all of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(feats, w, nbr):
    out = torch.zeros((nbr.size(1), w.size(2)), dtype=torch.float64)
    for k in range(w.size(0)):
        rows = nbr[k]
        hit = rows >= 0
        out[hit] += feats[rows[hit].long()].double() @ w[k].double()
    return out


@pytest.mark.parametrize("n,c_in,c_out,K,fill", [
    (1, 4, 4, 1, 1.0), (31, 32, 32, 27, 0.6), (33, 36, 20, 27, 0.02), (65, 64, 100, 8, 1.0), (1000, 4, 64, 27, 0.5),
    (1025, 100, 32, 5, 0.9), (4097, 32, 64, 27, 0.45), (40001, 32, 36, 27, 0.3),
])
def test_f32_passes_match_float64(n, c_in, c_out, K, fill):
    from riemannengine_b200 import ops
    g = torch.Generator().manual_seed(n + c_in)
    n_src = n + 7
    nbr = torch.randint(0, n_src, (K, n), generator=g, dtype=torch.int32)
    nbr[torch.rand((K, n), generator=g) >= fill] = -1
    feats = torch.randn((n_src, c_in), generator=g)
    w = torch.randn((K, c_in, c_out), generator=g)
    grad = torch.randn((n, c_out), generator=g)
    shift, scale = torch.randn(c_out, generator=g), torch.randn(c_out, generator=g)

    def close(got, want):
        want = want.double()
        assert got.shape == want.shape
        assert float((got.cpu().double() - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max()))

    d = lambda t: t.cuda()  # noqa: E731
    want = _reference(feats, w, nbr)
    close(ops.conv_forward(d(feats), d(w), d(nbr)), want)
    close(ops.conv_forward(d(feats), d(w), d(nbr), scale=d(scale), shift=d(shift), relu=True),
          torch.relu(want * scale.double() + shift.double()))
    # the same table read as an input-gradient table: rows of `feats` stand for output gradients
    close(ops.conv_backward_input(d(feats), d(w.transpose(1, 2).contiguous()), d(nbr)), want)
    want_w = torch.stack([feats[nbr[k][nbr[k] >= 0].long()].double().t() @ grad[nbr[k] >= 0].double() for k in range(K)])
    close(ops.conv_backward_weight(d(feats), d(grad), d(nbr)), want_w)


def test_weight_gradient_of_more_channel_tiles_than_a_launch_takes():
    from riemannengine_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    feats, grad = torch.randn((3, 16384), generator=g, device="cuda"), torch.randn((3, 8192), generator=g, device="cuda")
    nbr = torch.tensor([[2, -1, 0]], dtype=torch.int32, device="cuda")
    got = ops.conv_backward_weight(feats, grad, nbr)[0]
    want = feats[2][:, None] * grad[0] + feats[0][:, None] * grad[2]
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())


def test_transpose_weights_reverses_the_offsets():
    from riemannengine_b200 import capi, ops
    for dtype, code in ((torch.float32, capi.F32), (torch.bfloat16, capi.BF16)):
        w = torch.randn(27, 33, 70).to(dtype).cuda()
        for reverse in (0, 1):
            out = torch.empty((27, 70, 33), dtype=dtype, device="cuda")
            capi.check(capi.lib().rmn_conv_transpose_weights(ops._ptr(w), 27, 33, 70, code, reverse, ops._ptr(out),
                                                             ops._stream()), "rmn_conv_transpose_weights")
            want = w.transpose(1, 2)
            assert torch.equal(out, (want.flip(0) if reverse else want).contiguous())
