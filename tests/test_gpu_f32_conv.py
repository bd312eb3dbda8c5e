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


# Row counts around a row tile and a pair of them; channel counts that fill a
# 32-channel stage or a block of 32 or 64 columns or not; one stage, an odd number, two blocks of channels per offset.
@pytest.mark.parametrize("n,c_in,c_out,K,fill", [
    (1, 16, 36, 1, 1.0), (127, 32, 64, 2, 0.5), (129, 64, 64, 27, 0.0), (257, 40, 36, 27, 0.6), (3071, 32, 64, 5, 0.02),
    (18_084, 32, 32, 27, 0.5), (8192, 16, 4, 8, 1.0), (19_073, 96, 100, 3, 0.4), (40_003, 48, 64, 27, 0.3), (1000, 64, 200, 27, 0.5),
])
@pytest.mark.parametrize("transpose,reverse", [(0, 0), (1, 0), (1, 1)])
def test_f32_on_tensor_cores_matches_float64(n, c_in, c_out, K, fill, transpose, reverse):
    from riemannengine_b200 import capi, ops
    g = torch.Generator(device="cuda").manual_seed(n + c_in)
    n_src = n + 5
    nbr = torch.randint(0, n_src, (K, n), generator=g, dtype=torch.int32, device="cuda")
    nbr[torch.rand((K, n), generator=g, device="cuda") >= fill] = -1
    feats = torch.randn((n_src, c_in), generator=g, device="cuda")
    w = torch.randn((K, c_in, c_out), generator=g, device="cuda")
    scale, shift = (torch.randn(c_out, generator=g, device="cuda") for _ in range(2))
    given = w.flip(0) if reverse else w
    given = (given.transpose(1, 2) if transpose else given).contiguous()
    lib = capi.lib()
    size = lib.rmn_conv_f32_scratch_bytes(n, K, c_in, c_out)
    scratch, out = torch.empty(size, dtype=torch.uint8, device="cuda"), torch.empty((n, c_out), device="cuda")
    want, most = (torch.zeros((n, c_out), dtype=torch.float64, device="cuda") for _ in range(2))
    for k in range(K):
        hit = nbr[k] >= 0
        x, y = feats[nbr[k][hit].long()].double(), w[k].double()
        want[hit] += x @ y
        most[hit] += x.abs() @ y.abs()

    def run(relu, *epilogue):
        capi.check(lib.rmn_conv_forward_f32(ops._ptr(feats), n_src, c_in, ops._ptr(given), K, c_out, transpose, reverse,
                                            ops._ptr(nbr), n, ops._ptr(out), *epilogue, relu, ops._ptr(scratch), size,
                                            ops._stream()), "rmn_conv_forward_f32")
        return out.double()

    # Each product within 2^-23 (parts left out, and the last ones rounded); 32 of them and the parts' sums truncated to the
    # largest, 2^-23 of it at most in each of four steps; sums of K stages rounded, 2^-24 each. 2^-20 of the magnitudes covers it.
    assert size > 0 and bool(((run(0, None, None) - want).abs() <= 2.0 ** -20 * most).all())
    got = run(1, ops._ptr(scale), ops._ptr(shift))
    limit = 2.0 ** -20 * (most * scale.abs() + shift.abs())
    assert bool(((got - torch.relu(want * scale.double() + shift.double())).abs() <= limit).all())


def test_f32_on_tensor_cores_keeps_what_bf16_parts_cannot_hold():
    """Infinities, NaN, numbers next to the largest one and tiny ones: as the fp32 multiply-adds give them."""
    from riemannengine_b200 import capi, ops
    g = torch.Generator(device="cuda").manual_seed(3)
    n, K, c = 700, 3, 64
    nbr = torch.arange(n, dtype=torch.int32, device="cuda").repeat(K, 1)
    nbr[1:][torch.rand((K - 1, n), generator=g, device="cuda") < 0.5] = -1
    feats = torch.randn((n, c), generator=g, device="cuda")
    most = torch.finfo(torch.float32).max
    for row, value in ((3, float("inf")), (40, float("-inf")), (200, float("nan")), (301, most), (333, -most), (420, 3.39e38)):
        feats[row, row % c] = value
    feats[500:600] *= 1e-34   # their third parts lie below the smallest bf16 number
    feats[600:610] = 0
    w = torch.randn((K, c, c), generator=g, device="cuda") * 0.01
    w[:, 5] = 0               # infinity times zero
    feats[650, 5] = float("inf")
    out, again = torch.empty((n, c), device="cuda"), torch.empty((n, c), device="cuda")
    assert ops._conv_f32(feats, w, False, nbr, out, always=True)
    capi.check(capi.lib().rmn_conv_forward(ops._ptr(feats), n, c, ops._ptr(w), K, c, ops._ptr(nbr), n, ops._ptr(again),
                                           capi.F32, ops._stream()), "rmn_conv_forward")
    assert torch.equal(out.isnan(), again.isnan()) and torch.equal(out.isposinf(), again.isposinf())
    assert torch.equal(out.isneginf(), again.isneginf()) and bool(out.isnan().any()) and bool(out.isinf().any())
    finite = again.isfinite()
    size = torch.where(finite, again, 0).abs().amax(1, keepdim=True).expand_as(out)[finite]   # (sums of 64 products and more)
    assert bool(((out[finite].double() - again[finite].double()).abs() <= 1e-5 * size.double()).all())


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


@pytest.mark.parametrize("n,c_in,c_out,K,fill", [(30_000, 32, 32, 27, 0.66), (9000, 64, 64, 27, 0.5), (20_000, 32, 64, 27, 0.05),
                                                 (11_000, 32, 64, 8, 0.55), (5000, 256, 64, 27, 0.5), (30_000, 64, 64, 1, 1.0)])
@pytest.mark.parametrize("kind", ["normal", "positive", "near one", "integers"])
def test_f32_on_tensor_cores_is_as_close_to_float64_as_multiply_adds(n, c_in, c_out, K, fill, kind):
    """Sums of either sign and of one sign (where an error that does not average out would show), and exact ones."""
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    g = torch.Generator(device="cuda").manual_seed(n + c_in)
    nbr = torch.randint(0, n, (K, n), generator=g, dtype=torch.int32, device="cuda")
    nbr[torch.rand((K, n), generator=g, device="cuda") >= fill] = -1
    x = torch.randn((n, c_in), generator=g, device="cuda")
    w = torch.randn((K, c_in, c_out), generator=g, device="cuda")
    if kind == "positive":
        x, w = x.abs(), w.abs()
    elif kind == "near one":
        x, w = 1 + 0.1 * x.abs(), 1 + 0.1 * w.abs()
    elif kind == "integers":
        x, w = (4 * x).round(), (4 * w).round()
    want = torch.zeros((n, c_out), dtype=torch.float64, device="cuda")
    for k in range(K):
        hit = nbr[k] >= 0
        want[hit] += x[nbr[k][hit].long()].double() @ w[k].double()
    size = lib.rmn_conv_f32_scratch_bytes(n, K, c_in, c_out)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    out, plain = torch.empty((n, c_out), device="cuda"), torch.empty((n, c_out), device="cuda")
    capi.check(lib.rmn_conv_forward_f32(ops._ptr(x), n, c_in, ops._ptr(w), K, c_out, 0, 0, ops._ptr(nbr), n, ops._ptr(out), None,
                                        None, 0, ops._ptr(scratch), size, ops._stream()), "rmn_conv_forward_f32")
    capi.check(lib.rmn_conv_forward(ops._ptr(x), n, c_in, ops._ptr(w), K, c_out, ops._ptr(nbr), n, ops._ptr(plain), capi.F32,
                                    ops._stream()), "rmn_conv_forward")
    if kind == "integers":
        assert torch.equal(out.double(), want)
    else:
        assert float((out.double() - want).norm()) <= float((plain.double() - want).norm())


@pytest.mark.parametrize("x_exponent,w_exponent,both", [
    (-118, 40, False), (-124, 60, False), (40, -118, False), (60, -124, False),   # one side's last parts below bf16's numbers
    (-140, 60, False), (60, -140, False),                                        # no parts at all: sums of zero
    (-70, -70, False), (-60, -45, False),                                        # products below the smallest numbers
    (-118, 40, True), (30, -120, True), (-140, 60, True),                        # beside operands of ordinary size
])
@pytest.mark.parametrize("transpose", [0, 1])
def test_tiny_operands_of_either_side(x_exponent, w_exponent, both, transpose):
    """The loss of bits depends on the operands, not on the sum: tiny features beside large weights, and the reverse."""
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    g = torch.Generator(device="cuda").manual_seed(x_exponent + 2 * w_exponent)
    n, K, c = 1500, 27, 32
    nbr = torch.randint(-n, n, (K, n), generator=g, dtype=torch.int32, device="cuda").clamp_(min=-1)
    # (magnitudes of 1 to 2, so that a sum has as many bits as its operands)
    x = (1 + torch.rand((n, c), generator=g, device="cuda", dtype=torch.float64)) * 2.0 ** x_exponent
    w = (1 + torch.rand((K, c, c), generator=g, device="cuda", dtype=torch.float64)) * 2.0 ** w_exponent
    if both:   # rows and columns of ordinary numbers, and rows of zeros
        x[::3] = torch.randn((n, c), generator=g, device="cuda", dtype=torch.float64)[::3]
        x[1::5] = 0
        w[:, :, ::2] = torch.randn((K, c, c), generator=g, device="cuda", dtype=torch.float64)[:, :, ::2]
    x, w = x.float(), w.float()
    given = (w.transpose(1, 2) if transpose else w).contiguous()
    size = lib.rmn_conv_f32_scratch_bytes(n, K, c, c)
    scratch, out = torch.empty(size, dtype=torch.uint8, device="cuda"), torch.empty((n, c), device="cuda")
    capi.check(lib.rmn_conv_forward_f32(ops._ptr(x), n, c, ops._ptr(given), K, c, transpose, 0, ops._ptr(nbr), n, ops._ptr(out),
                                        None, None, 0, ops._ptr(scratch), size, ops._stream()), "rmn_conv_forward_f32")
    want, most = (torch.zeros((n, c), dtype=torch.float64, device="cuda") for _ in range(2))
    for k in range(K):
        hit = nbr[k] >= 0
        a, b = x[nbr[k][hit].long()].double(), w[k].double()
        want[hit] += a @ b
        most[hit] += a.abs() @ b.abs()
    # 32 multiply-adds of an offset, 27 offsets: 2^-24 of the magnitudes each, 2^-150 where numbers are subnormal
    assert bool(((out.double() - want).abs() <= 59 * (2.0 ** -24 * most + 2.0 ** -150)).all())


def test_weights_in_the_middle_of_a_buffer():
    """Parameters flattened into one buffer start at any element: the same results as aligned ones, in every pass."""
    from riemannengine_b200 import capi, ops
    g = torch.Generator(device="cuda").manual_seed(4)
    n, c, K = 20_000, 32, 27
    assert capi.lib().rmn_conv_f32_pays(n, K, c, c)
    nbr = torch.randint(-n, n, (K, n), generator=g, dtype=torch.int32, device="cuda").clamp_(min=-1)
    feats = torch.randn((n, c), generator=g, device="cuda")
    w = torch.randn((K, c, c), generator=g, device="cuda")
    for first in (1, 2, 3):
        inside = torch.zeros(w.numel() + 4, device="cuda")[first:first + w.numel()].view(w.shape).copy_(w)
        assert inside.is_contiguous() and inside.data_ptr() % 16
        assert torch.equal(ops.conv_forward(feats, inside, nbr), ops.conv_forward(feats, w, nbr))
        assert torch.equal(ops.conv_backward_input(feats, inside, nbr), ops.conv_backward_input(feats, w, nbr))


@pytest.mark.parametrize("c_in,c_out,transpose,reverse", [(32, 32, 0, 0), (64, 64, 1, 0), (64, 100, 1, 1), (40, 36, 0, 1)])
def test_rows_that_are_computed_again(c_in, c_out, transpose, reverse):
    """Rows of every tile and quarter of a tile, a few of them and all: the multiply-add kernel's values, in about its time
    (they used to be a serial chain inside the pipeline, an order of magnitude slower than that kernel)."""
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    g = torch.Generator(device="cuda").manual_seed(c_in + c_out)
    n, K = 40_003, 27
    nbr = torch.randint(-n, n, (K, n), generator=g, dtype=torch.int32, device="cuda").clamp_(min=-1)
    nbr[:, 5::7919] = torch.arange(5, n, 7919, dtype=torch.int32, device="cuda")
    feats = torch.randn((n, c_in), generator=g, device="cuda")
    w = torch.randn((K, c_in, c_out), generator=g, device="cuda")
    given = w.flip(0) if reverse else w
    given = (given.transpose(1, 2) if transpose else given).contiguous()
    shift = torch.randn(c_out, generator=g, device="cuda")
    size = lib.rmn_conv_f32_scratch_bytes(n, K, c_in, c_out)
    scratch, out = torch.empty(size, dtype=torch.uint8, device="cuda"), torch.empty((n, c_out), device="cuda")

    def fast():
        capi.check(lib.rmn_conv_forward_f32(ops._ptr(feats), n, c_in, ops._ptr(given), K, c_out, transpose, reverse, ops._ptr(nbr),
                                            n, ops._ptr(out), None, ops._ptr(shift), 0, ops._ptr(scratch), size, ops._stream()),
                   "rmn_conv_forward_f32")
        return out

    def plain():
        again = torch.empty((n, c_out), device="cuda")
        capi.check(lib.rmn_conv_forward_fused(ops._ptr(feats), n, c_in, ops._ptr(w), K, c_out, ops._ptr(nbr), n, ops._ptr(again),
                                              capi.F32, None, ops._ptr(shift), 0, ops._stream()), "rmn_conv_forward_fused")
        return again

    def time(f):
        best = 1e9
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            f()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    normal = time(plain)
    feats[5::7919] = float("nan")
    got, want = fast(), plain()
    assert torch.equal(got.isnan(), want.isnan()) and bool(got[5::7919].isnan().all()) and bool(got.isfinite().any())
    ok = want.isfinite()
    # within twice the bound of a sum of K c_in multiply-adds of this size (see above) of each other
    assert float((got[ok] - want[ok]).abs().max()) <= 2.0 ** -18 * float(want[ok].abs().max())
    feats.fill_(float("inf"))
    assert torch.equal(fast().nan_to_num(7.0), plain().nan_to_num(7.0))
    assert time(fast) <= 8 * normal
    capi.check(lib.rmn_device_status(ops._stream()), "rmn_device_status")


# the lines of the rule (15 625 rows x 125 offsets, 361 690 rows x 27 offsets of 64 -> 64 channels) from both sides, fills around
# one in sixteen, an empty and a full table
@pytest.mark.parametrize("n,c_in,c_out,K,fill,thin", [(15_700, 64, 64, 125, 0.01, True), (15_700, 64, 64, 125, 0.055, True),
                                                      (15_700, 64, 64, 125, 0.07, False), (15_700, 64, 64, 125, 1.0, False),
                                                      (15_700, 64, 64, 125, 0.0, True), (15_500, 64, 64, 125, 0.01, False),
                                                      (62_600, 32, 32, 125, 0.02, True), (21_300, 40, 76, 124, 0.02, True),
                                                      (362_000, 64, 64, 27, 0.04, True), (361_000, 64, 64, 27, 0.04, False)])
@pytest.mark.parametrize("transpose,reverse,first", [(0, 0, 0), (1, 0, 0), (0, 1, 1), (1, 1, 3)])
def test_large_passes_over_thin_tables_are_the_multiply_add_kernels(n, c_in, c_out, K, fill, thin, transpose, reverse, first):
    """Which kernel did it shows in the last bits: those of rmn_conv_forward_fused where the table is thin."""
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    g = torch.Generator(device="cuda").manual_seed(n + K + int(100 * fill))
    nbr = torch.randint(0, n, (K, n), generator=g, dtype=torch.int32, device="cuda")
    nbr[torch.rand((K, n), generator=g, device="cuda") >= fill] = -1
    x = torch.randn((n, c_in), generator=g, device="cuda")
    w = torch.randn((K, c_in, c_out), generator=g, device="cuda")
    given = w.flip(0) if reverse else w
    given = (given.transpose(1, 2) if transpose else given).contiguous()
    given = torch.zeros(given.numel() + 4, device="cuda")[first:first + given.numel()].view(given.shape).copy_(given)
    scale, shift = torch.randn((2, c_out), generator=g, device="cuda")
    size = lib.rmn_conv_f32_scratch_bytes(n, K, c_in, c_out)
    scratch = torch.full((size + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    out, plain = (torch.full((n, c_out), 7.0, device="cuda") for _ in range(2))
    capi.check(lib.rmn_conv_forward_f32(ops._ptr(x), n, c_in, ops._ptr(given), K, c_out, transpose, reverse, ops._ptr(nbr), n,
                                        ops._ptr(out), ops._ptr(scale), ops._ptr(shift), 1, ops._ptr(scratch), size,
                                        ops._stream()), "rmn_conv_forward_f32")
    capi.check(lib.rmn_conv_forward_fused(ops._ptr(x), n, c_in, ops._ptr(w), K, c_out, ops._ptr(nbr), n, ops._ptr(plain), capi.F32,
                                          ops._ptr(scale), ops._ptr(shift), 1, ops._stream()), "rmn_conv_forward_fused")
    assert torch.equal(out, plain) == (thin or fill == 0.0)
    # two sums of up to K c_in products, each within 2^-24 of the magnitudes a term (the grouped sum far less)
    assert float((out - plain).abs().max()) <= 2.0 ** -18 * max(1.0, float(plain.abs().max()))
    assert bool((scratch[size:] == 0xA5).all())


@pytest.mark.parametrize("n,c_in,c_out,K,fill", [(20_000, 32, 32, 64, 0.66), (20_000, 32, 32, 125, 0.5), (8000, 64, 64, 125, 0.5),
                                                 (12_000, 32, 32, 343, 0.66), (4000, 64, 64, 343, 0.66), (6000, 32, 32, 729, 0.66),
                                                 (4000, 256, 64, 125, 0.5), (20_000, 256, 32, 125, 0.5)])
@pytest.mark.parametrize("kind", ["normal", "positive", "near one", "integers"])
def test_f32_sums_of_many_stages_are_as_close_to_float64_as_multiply_adds(n, c_in, c_out, K, fill, kind):
    """Kernels of five and more along an axis: hundreds of partial sums, whose roundings must not add up. Tables above the line of
    one neighbour in sixteen: the tensor cores' kernel, with single row tiles and with two."""
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    g = torch.Generator(device="cuda").manual_seed(n + c_in + K)
    nbr = torch.randint(0, n, (K, n), generator=g, dtype=torch.int32, device="cuda")
    nbr[torch.rand((K, n), generator=g, device="cuda") >= fill] = -1
    x = torch.randn((n, c_in), generator=g, device="cuda")
    w = torch.randn((K, c_in, c_out), generator=g, device="cuda")
    if kind == "positive":
        x, w = x.abs(), w.abs()
    elif kind == "near one":
        x, w = 1 + 0.1 * x.abs(), 1 + 0.1 * w.abs()
    elif kind == "integers":
        x, w = x.round(), w.round()
    want = torch.zeros((n, c_out), dtype=torch.float64, device="cuda")
    for k in range(K):
        hit = nbr[k] >= 0
        want[hit] += x[nbr[k][hit].long()].double() @ w[k].double()
    size = lib.rmn_conv_f32_scratch_bytes(n, K, c_in, c_out)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    out, plain = torch.empty((n, c_out), device="cuda"), torch.empty((n, c_out), device="cuda")
    capi.check(lib.rmn_conv_forward_f32(ops._ptr(x), n, c_in, ops._ptr(w), K, c_out, 0, 0, ops._ptr(nbr), n, ops._ptr(out), None,
                                        None, 0, ops._ptr(scratch), size, ops._stream()), "rmn_conv_forward_f32")
    capi.check(lib.rmn_conv_forward(ops._ptr(x), n, c_in, ops._ptr(w), K, c_out, ops._ptr(nbr), n, ops._ptr(plain), capi.F32,
                                    ops._stream()), "rmn_conv_forward")
    if kind == "integers":
        assert torch.equal(out.double(), want)
    else:
        assert float((out.double() - want).norm()) <= float((plain.double() - want).norm())


@pytest.mark.parametrize("n,c_in,c_out,K,fill", [(30_000, 32, 64, 4, 0.55), (30_000, 32, 64, 7, 0.55), (30_000, 64, 64, 2, 0.55),
                                                 (30_000, 64, 64, 3, 0.6), (30_000, 16, 64, 7, 0.55), (30_000, 24, 32, 5, 1.0),
                                                 (12_000, 32, 64, 7, 0.55), (30_000, 32, 64, 3, 0.6)])
@pytest.mark.parametrize("kind", ["normal", "positive", "near one", "integers"])
def test_f32_sums_of_few_stages_are_as_close_to_float64_as_multiply_adds(n, c_in, c_out, K, fill, kind):
    """Kernels of a few offsets (a cross of seven), whose sums are one group or two; single row tiles and two."""
    test_f32_sums_of_many_stages_are_as_close_to_float64_as_multiply_adds(n, c_in, c_out, K, fill, kind)
