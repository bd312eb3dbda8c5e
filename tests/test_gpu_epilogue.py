"""What the kernels do behind the sum: ReLU, residual and folded batch norm of the convolutions and the affine pass."""
import ctypes

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


class _Fold(ctypes.Structure):   # rmn_bn_fold of include/rmn_b200.h
    _fields_ = [(n, ctypes.c_void_p) for n in ("mean", "var", "gamma", "beta", "conv_bias")] + [
        ("param_dtype", ctypes.c_int), ("eps", ctypes.c_float), ("scale", ctypes.c_void_p), ("shift", ctypes.c_void_p)]


# single 64-column blocks (up to 74 row tiles; the second and fourth block of the columns among them) and super-tiles, rows
# around a tile's edge, narrower weights, every absent parameter, both parameter types
@pytest.mark.parametrize("n,w_in,w_out,c_in,c_out,params,dtype,relu", [
    (1, 64, 64, 64, 64, "mvgbc", torch.float32, 1), (127, 64, 128, 64, 128, "mvgbc", torch.bfloat16, 1),
    (129, 100, 250, 128, 256, "mv", torch.float32, 0), (257, 128, 256, 128, 256, "mvg", torch.bfloat16, 1),
    (20_003, 128, 128, 128, 128, "mvb", torch.float32, 1), (20_003, 33, 20, 64, 32, "mvgbc", torch.bfloat16, 0),
    (60_001, 256, 256, 256, 256, "mvgbc", torch.float32, 1), (100_003, 32, 64, 32, 64, "mvc", torch.float32, 1),
])
def test_folded_batch_norm_and_residual_match_float64(n, w_in, w_out, c_in, c_out, params, dtype, relu):
    from riemannengine_b200 import capi, ops
    K = 3
    g = torch.Generator(device="cuda").manual_seed(n)
    nbr = torch.randint(0, n, (K, n), generator=g, dtype=torch.int32, device="cuda")
    nbr[torch.rand((K, n), generator=g, device="cuda") >= 0.6] = -1
    feats = torch.zeros((n, c_in), device="cuda", dtype=torch.bfloat16)
    feats[:, :w_in] = torch.randn((n, w_in), generator=g, device="cuda")
    w = (torch.randn((K, w_in, w_out), generator=g, device="cuda") / w_in ** 0.5).bfloat16()
    add = torch.randn((n, c_out), generator=g, device="cuda").bfloat16()
    values = {"m": torch.randn(w_out, generator=g, device="cuda").to(dtype), "v": torch.rand(w_out, generator=g, device="cuda").add(0.5).to(dtype),
              "g": torch.randn(w_out, generator=g, device="cuda").to(dtype), "b": torch.randn(w_out, generator=g, device="cuda").to(dtype),
              "c": torch.randn(w_out, generator=g, device="cuda").to(dtype)}
    given = [values[p].data_ptr() if p in params else None for p in "mvgbc"]
    vectors = torch.full((2, c_out), 7.0, device="cuda")
    fold = _Fold(*given, capi.F32 if dtype == torch.float32 else capi.BF16, 1e-5, vectors[0].data_ptr(), vectors[1].data_ptr())
    lib = capi.lib()
    image = torch.empty(lib.rmn_conv_weight_image_bytes(K, c_in, c_out, capi.BF16), dtype=torch.uint8, device="cuda")
    capi.check(lib.rmn_conv_weight_image(ops._ptr(w), K, w_in, w_out, c_in, c_out, capi.BF16, 0, 0, ctypes.byref(fold),
                                         ops._ptr(image), ops._stream()), "rmn_conv_weight_image")
    out = torch.empty((n, c_out), dtype=torch.bfloat16, device="cuda")
    capi.check(lib.rmn_conv_forward_image(ops._ptr(feats), n, c_in, ops._ptr(image), K, c_out, ops._ptr(nbr), None, n,
                                          ops._ptr(out), vectors[0].data_ptr(), vectors[1].data_ptr(), ops._ptr(add), relu,
                                          ops._stream()), "rmn_conv_forward_image")
    d = {p: values[p].double() if p in params else torch.full((w_out,), 1.0 if p == "g" else 0.0, device="cuda").double()
         for p in "mvgbc"}
    scale = d["g"] / torch.sqrt(d["v"] + 1e-5)
    shift = d["b"] + (d["c"] - d["m"]) * scale
    assert torch.allclose(vectors[0, :w_out].double(), scale, rtol=1e-5, atol=1e-6)
    assert torch.allclose(vectors[1, :w_out].double(), shift, rtol=1e-5, atol=1e-5)
    want = torch.zeros((n, w_out), dtype=torch.float64, device="cuda")
    for k in range(K):
        hit = nbr[k] >= 0
        want[hit] += feats[nbr[k][hit].long()][:, :w_in].double() @ w[k].double()
    want = want * scale + shift + add[:, :w_out].double()
    if relu:
        want = torch.relu(want)
    # fp32 sums rounded to bf16 once: 2^-9 of a value, and the sum's own error
    assert bool(((out[:, :w_out].double() - want).abs() <= 2 ** -8 * want.abs() + 1e-4 * want.abs().max()).all())


class _Job(ctypes.Structure):   # rmn_weight_job of include/rmn_b200.h
    _fields_ = [("weights", ctypes.c_void_p), ("image", ctypes.c_void_p)] + [
        (n, ctypes.c_int) for n in ("K", "w_in", "w_out", "c_in", "c_out")] + [("fold", _Fold)]


@pytest.mark.parametrize("n_jobs", [1, 24, 25, 61])   # (24 to a launch)
def test_weights_of_layers_prepared_together_are_those_prepared_alone(n_jobs):
    """Layers of mixed shapes, padded ones, batch norms of both parameter types with their own statistics, absent parameters and
    none at all: the same images, scales and shifts, bit for bit, and nothing beyond them."""
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    g = torch.Generator(device="cuda").manual_seed(n_jobs)
    shapes = [(27, 4, 32, 32, 32), (8, 64, 128, 64, 128), (27, 32, 64, 32, 64), (1, 32, 20, 32, 32), (27, 256, 256, 256, 256),
              (9, 100, 250, 128, 256), (81, 64, 33, 64, 64)]
    together, alone, keep = [], [], []
    for j in range(n_jobs):
        K, w_in, w_out, c_in, c_out = shapes[j % len(shapes)]
        dtype = torch.float32 if j % 2 else torch.bfloat16
        w = torch.randn((K, w_in, w_out), generator=g, device="cuda").bfloat16()
        params = [(torch.rand(w_out, generator=g, device="cuda") + 0.5 * i).to(dtype) for i in range(5)]
        given = [p.data_ptr() if i < 2 or (j >> i) & 1 == 0 else None for i, p in enumerate(params)]
        size = lib.rmn_conv_weight_image_bytes(K, c_in, c_out, capi.BF16)
        for jobs in (together, alone):
            image = torch.full((size + 64,), 0xA5, dtype=torch.uint8, device="cuda")
            vectors = torch.full((2 * c_out + 8,), 7.0, device="cuda")
            fold = _Fold(*given, capi.F32 if j % 2 else capi.BF16, 1e-3, vectors.data_ptr(), vectors[c_out:].data_ptr())
            if j % 5 == 3:
                fold = _Fold()
            jobs.append((_Job(w.data_ptr(), image.data_ptr(), K, w_in, w_out, c_in, c_out, fold), image, vectors))
        keep.append((w, params))
    capi.check(lib.rmn_conv_weight_images((_Job * n_jobs)(*[job for job, _, _ in together]), n_jobs, ops._stream()), "images")
    for job, image, _ in alone:
        fold = ctypes.byref(job.fold) if job.fold.scale else None
        capi.check(lib.rmn_conv_weight_image(job.weights, job.K, job.w_in, job.w_out, job.c_in, job.c_out, capi.BF16, 0, 0, fold,
                                             job.image, ops._stream()), "rmn_conv_weight_image")
    for (_, image, vectors), (_, want_image, want_vectors) in zip(together, alone):
        assert torch.equal(image, want_image) and torch.equal(vectors, want_vectors)


# single tiles whose even and odd stages are summed apart, single tiles of more columns, super-tiles; rows around a tile's edge
@pytest.mark.parametrize("n,c_in,c_out,K", [(1, 64, 64, 27), (129, 32, 32, 27), (5003, 64, 64, 1), (9000, 128, 256, 27),
                                            (20_003, 32, 32, 81), (60_001, 64, 128, 27), (100_003, 256, 256, 8)])
@pytest.mark.parametrize("with_add,with_scale,relu", [(True, True, 1), (True, False, 0), (False, True, 1), (False, False, 0)])
def test_an_ordered_map_stores_and_adds_every_row_where_it_belongs(n, c_in, c_out, K, with_add, with_scale, relu):
    """rmn_conv_forward_ordered over a permuted table: bit for bit the rows of rmn_conv_forward_image over the public one."""
    from riemannengine_b200 import capi, ops
    lib = capi.lib()
    g = torch.Generator(device="cuda").manual_seed(n + K)
    nbr = torch.randint(-n, n, (K, n), generator=g, dtype=torch.int32, device="cuda").clamp_(min=-1)
    order = torch.randperm(n, generator=g, device="cuda").int()
    ordered = nbr[:, order.long()].contiguous()
    feats = torch.randn((n, c_in), generator=g, device="cuda").bfloat16()
    w = (torch.randn((K, c_in, c_out), generator=g, device="cuda") / c_in ** 0.5).bfloat16()
    add = torch.randn((n, c_out), generator=g, device="cuda").bfloat16() if with_add else None
    scale, shift = (torch.randn(c_out, generator=g, device="cuda") if with_scale else None for _ in range(2))
    image = torch.empty(lib.rmn_conv_weight_image_bytes(K, c_in, c_out, capi.BF16), dtype=torch.uint8, device="cuda")
    capi.check(lib.rmn_conv_weight_image(ops._ptr(w), K, c_in, c_out, c_in, c_out, capi.BF16, 0, 0, None, ops._ptr(image),
                                         ops._stream()), "rmn_conv_weight_image")
    got, want = (torch.full((n, c_out), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    capi.check(lib.rmn_conv_forward_ordered(ops._ptr(feats), n, c_in, ops._ptr(image), K, c_out, ops._ptr(ordered), ops._ptr(order),
                                            n, ops._ptr(got), ops._ptr(scale), ops._ptr(shift), ops._ptr(add), relu,
                                            ops._stream()), "rmn_conv_forward_ordered")
    capi.check(lib.rmn_conv_forward_image(ops._ptr(feats), n, c_in, ops._ptr(image), K, c_out, ops._ptr(nbr), None, n,
                                          ops._ptr(want), ops._ptr(scale), ops._ptr(shift), ops._ptr(add), relu, ops._stream()),
               "rmn_conv_forward_image")
    assert torch.equal(got, want)
