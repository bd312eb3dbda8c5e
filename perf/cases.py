"""Representative workloads of the framework, as a program that uses the C++ host layer (``riemann_cpp``) runs them.

Every pass starts from what such a program holds on the GPU (voxel or point coordinates, features, layers with their
weights) and builds its coordinate maps anew, because every batch of scenes brings other coordinates. The sizes are
those of the benchmark's five configurations and of the tests; scenes are generated on the GPU with the statistics of
``riemannengine_b200.synthetic`` (surfaces of a room, a spherical shell, a spinning lidar). The seed mirrors, turns,
moves and shuffles them, in steps of the coarsest grid, so that every seed brings other coordinates in another order
but the same number of rows at every level.
"""
import math

import torch

from riemannengine_b200 import cpp

DEV = "cuda:0"
FULL_ROOM = 150_000           # voxels of one whole room
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}

# Neighbour pairs per voxel of the 3^3 map (3^4 for the clips) of each kind of scene, measured once: they only serve
# work(), which counts 2 * pairs * c_in * c_out flops for a convolution pass.
PAIRS = {"shell": 17.7, "rooms": 12.4, "sweeps": 1.35, "clips": 26.2}
# rows of the next coarser level per row (stride 2 on every axis), same purpose
COARSER = {"shell": 0.22, "rooms": 0.22, "sweeps": 0.8}


def listed():
    return [
        # one small object, fp32 (the layers' default type): what a single call costs when latency is all there is
        {"name": "object-f32", "op": "conv", "scene": "shell", "radius": 6, "dtype": "f32", "c_in": 32, "c_out": 32,
         "kernel": 3, "stride": 1, "train": False, "pairs": False},
        # the benchmark's first configuration: a shell of 101 930 voxels, fp32, one 3^3 layer
        {"name": "shell-f32", "op": "conv", "scene": "shell", "radius": 64, "dtype": "f32", "c_in": 32, "c_out": 32,
         "kernel": 3, "stride": 1, "train": False, "pairs": False},
        # training in fp32: part of a room, ragged row count, bias, widening layer, forward and backward
        {"name": "room-f32-train", "op": "conv", "scene": "rooms", "scenes": 1, "voxels": 48_503, "dtype": "f32",
         "c_in": 32, "c_out": 64, "kernel": 3, "stride": 1, "train": True, "pairs": False},
        # the headline layer on the headline batch, with the pair lists of its kernel map
        {"name": "rooms8-bf16", "op": "conv", "scene": "rooms", "scenes": 8, "voxels": FULL_ROOM, "dtype": "bf16",
         "c_in": 64, "c_out": 64, "kernel": 3, "stride": 1, "train": False, "pairs": True},
        # the same layer trained: forward, input gradient, weight gradient
        {"name": "rooms8-bf16-train", "op": "conv", "scene": "rooms", "scenes": 8, "voxels": FULL_ROOM,
         "dtype": "bf16", "c_in": 64, "c_out": 64, "kernel": 3, "stride": 1, "train": True, "pairs": False},
        # the second layer of that configuration: 2^3 stride 2 down to a new, coarser map
        {"name": "rooms8-bf16-down", "op": "conv", "scene": "rooms", "scenes": 8, "voxels": FULL_ROOM, "dtype": "bf16",
         "c_in": 64, "c_out": 128, "kernel": 2, "stride": 2, "train": False, "pairs": False},
        # two lidar sweeps through the five-layer chain (4-channel stem, down, transposed up), trained
        {"name": "sweeps2-bf16-train", "op": "chain", "sweeps": 2, "points": 120_000},
        # 4-D clips: 81 offsets, the largest map of the configurations
        {"name": "clips4-bf16", "op": "clips", "clips": 4, "frames": 8, "voxels": FULL_ROOM},
        # a training step of an encoder/decoder: batch norm, ReLU, down, transposed up, skip, head, cross entropy
        {"name": "encdec-bf16-train", "op": "encdec", "scenes": 4, "voxels": FULL_ROOM},
        # the benchmark's network (four levels, some thirty layers) serving one ordinary frame
        {"name": "unet-bf16-infer", "op": "unet", "scenes": 1, "voxels": 80_003},
        # the input step: raw points of eight sweeps to averaged voxels
        {"name": "sweeps8-voxelize", "op": "voxelize", "sweeps": 8, "points": 120_000, "channels": 4, "voxel": 0.2},
        # 2^3 maximum pooling of a feature map, forward and backward
        {"name": "rooms2-bf16-pool", "op": "pool", "scenes": 2, "voxels": FULL_ROOM, "dtype": "bf16", "channels": 64,
         "mode": "max"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["conv", "conv", "conv", "conv", "chain", "clips", "encdec", "unet", "voxelize", "pool"])
    if op == "conv":
        dtype = rng.choice(["f32", "bf16", "bf16"])
        bf16, train = dtype == "bf16", rng.random() < 0.5
        case = {"op": op, "dtype": dtype, "c_in": rng.choice([4, 32, 48, 64, 96, 128] if bf16 else [4, 32, 48, 64]),
                "c_out": rng.choice([32, 64, 96, 128] if bf16 else [32, 48, 64]), "train": train, "pairs": False}
        case["kernel"], case["stride"] = rng.choice([(3, 1), (3, 1), (3, 1), (2, 2)])
        most = 1_200_000 if bf16 else 120_000
        if rng.random() < 0.3:
            return dict(case, scene="shell", radius=_log(rng, 6, math.sqrt(most / 25.0)))
        rows = _log(rng, 1_000, most)
        scenes = -(-rows // FULL_ROOM)
        return dict(case, scene="rooms", scenes=scenes, voxels=rows // scenes, pairs=not train and rng.random() < 0.5)
    if op == "chain":
        return {"op": op, "sweeps": rng.randint(1, 4), "points": _log(rng, 20_000, 120_000)}
    if op == "clips":
        return {"op": op, "clips": rng.randint(1, 4), "frames": rng.randint(2, 8), "voxels": _log(rng, 5_000, FULL_ROOM)}
    if op == "encdec":
        return {"op": op, "scenes": rng.randint(2, 4), "voxels": _log(rng, 60_000, FULL_ROOM)}
    if op == "unet":
        return {"op": op, "scenes": rng.randint(1, 4), "voxels": _log(rng, 10_000, FULL_ROOM)}
    if op == "voxelize":
        return {"op": op, "sweeps": rng.randint(1, 8), "points": _log(rng, 5_000, 120_000),
                "channels": rng.choice([1, 3, 4, 16]), "voxel": rng.choice([0.1, 0.2, 0.4])}
    return {"op": op, "scenes": rng.randint(1, 8), "voxels": _log(rng, 2_000, FULL_ROOM),
            "dtype": rng.choice(["f32", "bf16"]), "channels": rng.choice([16, 32, 64, 128]),
            "mode": rng.choice(["max", "avg", "sum"])}


# --- scenes ---------------------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _room(index, n):
    """``n`` voxels [n, 3] of room number ``index``: floor, four walls, ten boxes on a 200 x 200 x 60 grid, jittered
    by one voxel. Fewer than a whole room's voxels are the ones nearest to one of them (a crop, not a thinner room)."""
    g = _generator(2000 + index)
    size = torch.tensor([200, 200, 60], device=DEV)
    per = FULL_ROOM
    parts = []

    def surface(lo, hi, axis, value, count):
        lo, hi = torch.tensor(lo, device=DEV), torch.tensor(hi, device=DEV)
        p = lo + (torch.rand((count, 3), generator=g, device=DEV) * (hi - lo + 1)).long()
        p[:, axis] = value
        parts.append(p)

    surface((0, 0, 0), (199, 199, 0), 2, 0, per)
    for axis in (0, 1):
        for value in (0, 199):
            surface((0, 0, 0), (0, 199, 59) if axis == 0 else (199, 0, 59), axis, value, per // 3)
    boxes = torch.rand((10, 5), generator=g, device=DEV).tolist()
    for b in boxes:
        lo = (10 + int(b[0] * 141), 10 + int(b[1] * 141), 0)
        hi = (min(lo[0] + 10 + int(b[2] * 31), 199), min(lo[1] + 10 + int(b[3] * 31), 199), 5 + int(b[4] * 36))
        for axis in range(3):
            for value in (lo[axis], hi[axis]):
                surface(lo, hi, axis, value, per // 12)
    p = torch.cat(parts)
    p = (p + torch.randint(-1, 2, p.shape, generator=g, device=DEV)).clamp_(min=0).minimum(size - 1)
    key = torch.unique((p[:, 0] * 200 + p[:, 1]) * 60 + p[:, 2])
    key = key[torch.randperm(key.numel(), generator=g, device=DEV)][:FULL_ROOM]
    p = torch.stack([key // 12000, (key // 60) % 200, key % 60], 1)
    return p[((p - p[0]) ** 2).sum(1).argsort(stable=True)[:n]].int()


def _shell(radius):
    """All voxels of the shell | |x| - radius | < 1."""
    r = torch.arange(-(radius + 1), radius + 2, device=DEV)
    d = torch.sqrt((r[:, None, None] ** 2 + r[None, :, None] ** 2 + r[None, None, :] ** 2).double())
    return (torch.nonzero((d - radius).abs() < 1) - (radius + 1)).int()


def _sweep(index, points):
    """``points`` returns [points, 3] in metres of a 64-beam sensor: elevation -25..3 degrees, 2048 azimuth steps,
    range uniform in 2..70 m."""
    g = _generator(3000 + index)
    pick = torch.randperm(64 * 2048, generator=g, device=DEV)[:points]
    e = torch.deg2rad(-25.0 + (pick // 2048) * (28.0 / 63.0))
    a = (pick % 2048) * (2.0 * math.pi / 2048.0)
    r = 2.0 + 68.0 * torch.rand(points, generator=g, device=DEV)
    return torch.stack([r * torch.cos(e) * torch.cos(a), r * torch.cos(e) * torch.sin(a), r * torch.sin(e)], 1)


def _sweep_voxels(index, points):
    """The sweep's voxels of 0.1 m."""
    v = torch.floor(_sweep(index, points) / 0.1).long() + 2048
    key = torch.unique((v[:, 0] * 4096 + v[:, 1]) * 4096 + v[:, 2])
    return (torch.stack([key // (4096 * 4096), (key // 4096) % 4096, key % 4096], 1) - 2048).int()


def _clip(index, frames, voxels):
    """One room translated by a constant velocity of 0..2 voxels per frame and axis: (x, y, z, t)."""
    room = _room(index, voxels)
    v = torch.randint(0, 3, (3,), generator=_generator(4000 + index), device=DEV, dtype=torch.int32)
    return torch.cat([torch.cat([room + t * v, torch.full((room.size(0), 1), t, dtype=torch.int32, device=DEV)], 1)
                      for t in range(frames)])


def _batch(g, scenes):
    """The scenes as one batch [N, 1 + D], each mirrored, turned and moved (voxels only) at random, its rows in random
    order."""
    out = []
    for b, p in enumerate(scenes):
        p = p.clone()
        turn = torch.randint(0, 8, (3,), generator=g, device=DEV).tolist()
        for axis in (0, 1):
            if turn[axis] & 1:   # cell c becomes -1 - c: rows that share a cell of a coarser grid still do
                p[:, axis] = -1 - p[:, axis] if p.dtype == torch.int32 else -p[:, axis]
        if turn[2] & 1:
            p[:, :2] = p[:, :2].flip(1)
        if p.dtype == torch.int32:
            p[:, 0] += 16 * turn[0]
            p[:, 1] += 16 * turn[1]
        p = p[torch.randperm(p.size(0), generator=g, device=DEV)]
        out.append(torch.cat([torch.full((p.size(0), 1), b, dtype=p.dtype, device=DEV), p], 1))
    return torch.cat(out).contiguous()


# --- preparation ----------------------------------------------------------------------------------------------

def _layer(cls, g, c_in, c_out, kernel, stride, dtype, bias=False, dimension=3):
    layer = cls(c_in, c_out, kernel_size=kernel, stride=stride, bias=bias, dimension=dimension)
    layer.to(DEV)
    layer.to(dtype)
    fan = (c_out if cls.__name__.endswith("Transpose") else c_in) * kernel ** dimension
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_((torch.rand(p.shape, generator=g, device=DEV) * 2 - 1) / math.sqrt(fan))
    return layer


def _normal(g, rows, channels, dtype):
    return torch.randn((rows, channels), generator=g, device=DEV).to(dtype)


def prepare(case, seed):
    C = cpp.load()
    g = _generator(seed)
    op = case["op"]
    state = {"C": C, "case": case}
    if op == "conv":
        coords = _batch(g, [_shell(case["radius"])] if case["scene"] == "shell" else
                        [_room(i, case["voxels"]) for i in range(case["scenes"])])
        dtype = DTYPES[case["dtype"]]
        layer = _layer(C.RiemannConvolution, g, case["c_in"], case["c_out"], case["kernel"], case["stride"], dtype,
                       bias=case["train"])
        state.update(coords=coords, feats=_normal(g, coords.size(0), case["c_in"], dtype), layer=layer)
        if case["train"]:
            rows = coords.size(0) if case["stride"] == 1 else _coarse_rows(coords, case["stride"])
            state.update(feats=state["feats"].requires_grad_(True), grad=_normal(g, rows, case["c_out"], dtype))
    elif op == "chain":
        bf, conv, up = torch.bfloat16, C.RiemannConvolution, C.RiemannConvolutionTranspose
        coords = _batch(g, [_sweep_voxels(i, case["points"]) for i in range(case["sweeps"])])
        layers = [_layer(conv, g, 4, 32, 3, 1, bf), _layer(conv, g, 32, 64, 3, 1, bf), _layer(conv, g, 64, 64, 2, 2, bf),
                  _layer(conv, g, 64, 128, 3, 1, bf), _layer(up, g, 128, 64, 2, 2, bf)]
        state.update(coords=coords, feats=_normal(g, coords.size(0), 4, bf), layers=layers,
                     grad=_normal(g, coords.size(0), 64, bf))
    elif op == "clips":
        coords = _batch(g, [_clip(i, case["frames"], case["voxels"]) for i in range(case["clips"])])
        state.update(coords=coords, feats=_normal(g, coords.size(0), 32, torch.bfloat16),
                     layer=_layer(C.RiemannConvolution, g, 32, 32, 3, 1, torch.bfloat16, dimension=4))
    elif op == "encdec":
        bf, conv, up = torch.bfloat16, C.RiemannConvolution, C.RiemannConvolutionTranspose
        coords = _batch(g, [_room(i, case["voxels"]) for i in range(case["scenes"])])
        layers = {"stem": _layer(conv, g, 4, 32, 3, 1, bf), "down": _layer(conv, g, 32, 64, 2, 2, bf),
                  "up": _layer(up, g, 64, 32, 2, 2, bf), "fuse": _layer(conv, g, 64, 32, 3, 1, bf),
                  "head": _layer(conv, g, 32, 20, 1, 1, bf, bias=True)}
        norms = {"stem": C.RiemannBatchNorm(32), "down": C.RiemannBatchNorm(64), "up": C.RiemannBatchNorm(32),
                 "fuse": C.RiemannBatchNorm(32)}
        for norm in norms.values():
            norm.to(DEV)
            norm.to(bf)
            norm.train(True)
        # position and one noisy channel in, the height band of the voxel as its class
        place = coords[:, 1:].float() / 100.0 - 1.0
        feats = torch.cat([place, 0.1 * _normal(g, coords.size(0), 1, torch.float32)], 1).to(bf)
        state.update(coords=coords, feats=feats, layers=layers, norms=norms, relu=C.RiemannReLU(False),
                     labels=(coords[:, 3] // 6).long().clamp_(0, 19))
    elif op == "unet":
        coords = _batch(g, [_room(i, case["voxels"]) for i in range(case["scenes"])])
        torch.manual_seed(seed)
        net = C.MinkUNet(4, 20, width=32, dimension=3)
        net.to(DEV)
        net.to(torch.bfloat16)
        net.train(False)
        state.update(coords=coords, feats=_normal(g, coords.size(0), 4, torch.bfloat16), net=net)
    elif op == "voxelize":
        scenes = [_sweep(i, case["points"]) / case["voxel"] for i in range(case["sweeps"])]
        # (a point exactly on a cell's border is moved off it: mirrored it would change cells)
        points = _batch(g, [torch.where(p == p.floor(), p + 0.25, p) for p in scenes])
        state.update(points=points, feats=_normal(g, points.size(0), case["channels"], torch.float32))
    elif op == "pool":
        coords = _batch(g, [_room(i, case["voxels"]) for i in range(case["scenes"])])
        dtype = DTYPES[case["dtype"]]
        layer = {"max": C.RiemannMaxPooling, "avg": C.RiemannAvgPooling, "sum": C.RiemannSumPooling}[case["mode"]]
        state.update(coords=coords, layer=layer(2, 2, 1, 3),
                     feats=_normal(g, coords.size(0), case["channels"], dtype).requires_grad_(True),
                     grad=_normal(g, _coarse_rows(coords, 2), case["channels"], dtype))
    return state


def _coarse_rows(coords, stride):
    c = coords.long()
    c[:, 1:] = torch.div(c[:, 1:], stride, rounding_mode="floor")
    c = c - c.min(0).values
    span = c.max(0).values + 1
    key = c[:, 0]
    for a in range(1, c.size(1)):
        key = key * span[a] + c[:, a]
    return int(torch.unique(key).numel())


# --- one pass -------------------------------------------------------------------------------------------------

def run(state):
    C, case = state["C"], state["case"]
    op = case["op"]
    if op == "conv":
        layer = state["layer"]
        if case["train"]:
            layer.zero_grad()
            state["feats"].grad = None
            y = layer(C.SparseTensor(state["feats"], state["coords"]))
            y.F.backward(state["grad"])
            return {"out": y.F, "coords": y.C, "grad_in": state["feats"].grad, "grad_kernel": layer.kernel.grad,
                    "grad_bias": layer.bias.grad}
        with torch.no_grad():
            x = C.SparseTensor(state["feats"], state["coords"])
            y = layer(x)
        out = {"out": y.F, "coords": y.C}
        if case["pairs"]:
            k, s = [case["kernel"]] * 3, [case["stride"]] * 3
            out["pairs"] = x.coordinate_manager.kernel_map_pairs(x.coordinate_map_key, y.coordinate_map_key, k, s,
                                                                 [1] * 3)
        return out
    if op == "chain":
        for layer in state["layers"]:
            layer.zero_grad()
        x = C.SparseTensor(state["feats"], state["coords"])
        for layer in state["layers"]:
            x = layer(x)
        x.F.backward(state["grad"])
        return {"out": x.F, "grads": [layer.kernel.grad for layer in state["layers"]]}
    if op == "clips":
        with torch.no_grad():
            y = state["layer"](C.SparseTensor(state["feats"], state["coords"]))
        return {"out": y.F, "coords": y.C}
    if op == "encdec":
        layers, norms, relu = state["layers"], state["norms"], state["relu"]
        for layer in layers.values():
            layer.zero_grad()
        for norm in norms.values():
            norm.weight.grad = norm.bias.grad = None

        def block(name, x):
            return relu(norms[name](layers[name](x)))

        skip = block("stem", C.SparseTensor(state["feats"], state["coords"]))
        x = block("up", block("down", skip))
        y = layers["head"](block("fuse", C.cat([x, skip]))).F
        loss = torch.nn.functional.cross_entropy(y.float(), state["labels"])
        loss.backward()
        return {"out": y, "loss": loss, "kernels": {k: v.kernel.grad for k, v in layers.items()},
                "bias": layers["head"].bias.grad,
                "norms": {k: [v.weight.grad, v.bias.grad, v.running_mean, v.running_var] for k, v in norms.items()}}
    if op == "unet":
        with torch.no_grad():
            return {"out": state["net"](C.SparseTensor(state["feats"], state["coords"])).F}
    if op == "voxelize":
        y = C.TensorField(state["feats"], state["points"]).sparse()
        return {"out": y.F, "coords": y.C}
    state["feats"].grad = None
    y = state["layer"](C.SparseTensor(state["feats"], state["coords"]))
    y.F.backward(state["grad"])
    return {"out": y.F, "coords": y.C, "grad_in": state["feats"].grad}


# --- what a pass cannot do without ----------------------------------------------------------------------------

def _rows(case):
    if case.get("scene") == "shell":
        return 24.9 * case["radius"] ** 2
    if "clips" in case:
        return case["clips"] * case["frames"] * case["voxels"]
    if "sweeps" in case:
        return case["sweeps"] * case["points"]
    return case["scenes"] * case["voxels"]


def work(case):
    op, n = case["op"], _rows(case)
    if op == "conv":
        e = 4 if case["dtype"] == "f32" else 2
        down = case["stride"] > 1
        rows_out = n * COARSER[case["scene"]] if down else n
        pairs = n if down else n * PAIRS[case["scene"]]
        weights = case["kernel"] ** 3 * case["c_in"] * case["c_out"] * e
        flops = 2.0 * pairs * case["c_in"] * case["c_out"]
        # coordinates and features in, coordinates and features out, weights once
        size = 16 * (n + rows_out) + e * (n * case["c_in"] + rows_out * case["c_out"]) + weights
        if case["train"]:  # gradient of the output in, gradients of the input and of the weights out
            size += e * (rows_out * case["c_out"] + n * case["c_in"]) + weights
            flops *= 3
        if case["pairs"]:
            size += 8 * pairs
        return {"bytes": size, "flops": flops}
    if op == "chain":
        p, m = n * PAIRS["sweeps"], n * COARSER["sweeps"] * PAIRS["sweeps"]
        fwd = 2.0 * (p * (4 * 32 + 32 * 64) + n * 64 * 64 + m * 64 * 128 + n * 128 * 64)
        weights = 2 * (27 * (4 * 32 + 32 * 64 + 64 * 128) + 8 * (64 * 64 + 128 * 64))
        return {"bytes": n * (16 + 2 * (4 + 64 + 64)) + 2 * weights, "flops": 3 * fwd - 2.0 * p * 4 * 32}
    if op == "clips":
        return {"bytes": n * (2 * 20 + 2 * 64) + 81 * 32 * 32 * 2, "flops": 2.0 * n * PAIRS["clips"] * 32 * 32}
    if op in ("encdec", "unet"):
        rows = [n * COARSER["rooms"] ** s for s in range(4)]
        p = [r * PAIRS["rooms"] for r in rows]
        stem, head = 2.0 * p[0] * 4 * 32, 2.0 * rows[0] * 32 * 20
        if op == "encdec":
            fwd = stem + 4.0 * rows[0] * 32 * 64 + 2.0 * p[0] * 64 * 32 + head
            weights = 2 * (27 * (4 * 32 + 64 * 32) + 16 * 32 * 64 + 32 * 20)
            return {"bytes": n * (16 + 8 + 2 * 20 + 8) + 2 * weights, "flops": 3 * fwd - stem}
        # the network at width 32: c = 32 * 2^s channels on level s, see riemann_cpp/networks.hpp
        fwd, weights = stem + head, 27 * 4 * 32 + 32 * 20
        for s in range(4):
            c = 32 * 2 ** s
            fwd += 8.0 * p[s] * c * c
            weights += 27 * 4 * c * c
            if s > 0:
                h = c // 2
                fwd += 4.0 * rows[s - 1] * h * c + 2.0 * p[s - 1] * (c * h + 2 * h * h)
                weights += 16 * h * c + 27 * (c * h + 2 * h * h)
        return {"bytes": n * (16 + 2 * (4 + 20)) + 2 * weights, "flops": fwd}
    if op == "voxelize":
        return {"bytes": n * (16 + 4 * case["channels"]) * 2, "flops": n * case["channels"]}
    e = 4 if case["dtype"] == "f32" else 2
    coarse = n * COARSER["rooms"]
    return {"bytes": 16 * (n + coarse) + 2 * e * case["channels"] * (n + coarse), "flops": n * case["channels"]}


def tolerance(case):
    op = case["op"]
    if op == "pool" and case["mode"] == "max":
        return "exact"           # values are selected and copied
    if op == "voxelize" or case.get("dtype") == "f32":
        return {"rel": 1e-5}     # fp32 sums in another order
    if op in ("encdec", "unet"):
        return {"rel": 3e-2}     # many layers, each rounding what it hands on to bf16, and gradients back through them
    return {"rel": 1e-2}         # fp32 sums rounded to bf16
