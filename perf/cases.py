"""The performance cases of the foveated path: what a program built on fovi_b200 has it do, through its public classes.

Eight kinds of work.  All sizes come from the benchmark, the tests and the shipped configurations, or are generic.

  sensor      RetinalTransform.forward, the reference's layout [B,F,C,N]: every model's first step
  front       FoveatedFrontEnd.forward, device tensors: sensor + five-layer KNNConv stack (the benchmark's workload)
  host        FoveatedFrontEnd.run_from_host: the same from pinned host images to pinned host activations
  tokens      sensor -> foveated patch embedding, the first stage of the vision-transformer configurations
  layer       sensor -> one KNNConvLayer with precision='fp32' (the exact float32 kernel)
  classify    FoveatedAlexNet.forward with the shipped backbone: images and fixations to logits, evaluation mode
  train       forward and backward of the five-layer stack in bf16, given the upstream gradient
  train_net   a supervised training step of the shipped backbone: sensor, network with batch statistics, cross entropy, backward

A program holds one model and meets many inputs, so models are built once per configuration with fixed parameters;
`prepare` makes the inputs (images uniform in [0,1), or bytes; fixation centres uniform in the central half of the image).
The two training kinds load the parameters from a master copy in every step, as a program does whose optimizer has just
changed them, so that whatever a layer derives from its parameters is derived anew in every step.
"""
import functools
import math

import numpy as np
import torch

DEVICE = "cuda"
FOV = 16
CHANNELS = [3, 64, 192, 384, 256, 256]            # the benchmark's stack: five layers on the a = 1 sensor
STRIDES, NEIGHBOURS = [2, 2, 1, 1, 1], [121, 25, 9, 9, 9]
SHIPPED = dict(in_res=64, in_channels=3, features_per_layer=[96, 256, 384, 384, 256], stride_per_layer=[2, 1, 1, 1, 1],
               pool_after=[0, 1, 4], k_per_layer=[121, 25, 9, 9, 9], out_res=1, auto_match_cart_resources=1, fov=16.0, cmf_a=0.5,
               norm_type="force_batch", ref_frame_mult=2, sample_cortex=True, n_classes=1000)
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "u8": torch.uint8}


# ------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a demonstration or an interactive loop: one image, one fixation, the transform's default sampler and sensor
        dict(name="sensor_one", kind="sensor", images=1, fixations=1, height=256, width=256, dtype="f32", a=0.5, mode="grid_nn"),
        # a data loader's batch with four fixations each, float32 as the reference's transform returns it
        dict(name="sensor_batch", kind="sensor", images=512, fixations=4, height=256, width=256, dtype="f32", a=1.0, mode="grid_bilinear"),
        # photographs at their own size, as bytes: rows that start on no 16-byte boundary
        dict(name="sensor_ragged", kind="sensor", images=61, fixations=3, height=375, width=500, dtype="u8", a=2.78, mode="grid_bilinear"),
        # serving: one image with four fixations through the benchmark's stack
        dict(name="front_single", kind="front", images=1, fixations=4, size=256, dtype="f32"),
        # the benchmark's workload
        dict(name="front_batch", kind="front", images=256, fixations=4, size=256, dtype="f32"),
        # the same work fed with the bytes that a data loader holds, from and to host memory
        dict(name="host_batch", kind="host", images=256, fixations=4, size=256, dtype="u8"),
        # the small and the large vision-transformer front ends (D = 384 and 1280, 63 tokens)
        dict(name="tokens_batch", kind="tokens", images=256, fixations=4, size=224, dtype="bf16", dim=384, patch=8),
        dict(name="tokens_large", kind="tokens", images=1024, fixations=8, size=256, dtype="bf16", dim=1280, patch=8),
        # the exact float32 layer, 49 neighbours in a 7x7 frame (parity runs, small float32 models)
        dict(name="layer_exact", kind="layer", images=8, size=224, channels=64, k=49),
        # evaluation of the shipped classifier on an uneven last batch
        dict(name="classify_ragged", kind="classify", images=75, fixations=4, size=256, dtype="f32"),
        # training: the stack as the benchmark trains it, and the shipped backbone
        dict(name="train_stack", kind="train", rows=1024),
        dict(name="train_backbone", kind="train_net", images=64, fixations=2, size=256),
    ]


def _between(rng, lo, hi):
    """An integer in [lo, hi], uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["sensor", "sensor", "front", "front", "host", "tokens", "tokens", "layer", "classify", "train", "train_net"])
    if kind == "sensor":
        h, w = _between(rng, 96, 512), _between(rng, 96, 512)
        if rng.random() < 0.5:          # half of the programs resize to a square of a round size first
            h = w = rng.choice([128, 192, 224, 256, 384])
        f = rng.randint(1, 8)
        most = max(1, min(512, int(512 * 4 / f), int(512 * 65536 / (h * w))))
        return dict(kind=kind, images=_between(rng, 1, most), fixations=f, height=h, width=w, dtype=rng.choice(["f32", "bf16", "u8"]),
                    a=rng.choice([0.5, 1.0, 2.78, 60.94]), mode=rng.choice(["grid_nn", "grid_bilinear"]))
    if kind in ("front", "host"):
        f = rng.randint(1, 8)
        return dict(kind=kind, images=_between(rng, 1, 1024 // f), fixations=f, size=rng.choice([224, 256]), dtype=rng.choice(["f32", "bf16", "u8"]))
    if kind == "tokens":
        f = rng.randint(1, 8)
        dim, patch = rng.choice([192, 384, 768, 1024, 1280]), rng.choice([4, 8])
        return dict(kind=kind, images=_between(rng, 1, 8192 // f // (4 if patch == 4 else 1)), fixations=f, size=rng.choice([224, 256]),
                    dtype=rng.choice(["f32", "bf16"]), dim=dim, patch=patch)
    if kind == "layer":
        return dict(kind=kind, images=_between(rng, 1, 64), size=rng.choice([224, 256]), channels=rng.choice([32, 64, 96]), k=rng.choice([9, 25, 49]))
    if kind == "classify":
        f = rng.randint(1, 8)
        return dict(kind=kind, images=_between(rng, 1, 1024 // f), fixations=f, size=rng.choice([224, 256]), dtype=rng.choice(["f32", "u8"]))
    if kind == "train":
        return dict(kind=kind, rows=_between(rng, 64, 1024))
    f = rng.randint(1, 4)
    return dict(kind=kind, images=_between(rng, 16, 256 // f), fixations=f, size=rng.choice([224, 256]))


# ----------------------------------------------------------------------------------------------------------- the models
@functools.lru_cache(maxsize=None)
def _retina(a, size, mode):
    from fovi_b200.sensing import RetinalTransform
    return RetinalTransform(resolution=64, start_res=size, fov=FOV, cmf_a=a, sampler=mode, fixation_size=size, device=DEVICE)


def _fill(tensor, rs, scale):
    """Parameters from NumPy's frozen stream: the same in every process."""
    tensor.data.copy_(torch.from_numpy((rs.standard_normal(tuple(tensor.shape)) * scale).astype(np.float32)))


@functools.lru_cache(maxsize=None)
def _stack(purpose):
    """The benchmark's stack; one for inference and one for training (a trained stack's parameters change)."""
    from fovi_b200.coords import auto_match_num_coords, get_in_out_coords
    from fovi_b200.knn import KNNConvLayer, KNNConvStack
    rs = np.random.RandomState(1)
    in_res, cart_res = auto_match_num_coords(FOV, 1.0, 64, "isotropic", 1)
    layers = []
    for i, k in enumerate(NEIGHBOURS):
        ic, oc, out_cart = get_in_out_coords(in_res, FOV, 1.0, STRIDES[i], auto_match_cart_resources=1, in_cart_res=cart_res)
        layer = KNNConvLayer(CHANNELS[i], CHANNELS[i + 1], k, ic, oc, device=DEVICE, ref_frame_side_length=int(np.ceil(2 * np.sqrt(k))), bias=True)
        _fill(layer.weight, rs, math.sqrt(2.0 / layer.weight.shape[1]))
        _fill(layer.bias, rs, 0.1)
        layers.append(layer)
        in_res, cart_res = oc.resolution, out_cart
    return KNNConvStack(layers).requires_grad_(purpose == "train")


@functools.lru_cache(maxsize=None)
def _front(size):
    from fovi_b200.pipeline import FoveatedFrontEnd
    return FoveatedFrontEnd(_retina(1.0, size, "grid_bilinear"), _stack("infer"))


@functools.lru_cache(maxsize=None)
def _embedding(dim, patch):
    from fovi_b200.knn import KNNPartitioningPatchEmbedding
    pe = KNNPartitioningPatchEmbedding(3, dim, in_res=64, fov=FOV, cmf_a=2.78, in_cart_res=64, cart_patch_size=patch, ref_frame_side_length=16,
                                       max_coord_val="auto", sample_cortex=True, bias=True, transposed=True, device=DEVICE)
    rs = np.random.RandomState(2)
    _fill(pe.weight, rs, math.sqrt(2.0 / pe.weight.shape[1]))
    _fill(pe.bias, rs, 0.1)
    return pe.requires_grad_(False)


@functools.lru_cache(maxsize=None)
def _exact_layer(channels, k):
    from fovi_b200.knn import KNNConvLayer
    coords = _retina(2.78, 224, "grid_bilinear").sampler.coords
    layer = KNNConvLayer(3, channels, k, coords, coords, device=DEVICE, ref_frame_side_length=int(math.isqrt(k)), bias=True, precision="fp32")
    rs = np.random.RandomState(3)
    _fill(layer.weight, rs, math.sqrt(2.0 / layer.weight.shape[1]))
    _fill(layer.bias, rs, 0.1)
    return layer.requires_grad_(False)


@functools.lru_cache(maxsize=None)
def _backbone(purpose):
    from fovi_b200.alexnet import KNNAlexNet
    net = KNNAlexNet(device=DEVICE, **SHIPPED)
    rs = np.random.RandomState(4)
    for block in net.layers:
        if hasattr(block, "conv"):
            _fill(block.conv.weight, rs, math.sqrt(2.0 / block.conv.weight.shape[1]))
            for t, centre, spread in ((block.norm.weight, 1.0, 0.2), (block.norm.bias, 0.0, 0.2), (block.norm.running_mean, 0.0, 0.1),
                                      (block.norm.running_var, 1.0, 0.2)):
                t.data.copy_(torch.from_numpy((centre + spread * (2 * rs.random_sample(tuple(t.shape)) - 1)).astype(np.float32)))
    _fill(net.classifier.weight, rs, 1 / math.sqrt(net.classifier.weight.shape[1]))
    _fill(net.classifier.bias, rs, 0.1)
    return net.train() if purpose == "train" else net.eval().requires_grad_(False)


# ----------------------------------------------------------------------------------------------------------- the inputs
def _images(gen, n, h, w, dtype):
    if dtype == "u8":
        return torch.randint(0, 256, (n, 3, h, w), generator=gen, device=DEVICE, dtype=torch.uint8)
    return torch.rand((n, 3, h, w), generator=gen, device=DEVICE).to(DTYPES[dtype])


def _fixations(gen, n, f):
    return 0.25 + 0.5 * torch.rand((n, f, 2), generator=gen, device=DEVICE)


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    s = dict(case=case)
    if kind == "sensor":
        s["retina"] = _retina(case["a"], min(case["height"], case["width"]), case["mode"])
        s["img"] = _images(gen, case["images"], case["height"], case["width"], case["dtype"])
        s["fix"] = _fixations(gen, case["images"], case["fixations"])
    elif kind in ("front", "host"):
        s["front"] = _front(case["size"])
        s["img"] = _images(gen, case["images"], case["size"], case["size"], case["dtype"])
        s["fix"] = _fixations(gen, case["images"], case["fixations"])
        if kind == "host":
            last = s["front"].stack.layers[-1]
            s["img"], s["fix"] = s["img"].cpu().pin_memory(), s["fix"].cpu().pin_memory()
            s["out"] = torch.empty((case["images"], case["fixations"], last.plan.n_out, last.out_channels), dtype=torch.bfloat16, pin_memory=True)
    elif kind == "tokens":
        s["retina"], s["embed"] = _retina(2.78, case["size"], "grid_bilinear"), _embedding(case["dim"], case["patch"])
        s["img"] = _images(gen, case["images"], case["size"], case["size"], case["dtype"])
        s["fix"] = _fixations(gen, case["images"], case["fixations"])
    elif kind == "layer":
        s["retina"], s["layer"] = _retina(2.78, case["size"], "grid_bilinear"), _exact_layer(case["channels"], case["k"])
        s["img"] = _images(gen, case["images"], case["size"], case["size"], "f32")
        s["fix"] = _fixations(gen, case["images"], 1)[:, 0].contiguous()
    elif kind == "classify":
        from fovi_b200.alexnet import FoveatedAlexNet
        s["net"] = FoveatedAlexNet(_retina(0.5, case["size"], "grid_bilinear"), _backbone("infer"))
        s["img"] = _images(gen, case["images"], case["size"], case["size"], case["dtype"])
        s["fix"] = _fixations(gen, case["images"], case["fixations"])
    elif kind == "train":
        s["stack"] = stack = _stack("train")
        rows, last = case["rows"], stack.layers[-1]
        s["x"] = torch.rand((rows, 3, stack.layers[0].plan.n_in), generator=gen, device=DEVICE).to(torch.bfloat16)
        # in the layout of the stack's result, a channels-last view
        s["gy"] = torch.randn((rows, last.plan.n_out, last.out_channels), generator=gen, device=DEVICE).to(torch.bfloat16).permute(0, 2, 1)
        s["master"] = [p.detach().clone() for p in stack.parameters()]
    elif kind == "train_net":
        s["retina"], s["net"] = _retina(0.5, case["size"], "grid_bilinear"), _backbone("train")
        s["img"] = _images(gen, case["images"], case["size"], case["size"], "f32")
        s["fix"] = _fixations(gen, case["images"], case["fixations"])
        s["label"] = torch.randint(0, SHIPPED["n_classes"], (case["images"] * case["fixations"],), generator=gen, device=DEVICE)
        s["master"] = [p.detach().clone() for p in s["net"].parameters()]
    else:
        raise ValueError(kind)
    return s


# ------------------------------------------------------------------------------------------------------------- one pass
def run(s):
    kind = s["case"]["kind"]
    if kind == "sensor":
        return s["retina"](s["img"], s["fix"])
    if kind == "front":
        return s["front"].forward(s["img"], s["fix"])
    if kind == "host":
        return s["front"].run_from_host(s["img"], s["fix"], s["out"])
    if kind == "tokens":
        points, rows = s["retina"].forward_points(s["img"], s["fix"], conv_plan=s["embed"].plan)
        return s["embed"].forward_points(points, batch=rows)
    if kind == "layer":
        return s["layer"](s["retina"](s["img"], s["fix"]))
    if kind == "classify":
        return s["net"](s["img"], s["fix"])
    if kind == "train":
        return _train_stack(s)
    return _train_backbone(s)


def _load(module, master):
    """The parameters as the optimizer left them; gradients of the last step are dropped."""
    params = list(module.parameters())
    with torch.no_grad():
        torch._foreach_copy_(params, master)
    for p in params:
        p.grad = None
    return params


def _train_stack(s):
    stack = s["stack"]
    params = _load(stack, s["master"])
    y = stack(s["x"])
    y.backward(s["gy"])
    return {"y": y.detach(), "grads": [p.grad for p in params]}


def _train_backbone(s):
    net = s["net"]
    params = _load(net, s["master"])
    x = s["retina"](s["img"], s["fix"])                              # [B,F,3,N]
    x = x.transpose(0, 1).reshape(-1, x.shape[2], x.shape[3])        # '(f b)', as the reference flattens fixations
    logits = net(x)
    loss = torch.nn.functional.cross_entropy(logits, s["label"])
    loss.backward()
    return {"logits": logits.detach(), "loss": loss.detach(), "grads": [p.grad for p in params]}


# --------------------------------------------------------------------------------------------------------- work, bounds
@functools.lru_cache(maxsize=None)
def _pixels(a, h, w, fixations, mode):
    """Distinct image pixels that one image's fixations read (mean of four draws), and the sensor's point count."""
    size = min(h, w)
    grid = _retina(a, size, mode).sampler.sampling_grid[0, 0].cpu().numpy().astype(np.float64)
    rs, total = np.random.RandomState(0), 0
    for _ in range(4):
        seen = np.zeros(h * w, bool)
        for r, c in 0.25 + 0.5 * rs.random_sample((fixations, 2)):
            ix, iy = grid[:, 0] * (size / 2) + c * w - 0.5, grid[:, 1] * (size / 2) + r * h - 0.5
            if mode == "grid_nn":
                taps = [(np.rint(ix), np.rint(iy))]
            else:
                x0, y0 = np.floor(ix), np.floor(iy)
                taps = [(x0 + i, y0 + j) for i in (0, 1) for j in (0, 1)]
            for x, y in taps:
                ok = (x >= 0) & (x < w) & (y >= 0) & (y < h)
                seen[(y[ok] * w + x[ok]).astype(np.int64)] = True
        total += int(seen.sum())
    return total / 4, grid.shape[0]


def _sensor_in(case, a, mode="grid_bilinear"):
    """Bytes of the pixels that a batch's fixations read, each once, and the sensor's point count."""
    h, w = case.get("height", case.get("size")), case.get("width", case.get("size"))
    px, n = _pixels(a, h, w, case.get("fixations", 1), mode)
    return case["images"] * 3 * px * {"f32": 4, "bf16": 2, "u8": 1}[case.get("dtype", "f32")], n


def work(case):
    kind = case["kind"]
    if kind == "sensor":
        inp, n = _sensor_in(case, case["a"], case["mode"])
        rows = case["images"] * case["fixations"]
        taps = 1 if case["mode"] == "grid_nn" else 4
        return {"bytes": inp + rows * 3 * n * 4, "flops": rows * n * 3 * 2 * taps}          # the transform returns float32
    if kind == "layer":
        layer = _exact_layer(case["channels"], case["k"])
        inp, _ = _sensor_in(case, 2.78)
        b = case["images"]
        return {"bytes": inp + layer.weight.numel() * 4 + b * layer.plan.n_out * case["channels"] * 4, "flops": b * layer.plan.flops_per_image()}
    if kind == "train":
        layers, rows = _stack("train").layers, case["rows"]
        fl = [rows * L.plan.flops_per_image() for L in layers]
        par = sum(L.weight.numel() for L in layers)
        last = layers[-1]
        return {"bytes": rows * 3 * layers[0].plan.n_in * 2 + 8 * par + 2 * rows * last.plan.n_out * last.out_channels * 2,
                "flops": 3 * sum(fl) - fl[0]}                                               # the first layer's input needs no gradient
    rows = case["images"] * case["fixations"]
    if kind in ("front", "host"):
        layers = _stack("infer").layers
        inp, _ = _sensor_in(case, 1.0)
        last = layers[-1]
        return {"bytes": inp + sum(L.weight.numel() for L in layers) * 2 + rows * last.plan.n_out * last.out_channels * 2,
                "flops": rows * sum(L.plan.flops_per_image() for L in layers)}
    if kind == "tokens":
        pe = _embedding(case["dim"], case["patch"])
        inp, _ = _sensor_in(case, 2.78)
        return {"bytes": inp + pe.weight.numel() * 2 + rows * pe.plan.n_out * case["dim"] * 2, "flops": rows * pe.plan.flops_per_image()}
    net = _backbone("infer" if kind == "classify" else "train")
    inp, _ = _sensor_in(case, 0.5)
    convs = [L.conv for L in net.layers if hasattr(L, "conv")]
    fl = [rows * c.plan.flops_per_image() for c in convs] + [2 * rows * net.classifier.weight.numel()]
    par = sum(p.numel() for p in net.parameters())
    if kind == "classify":
        return {"bytes": inp + 2 * par + rows * SHIPPED["n_classes"] * 4, "flops": sum(fl)}
    return {"bytes": inp + 8 * par, "flops": 3 * sum(fl) - fl[0]}


def tolerance(case):
    """Largest relative error another correct implementation at the same precision shows: about four times what the path
    differs by from the same computation in float64 (stack 2.5e-3, with bytes as inputs 5.4e-3; tokens 2.8e-3; classifier
    1.7e-3; exact layer 2.2e-7 on the same sensor output)."""
    return {
        "sensor": "exact",            # one rounding per operation in a stated order: bit-identical to the reference by contract
        "layer": {"rel": 2e-6},
        "front": {"rel": 2e-2}, "host": {"rel": 2e-2}, "tokens": {"rel": 1e-2}, "classify": {"rel": 1e-2},
        # Gradients pass through ReLU masks and pooling maxima, and each one that falls the other way replaces a whole term:
        # against float64 without any rounding the early layers' gradients differ by 0.03-0.14.  The bound is for an implementation that rounds
        # activations where this one does (bf16 operands, float32 sums), where only sums in another order move a mask.
        "train": {"rel": 3e-2}, "train_net": {"rel": 3e-2},
    }[case["kind"]]


# --------------------------------------------------------------------------------------------- the same in 64 bits, plain torch
def exact(case, seed):
    """What `run` returns for these inputs, in float64 (the neighbour and tap tables and the sensor's points are data).

    Inference is float64 throughout.  In the training kinds the forward pass rounds weights and activations to bf16 where
    the path states that it holds them in bf16, and everything else, the whole backward pass too, is float64: ReLU masks and
    pooling maxima are then those of the stated computation, so that a gradient's distance is the gradient's own error.
    The loss has no entry: the distance of a single number says nothing about precision, and the logits are compared."""
    s, kind = prepare(case, seed), case["kind"]
    if kind == "train":
        return _exact_train(s)
    if kind == "train_net":
        return _exact_train_net(s)
    front = s.get("front")
    x = _points64(front.retina if front else s["net"].retina if kind == "classify" else s["retina"], s["img"].to(DEVICE), s["fix"].to(DEVICE))
    if kind == "sensor":
        return x
    with torch.no_grad():
        if kind == "layer":
            return _conv64(x.transpose(1, 2), s["layer"]).transpose(1, 2)
        b, f = x.shape[:2]
        h = (x if kind == "host" else x.transpose(0, 1)).flatten(0, 1).transpose(1, 2)          # rows, points, channels
        if kind == "tokens":
            return _by_rows(lambda r: _conv64(r, s["embed"]), h)
        if kind == "classify":
            return _by_rows(lambda r: _net64(s["net"].network, r, batch_stats=False), h).unflatten(0, (f, b)).transpose(0, 1)
        y = _by_rows(lambda r: _stack64(front.stack.layers, r), h)
        return y.unflatten(0, (b, f)).cpu() if kind == "host" else y


def _by_rows(fn, h, step=512):
    return torch.cat([fn(r) for r in h.split(step)])


class _Bf16(torch.autograd.Function):
    """Rounds to bf16 on the way forward and hands the gradient on unchanged."""

    @staticmethod
    def forward(ctx, x):
        return x.to(torch.bfloat16).double()

    @staticmethod
    def backward(ctx, g):
        return g


def _points64(retina, img, fix):
    """All fixations' sensor points, [B,F,C,N] ([B,C,N] when `fix` has no fixation axis)."""
    many = fix.dim() == 3
    fix = fix if many else fix[:, None]
    b, c, h, w = img.shape
    size, sampler = float(retina.fixation_size), retina.sampler
    g = sampler.sampling_grid[0, 0].to(DEVICE).double()
    centre = fix.double()[:, :, None, :].flip(-1)                                                # (column, row)
    dims = torch.tensor([w, h], dtype=torch.float64, device=DEVICE)
    grid = 2 * (g * (size / 2) + centre * dims) / dims - 1                                       # [B,F,N,2]
    y = torch.nn.functional.grid_sample(img.double(), grid, mode=sampler.mode, padding_mode="zeros", align_corners=False)
    y = y.transpose(1, 2)
    return y if many else y[:, 0]


def _conv64(x, layer, weight=None, bias=None):
    """[rows, points, C] float64 -> [rows, output points, C_out]: one product per filter tap over the pairs that use it."""
    weight = layer.weight.double() if weight is None else weight
    bias = layer.bias.double() if bias is None and layer.bias is not None else bias
    idx, tap = layer.knn_indices_pad_token.numpy(), layer.tap.numpy()                            # [K,n_out], [n_out,K]
    k, n = np.nonzero(idx < x.shape[1])
    m, v = idx[k, n], tap[n, k]
    order = np.argsort(v, kind="stable")
    bounds = np.flatnonzero(np.r_[True, np.diff(v[order]) != 0, True])
    w = weight.reshape(weight.shape[0], x.shape[2], -1)
    y = torch.zeros((x.shape[0], tap.shape[0], weight.shape[0]), dtype=torch.float64, device=x.device)
    for lo, hi in zip(bounds[:-1], bounds[1:]):
        sel = order[lo:hi]
        src, dst = (torch.from_numpy(np.ascontiguousarray(t[sel]).astype(np.int64)).to(x.device) for t in (m, n))
        y = y.index_add_(1, dst, x.index_select(1, src) @ w[:, :, int(v[sel[0]])].t())
    return y if bias is None else y + bias


def _stack64(layers, h, round_=lambda t: t, params=None):
    for i, layer in enumerate(layers):
        w, b = (layer.weight.double(), layer.bias.double()) if params is None else params[2 * i:2 * i + 2]
        h = _conv64(round_(h), layer, round_(w), b)
        h = torch.relu(h) if i < len(layers) - 1 else h
    return h


def _net64(net, h, batch_stats, round_=lambda t: t, params=None):
    """The shipped backbone on [rows, points, C]: convolution, batch norm, ReLU, pooling; classifier on channel-major features."""
    p = {k: t.double() for k, t in net.named_parameters()} if params is None else params
    for i, layer in enumerate(net.layers):
        if hasattr(layer, "conv"):
            h = _conv64(round_(h), layer.conv, round_(p[f"layers.{i}.conv.weight"]), p.get(f"layers.{i}.conv.bias"))
            mean, var = (h.mean((0, 1)), h.var((0, 1), unbiased=False)) if batch_stats else (layer.norm.running_mean.double(), layer.norm.running_var.double())
            h = (h - mean) * torch.rsqrt(var + layer.norm.eps) * p[f"layers.{i}.norm.weight"] + p[f"layers.{i}.norm.bias"]
            h = torch.relu(h)
        pool = layer.pool if hasattr(layer, "conv") else layer
        if pool is not None:
            idx = pool.knn_indices_pad_token.to(h.device)                                        # [K,n_out], pads point past the end
            if pool.mode == "max":
                h = torch.nn.functional.pad(h, (0, 0, 0, 1), value=-math.inf)[:, idx].amax(1)
            else:
                h = torch.nn.functional.pad(h, (0, 0, 0, 1))[:, idx].sum(1) / (idx < pool._plan.n_in).sum(0)[:, None]
    return h.transpose(1, 2).flatten(1) @ p["classifier.weight"].t() + p["classifier.bias"]


def _exact_train(s):
    stack = s["stack"]
    params = [p.double().requires_grad_() for p in s["master"]]
    order = [n for n, _ in stack.named_parameters()]                                             # layers.i.weight, layers.i.bias
    by_layer = [params[order.index(f"layers.{i}.{t}")] for i in range(len(stack.layers)) for t in ("weight", "bias")]
    y = _stack64(stack.layers, s["x"].double().transpose(1, 2), _Bf16.apply, by_layer).transpose(1, 2)
    y.backward(s["gy"].double())
    return {"y": y.detach(), "grads": [p.grad for p in params]}


def _exact_train_net(s):
    net = s["net"]
    params = {n: p.double().requires_grad_() for (n, _), p in zip(net.named_parameters(), s["master"])}
    x = _points64(s["retina"], s["img"], s["fix"]).transpose(0, 1).flatten(0, 1).transpose(1, 2)
    logits = _net64(net, x, True, _Bf16.apply, params)
    torch.nn.functional.cross_entropy(logits, s["label"]).backward()
    return {"logits": logits.detach(), "loss": None, "grads": [p.grad for p in params.values()]}
