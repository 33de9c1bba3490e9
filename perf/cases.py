"""The work that the framework is timed on: single operators, the SS2D core and whole backbones, each in the direction,
data type and layout in which a VMamba program uses it.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` another one of the same ranges,
`prepare(case, seed)` what the program holds before the call, `run(state)` one pass through the public entry points,
`work(case)` the bytes and operations of a pass and `tolerance(case)` how far two correct implementations may differ.

Value distributions: maps and raw step sizes N(0, 1), step-size bias = inverse softplus of dt log-uniform in
[1e-3, 1e-1], A = -(1 .. N), D = 1, weights normal (std 0.02 for the dense layers of a backbone,
1 / sqrt(fan-in) for convolutions and the core's projections).
"""
import math

import torch

import vmamba_b200 as vb
from vmamba_b200.backbone import CONFIGS

ROUTES = 4
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}
CLASSES = 1000
MLP_RATIO = 4
# of a drawn case: bounds that keep it below the largest listed one
MOST_SCAN_UPDATES = 1 << 29         # (row, position, state)
MOST_SCAN_ELEMENTS = 1 << 26        # (row, position)
MOST_MAP_ELEMENTS = 1 << 25         # (image, channel, pixel)
MOST_BACKBONE_FLOPS = 1.0e12


# ------------------------------------------------------------------------------------------------ the cases
def _scan(train, dtype, batch, channels, states, length):
    return {"kind": "scan", "train": train, "dtype": dtype, "batch": batch, "channels": channels, "states": states, "length": length}


def _cross(train, dtype, batch, channels, height, width):
    return {"kind": "cross", "train": train, "dtype": dtype, "batch": batch, "channels": channels, "height": height, "width": width}


def _core(train, dtype, batch, channels, states, height, width):
    return {"kind": "core", "train": train, "dtype": dtype, "batch": batch, "channels": channels, "states": states,
            "height": height, "width": width}


def _backbone(model, call, features, dtype, batch, height, width):
    return {"kind": "backbone", "model": model, "call": call, "features": features, "dtype": dtype, "batch": batch,
            "height": height, "width": width}


def listed():
    return [
        # the selective scan of one image in the last stage of a classifier: the smallest call there is
        {"name": "scan_one_image", **_scan(False, "bf16", 1, 768, 1, 49)},
        # inference of the sixteen-state models (forward_type v0) on their first stage
        {"name": "scan_16_states", **_scan(False, "bf16", 16, 192, 16, 3136)},
        # few long rows: one image of a dense-prediction model, a length that no vector width divides
        {"name": "scan_long_rows", **_scan(False, "bf16", 1, 256, 1, 16385)},
        # training step of the operator at the first stage of VMamba-T, per GPU
        {"name": "scan_train", **_scan(True, "bf16", 32, 96, 1, 3136)},
        # training of a sixteen-state model in fp32, ragged length
        {"name": "scan_train_16_states", **_scan(True, "f32", 4, 384, 16, 1001)},
        # CrossScan and CrossMerge of a training step on a map with two odd sides
        {"name": "cross_train", **_cross(True, "bf16", 8, 192, 37, 53)},
        # the fused core as it stands in a reference model after enable_fused: batch-major map, second stage
        {"name": "core_fused", **_core(False, "bf16", 64, 192, 1, 28, 28)},
        # the differentiable core of a training step, first stage of VMamba-T
        {"name": "core_train", **_core(True, "bf16", 32, 96, 1, 56, 56)},
        # serving: one image from pinned host memory, logits back to the host
        {"name": "serve_one_image", **_backbone("vmamba_tiny_s1l8", "host", False, "bf16", 1, 224, 224)},
        # the throughput setting that VMamba-T is quoted on
        {"name": "tiny_batch_128", **_backbone("vmamba_tiny_s1l8", "graph", False, "bf16", 128, 224, 224)},
        # feature maps of photographs whose sides are no multiple of the stride, called without a captured graph
        {"name": "small_photographs", **_backbone("vmamba_small_s2l15", "module", True, "f16", 2, 427, 640)},
        # the dense-prediction backbone at 1024 x 1024, the share of one GPU of eight
        {"name": "base_1024", **_backbone("vmamba_base_s2l15", "graph", True, "bf16", 2, 1024, 1024)},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(max(low, high))))))


def _channels(rng, low, high):
    return 8 * _log_int(rng, low // 8, high // 8)       # the models' channel counts are multiples of 8 and more


def draw(rng):
    kind = rng.choice(("scan", "scan", "cross", "core", "core", "backbone", "backbone"))
    if kind == "scan":
        train, dtype, states = rng.random() < 0.5, rng.choice(("bf16", "bf16", "f16", "f32")), rng.choice((1, 1, 4, 8, 16, 16))
        channels, length = _channels(rng, 32, 1024), _log_int(rng, 49, 65536)
        most = min(MOST_SCAN_ELEMENTS, MOST_SCAN_UPDATES // states) // (ROUTES * length)      # images times channels
        channels = min(channels, most // 8 * 8)
        return _scan(train, dtype, _log_int(rng, 1, min(most // channels, 256)), channels, states, length)
    if kind in ("cross", "core"):
        train, dtype = rng.random() < 0.5, rng.choice(("bf16", "bf16", "f16", "f32"))
        height = _log_int(rng, 7, 256)
        width = height if rng.random() < 0.5 else min(256, max(7, int(height * rng.uniform(0.6, 1.7))))
        channels = min(_channels(rng, 64, 1024), MOST_MAP_ELEMENTS // (height * width) // 8 * 8)
        batch = _log_int(rng, 1, min(128, max(1, MOST_MAP_ELEMENTS // (channels * height * width))))
        if kind == "cross":
            return _cross(train, dtype, batch, channels, height, width)
        return _core(train, dtype, batch, channels, rng.choice((1, 1, 1, 16)), height, width)
    model = rng.choice(sorted(CONFIGS))
    features = rng.random() < 0.4
    height = _log_int(rng, 96, 1024)
    width = height if rng.random() < 0.5 else min(1024, max(96, int(height * rng.uniform(0.6, 1.7))))
    one = _backbone_flops(model, features, 1, height, width)
    batch = _log_int(rng, 1, min(128, max(1, int(MOST_BACKBONE_FLOPS / one))))
    return _backbone(model, rng.choice(("graph", "module", "host")), features, rng.choice(("bf16", "bf16", "f16")), batch, height, width)


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, shape, dtype=torch.float32, std=1.0):
    t = torch.randn(shape, device="cuda", generator=g)
    return (t if std == 1.0 else t.mul_(std)).to(dtype)


def _dt_bias(g, n):
    dt = torch.exp(torch.rand(n, device="cuda", generator=g) * (math.log(0.1) - math.log(1e-3)) + math.log(1e-3))
    return dt + torch.log(-torch.expm1(-dt))


def _rank(channels):
    return math.ceil(channels / 16)


def _core_parameters(g, channels, states, rank):
    """Parameters of one SS2D core under the names of a model's state dict, fp32."""
    rows = ROUTES * channels
    return {
        "x_proj.weight": _randn(g, (ROUTES * (rank + 2 * states), channels), std=channels ** -0.5),
        "dt_projs.weight": _randn(g, (rows, rank), std=rank ** -0.5),
        "dt_projs_bias": _dt_bias(g, rows).view(ROUTES, channels),
        "A_logs": torch.log(torch.arange(1, states + 1, device="cuda", dtype=torch.float32)).repeat(rows, 1),
        "Ds": torch.ones(rows, device="cuda"),
        "out_norm.weight": torch.ones(channels, device="cuda"),
        "out_norm.bias": torch.zeros(channels, device="cuda"),
    }


def _state_dict(g, model):
    """Random weights of a backbone with a classifier and the feature norms, in the key layout of its checkpoints."""
    cfg = CONFIGS[model]
    dims, depths = cfg["dims"], cfg["depths"]
    sd = {}

    def norm(name, n):
        sd[name + ".weight"], sd[name + ".bias"] = torch.ones(n, device="cuda"), torch.zeros(n, device="cuda")

    def dense(name, out, *fan, bias=True):
        sd[name + ".weight"] = _randn(g, (out,) + fan, std=0.02)
        if bias:
            sd[name + ".bias"] = torch.zeros(out, device="cuda")

    def conv(name, out, inn):
        std = (inn * 9) ** -0.5
        sd[name + ".weight"], sd[name + ".bias"] = _randn(g, (out, inn, 3, 3), std=std), _randn(g, (out,), std=std)

    conv("patch_embed.0", dims[0] // 2, 3)
    norm("patch_embed.2", dims[0] // 2)
    conv("patch_embed.5", dims[0], dims[0] // 2)
    norm("patch_embed.7", dims[0])
    for i, (dim, depth) in enumerate(zip(dims, depths)):
        inner = int(dim * cfg["ssm_ratio"])
        for j in range(depth):
            p = "layers.%d.blocks.%d." % (i, j)
            norm(p + "norm", dim)
            dense(p + "op.in_proj", inner, dim, bias=False)
            sd[p + "op.conv2d.weight"] = _randn(g, (inner, 1, 3, 3), std=1 / 3)
            for k, v in _core_parameters(g, inner, cfg["d_state"], _rank(dim)).items():
                sd[p + "op." + k] = v
            dense(p + "op.out_proj", dim, inner, bias=False)
            norm(p + "norm2", dim)
            dense(p + "mlp.fc1", MLP_RATIO * dim, dim)
            dense(p + "mlp.fc2", dim, MLP_RATIO * dim)
        norm("outnorm%d" % i, dim)
        if i + 1 < len(dims):
            conv("layers.%d.downsample.1" % i, dims[i + 1], dim)
            norm("layers.%d.downsample.3" % i, dims[i + 1])
    norm("classifier.norm", dims[-1])
    dense("classifier.head", CLASSES, dims[-1])
    return sd


def _leaf(t):
    return t.requires_grad_(True)


def prepare(case, seed):
    g = _generator(seed)
    dt = DTYPES[case["dtype"]]
    B = case["batch"]
    s = {"case": case}
    if case["kind"] == "scan":
        C, N, L = case["channels"], case["states"], case["length"]
        rows = ROUTES * C
        s["u"], s["delta"] = _randn(g, (B, rows, L), dt), _randn(g, (B, rows, L), dt)
        s["Bs"], s["Cs"] = _randn(g, (B, ROUTES, N, L), dt), _randn(g, (B, ROUTES, N, L), dt)
        s["A"] = -torch.arange(1, N + 1, device="cuda", dtype=torch.float32).repeat(rows, 1)
        s["D"], s["bias"] = torch.ones(rows, device="cuda"), _dt_bias(g, rows)
        if case["train"]:
            s["leaves"] = [_leaf(s[k]) for k in ("u", "delta", "A", "Bs", "Cs", "D", "bias")]
            s["dout"] = _randn(g, (B, rows, L))
    elif case["kind"] == "cross":
        C, H, W = case["channels"], case["height"], case["width"]
        s["x"] = _randn(g, (B, C, H, W), dt)
        s["ys"] = _randn(g, (B, ROUTES, C, H, W))               # the scan hands fp32 routes to the merge
        if case["train"]:
            _leaf(s["x"]), _leaf(s["ys"])
            s["dxs"], s["dy"] = _randn(g, (B, ROUTES, C, H * W), dt), _randn(g, (B, C, H * W))
    elif case["kind"] == "core":
        C, N, H, W = case["channels"], case["states"], case["height"], case["width"]
        R = _rank(C)
        par = _core_parameters(g, C, N, R)
        s["x"] = torch.nn.functional.silu(_randn(g, (B, C, H, W), dt))      # the core follows a SiLU
        order = [par[k] for k in ("x_proj.weight", "dt_projs.weight", "dt_projs_bias", "A_logs", "Ds", "out_norm.weight", "out_norm.bias")]
        if case["train"]:
            s["leaves"] = [_leaf(s["x"])] + [_leaf(t) for t in order]
            s["dout"] = _randn(g, (B, C, H, W), dt)
        else:
            s["weights"] = vb.CoreWeights.build(*order, d_state=N, dt_rank=R, dtype=dt)
    else:
        shape = (B, 3, case["height"], case["width"])
        model = vb.VSSMInfer.from_state_dict(_state_dict(g, case["model"]), dtype=dt)
        images = _randn(g, shape, dt)
        if case["call"] == "module":
            s["model"], s["images"] = model, images
        else:
            s["runner"] = vb.GraphedBackbone(model, shape, features=case["features"], dtype=dt)
            s["images"] = images
            if case["call"] == "host":
                out = s["runner"].output
                pinned = lambda t: torch.empty(t.shape, dtype=t.dtype, pin_memory=True)      # noqa: E731
                s["images"] = images.cpu().pin_memory()
                s["result"] = [pinned(t) for t in out] if case["features"] else pinned(out)
    return s


# ------------------------------------------------------------------------------------------------ a pass
def run(s):
    case = s["case"]
    if case["kind"] == "scan":
        y = vb.selective_scan_fn(s["u"], s["delta"], s["A"], s["Bs"], s["Cs"], s["D"], s["bias"], True)
        return [y, *torch.autograd.grad(y, s["leaves"], s["dout"])] if case["train"] else y
    if case["kind"] == "cross":
        xs, y = vb.cross_scan_fn(s["x"]), vb.cross_merge_fn(s["ys"])
        return [xs, y, *torch.autograd.grad([xs, y], [s["x"], s["ys"]], [s["dxs"], s["dy"]])] if case["train"] else [xs, y]
    if case["kind"] == "core":
        if not case["train"]:
            return vb.ss2d_core(s["x"], s["weights"])
        y = vb.ss2d_core_autograd(*s["leaves"], d_state=case["states"], dt_rank=_rank(case["channels"]))
        return [y, *torch.autograd.grad(y, s["leaves"], s["dout"])]
    if case["call"] == "module":
        return s["model"].features(s["images"]) if case["features"] else s["model"](s["images"])
    if case["call"] == "graph":
        return s["runner"](s["images"])
    return s["runner"].infer_host(s["images"], s["result"])


# ------------------------------------------------------------------------------------------------ what a pass has to do
def _scan_flops(rows, states, length):
    """Nine operations per (row, position, state) and one per (row, position) for the skip, as the models count it."""
    return rows * length * (9 * states + 1)


def _stage_sizes(height, width):
    """Map sizes after the patch embedding (two strided convolutions) and after each downsampling (one)."""
    half = lambda n: (n + 1) // 2               # noqa: E731
    h, w = half(height), half(width)
    sizes = [(h, w)]                            # between the two convolutions of the patch embedding
    for _ in range(4):
        h, w = half(h), half(w)
        sizes.append((h, w))
    return sizes


def _backbone_flops(model, features, batch, height, width):
    cfg = CONFIGS[model]
    dims, sizes = cfg["dims"], _stage_sizes(height, width)
    area = [h * w for h, w in sizes]
    n = 2 * 27 * (dims[0] // 2) * area[0] + 2 * 9 * (dims[0] // 2) * dims[0] * area[1]
    for i, (dim, depth) in enumerate(zip(dims, cfg["depths"])):
        inner, states, rank = int(dim * cfg["ssm_ratio"]), cfg["d_state"], _rank(dim)
        dense = 2 * dim * inner + 2 * MLP_RATIO * dim * dim + inner * ROUTES * (rank + 2 * states) + ROUTES * rank * inner + 9 * inner
        n += depth * (2 * dense * area[i + 1] + _scan_flops(ROUTES * inner, states, area[i + 1]))
        if i + 1 < len(dims):
            n += 2 * 9 * dim * dims[i + 1] * area[i + 2]
    return batch * (n + (0 if features else 2 * CLASSES * dims[-1]))


def _backbone_weights(model):
    cfg = CONFIGS[model]
    dims = cfg["dims"]
    n = 27 * (dims[0] // 2) + 9 * (dims[0] // 2) * dims[0] + CLASSES * dims[-1]
    for i, (dim, depth) in enumerate(zip(dims, cfg["depths"])):
        inner, rank = int(dim * cfg["ssm_ratio"]), _rank(dim)
        n += depth * (2 * dim * inner + 2 * MLP_RATIO * dim * dim + inner * (ROUTES * (2 * rank + 2 * cfg["d_state"]) + 9))
        n += 9 * dim * dims[i + 1] if i + 1 < len(dims) else 0
    return n


def work(case):
    B, e = case["batch"], SIZE[case["dtype"]]
    if case["kind"] == "scan":
        C, N, L = case["channels"], case["states"], case["length"]
        rows = B * ROUTES * C
        maps, small, par = rows * L, B * ROUTES * N * L, ROUTES * C * (N + 2) * 4
        if not case["train"]:       # u, delta, B, C in; fp32 result out
            return {"bytes": maps * (2 * e + 4) + 2 * small * e + par, "flops": _scan_flops(rows, N, L)}
        # and dout in; gradients of all of them out.  The reverse recurrence and the sums take about twice the forward's operations
        return {"bytes": maps * (2 * e + 4 + 4 + 2 * e) + 4 * small * e + 2 * par, "flops": 3 * _scan_flops(rows, N, L)}
    if case["kind"] == "cross":
        maps = B * case["channels"] * case["height"] * case["width"]
        once = maps * (e * (1 + ROUTES) + 4 * (ROUTES + 1))
        return {"bytes": (2 if case["train"] else 1) * once, "flops": (2 if case["train"] else 1) * maps * (ROUTES - 1)}
    if case["kind"] == "core":
        C, N, H, W = case["channels"], case["states"], case["height"], case["width"]
        L, R = H * W, _rank(C)
        par = ROUTES * C * (2 * R + 2 * N + N + 2)
        flops = B * (2 * L * C * ROUTES * (2 * R + 2 * N) + _scan_flops(ROUTES * C, N, L))
        maps = B * C * L * e
        if not case["train"]:
            return {"bytes": 2 * maps + par * e, "flops": flops}
        return {"bytes": 4 * maps + 2 * par * 4, "flops": 3 * flops}
    model, H, W = case["model"], case["height"], case["width"]
    if case["features"]:
        out = 4 * B * sum(d * h * w for d, (h, w) in zip(CONFIGS[model]["dims"], _stage_sizes(H, W)[1:]))
    else:
        out = B * CLASSES * e
    return {"bytes": B * 3 * H * W * e + _backbone_weights(model) * e + out, "flops": _backbone_flops(model, case["features"], B, H, W)}


def tolerance(case):
    half, short = case["dtype"] == "f16", case["dtype"] != "f32"
    if case["kind"] == "cross":
        return "exact"              # copies, and sums of four in a stated order
    if case["kind"] == "scan":
        if case["train"] and short:
            return {"rel": 1e-3 if half else 5e-3}              # gradients in 16 bits
        return {"rel": 2e-5}        # fp32 state and fp32 result, whatever the inputs are
    if case["kind"] == "core":      # 16-bit projections between the maps
        return {"rel": 2e-3 if half else 1e-2} if short else {"rel": 3e-5}
    return {"rel": 4e-3 if half else 2e-2}                      # 16-bit maps through fourteen to twenty-one blocks
