"""Kernels chosen by size and alignment, at the sizes where they can go wrong: edges of chunks, tiles and vectors, remainders, the
smallest and largest of their ranges.  Against the CPU oracle or a float64 statement.  Needs a GPU."""
import numpy as np
import pytest
import torch

from oracle import c_oracle as CO
from oracle import ss2d_oracle as O
from tests.test_gpu_bwd import NAMES, TD, TOL, _autograd, _random_case
from tests.test_gpu_ops import TOL_BF16, TOL_F32, _core_case, dev, host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vb():
    import vmamba_b200
    return vmamba_b200


@pytest.mark.parametrize("N,Cd,L,dt", [(2, 5, 31, "f32"), (3, 33, 64, "bf16"), (4, 32, 65, "f32"), (7, 9, 130, "f16"), (8, 40, 96, "bf16"),
                                       (16, 31, 33, "f32"), (16, 8, 1000, "bf16"), (16, 2, 2049, "f32"), (4, 800, 36, "bf16")])
def test_scan_states_forward_and_backward(vb, N, Cd, L, dt):
    """2 .. 16 states: padded state counts, rows that do not fill a CTA's 32, ragged chunks, single-element and vector rows, rows cut
    into segments (few rows, L >= 192)."""
    Bt, K = 2, 2
    u, delta, A, B, C, D, bias, dout = _random_case(Bt, K, Cd, N, L, seed=N * L)
    if dt != "f32":
        u, delta, B, C = (O._round_to(a, dt) for a in (u, delta, B, C))
    td = TD[dt]
    y = vb.selective_scan_fn(dev(u, td), dev(delta, td), dev(A), dev(B, td), dev(C, td), dev(D), dev(bias), True)
    assert O.max_rel_err(host(y), CO.selective_scan(u, delta, A, B, C, D, bias, True)) <= TOL_F32
    ref = O.selective_scan_bwd(u, delta, A, B, C, D, bias, dout, True, dt)
    for name, x, r in zip(NAMES, _autograd(vb, u, delta, A, B, C, D, bias, dout, True, True, dt), ref):
        assert O.max_rel_err(x, r) <= TOL[dt], name


@pytest.mark.parametrize("Cd,L,dt", [(1, 1, "f32"), (9, 7, "bf16"), (70, 64, "bf16"), (33, 65, "f32"), (5, 129, "f16"), (3, 255, "bf16"), (3, 257, "f32"),
                                     (2, 1026, "f32"), (2, 2500, "bf16"), (300, 260, "bf16"), (1, 4099, "bf16")])
def test_scan_one_state_forward_and_backward(vb, Cd, L, dt):
    """One state: rows sharing a warp, one and several warps per row, every alignment of the vectors, segments."""
    Bt, K = 2, 2
    u, delta, A, B, C, D, bias, dout = _random_case(Bt, K, Cd, 1, L, seed=L)
    if dt != "f32":
        u, delta, B, C = (O._round_to(a, dt) for a in (u, delta, B, C))
    td = TD[dt]
    y = vb.selective_scan_fn(dev(u, td), dev(delta, td), dev(A), dev(B, td), dev(C, td), dev(D), dev(bias), True)
    assert O.max_rel_err(host(y), CO.selective_scan(u, delta, A, B, C, D, bias, True)) <= TOL_F32
    ref = O.selective_scan_bwd(u, delta, A, B, C, D, bias, dout, True, dt)
    for name, x, r in zip(NAMES, _autograd(vb, u, delta, A, B, C, D, bias, dout, True, True, dt), ref):
        assert O.max_rel_err(x, r) <= TOL[dt], name


@pytest.mark.parametrize("shape", [(1, 1, 1, 3), (2, 5, 7, 7), (1, 90, 3, 5), (2, 3, 37, 53), (1, 2, 147, 183), (1, 3, 128, 129)])
@pytest.mark.parametrize("scans", [0, 1, 2])
@pytest.mark.parametrize("dt", ["f32", "bf16"])
def test_cross_padded_rows(vb, shape, scans, dt):
    """CrossScan, CrossMerge and the permutation of single rows with route rows padded to a multiple of eight."""
    from vmamba_b200 import _lib
    rng = np.random.default_rng(sum(shape))
    Bt, Cc, H, W = shape
    L, S = H * W, (H * W + 7) // 8 * 8
    td, code = TD[dt], {"f32": _lib.SS2D_F32, "bf16": _lib.SS2D_BF16}[dt]
    rnd = (lambda a: a) if dt == "f32" else O.round_bf16
    x, ys = rnd(rng.standard_normal(shape, dtype=np.float32)), rnd(rng.standard_normal((Bt, 4, Cc, L), dtype=np.float32))
    st = torch.cuda.current_stream().cuda_stream

    def call(fn, a, out, *more):
        p = _lib.CrossParams(a.data_ptr(), out.data_ptr(), code, scans, Bt, Cc, H, W, S)
        assert getattr(_lib.lib(), fn)(p, *more, st) == _lib.SS2D_OK
        return out
    pad = lambda a: torch.nn.functional.pad(dev(a, td), (0, S - L)).contiguous()      # noqa: E731
    want = O.cross_scan(x, scans).reshape(Bt, 4, Cc, L)
    got = call("ss2d_cross_scan", dev(x, td), torch.full((Bt, 4, Cc, S), 7.0, device="cuda", dtype=td))
    assert np.array_equal(host(got[..., :L]), want) and not host(got[..., L:]).any()
    if H * (W | 1) * 2 * (4 if dt == "f32" else 2) <= 200 * 1024:
        got = call("ss2d_cross_merge", pad(ys), torch.empty((Bt, Cc, L), device="cuda", dtype=td))
        if dt == "f32":
            assert np.array_equal(host(got), O.cross_merge(ys.reshape(Bt, 4, Cc, H, W), scans).reshape(Bt, Cc, L))
        else:                                          # rounded after every addition
            dense = vb.cross_merge_fn(dev(ys.reshape(Bt, 4, Cc, H, W), td), scans=scans)
            assert torch.equal(got, dense.view(Bt, Cc, L))
    rows = call("ss2d_cross_rows", pad(ys), torch.empty((Bt, 4, Cc, S), device="cuda", dtype=td), 0)
    per_route = np.stack([O.cross_scan(np.ascontiguousarray(ys[:, k]).reshape(shape), scans).reshape(Bt, 4, Cc, L)[:, k] for k in range(4)], 1)
    assert np.array_equal(host(rows[..., :L]), per_route)
    back = call("ss2d_cross_rows", rows, torch.empty_like(rows), 1)
    assert np.array_equal(host(back[..., :L]), ys)


@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("scans", [0, 1, 2, 3])
@pytest.mark.parametrize("H,W", [(48, 32), (40, 52), (32, 64), (64, 64), (66, 68), (130, 36), (72, 260)])
def test_cross_merge_of_whole_planes(vb, H, W, scans, dt):
    """Merge of planes with rows of whole vectors: one tile, several, ragged last ones, planes that do not fill a CTA."""
    ys = np.random.default_rng(H * W).standard_normal((1, 4, 5, H, W), dtype=np.float32)
    if dt != "f32":
        ys = O._round_to(ys, dt)
    got = host(vb.cross_merge_fn(dev(ys, TD[dt]), scans=scans)).reshape(1, 5, H * W)
    want = O.cross_merge(ys, scans).reshape(1, 5, H * W)
    assert np.abs(got - want).max() <= {"f32": 2e-6, "bf16": 0.1, "f16": 0.02}[dt]


@pytest.mark.parametrize("D,H,W,dt", [(16, 13, 13, "f32"), (15, 8, 17, "bf16"), (19, 27, 29, "f16"), (13, 57, 57, "bf16"), (14, 21, 21, "bf16"),
                                      (13, 54, 54, "f16"), (13, 36, 29, "f32"), (12, 75, 75, "bf16"), (13, 54, 80, "bf16"), (12, 96, 96, "bf16"),
                                      (17, 9, 9, "bf16"), (12, 101, 97, "f32"), (16, 7, 7, "bf16"), (40, 14, 14, "f16"), (24, 9, 11, "bf16")])
def test_core_any_plane_size(vb, D, H, W, dt):
    """The fused core on planes of any size (padded rows, both layouts) against the oracle."""
    c = _core_case(2, D, H, W, N=1, seed=H * W, Cmodel=24)
    ref = O.ss2d_core(c["x"], c["wx"], c["wdt"], c["bias"], c["A_logs"], c["Ds"], c["lw"], c["lb"], d_state=1, dt_rank=c["R"])
    td = TD[dt]
    w = vb.CoreWeights.build(*(dev(c[k]) for k in ("wx", "wdt", "bias", "A_logs", "Ds", "lw", "lb")), d_state=1, dt_rank=c["R"], dtype=td)
    x = dev(c["x"], td)
    y = vb.ss2d_core(x, w)
    assert O.max_rel_err(host(y), ref) <= (TOL_F32 if dt == "f32" else TOL_BF16)
    cm = vb.ss2d_core(x.transpose(0, 1).contiguous(), w, channel_major=True)
    assert O.max_rel_err(host(cm.transpose(0, 1)), host(y)) <= (TOL_F32 if dt == "f32" else TOL_BF16)
    assert torch.equal(y, vb.ss2d_core(x, w))


@pytest.mark.parametrize("D,N,H,W", [(16, 1, 14, 14), (17, 1, 13, 17), (14, 16, 5, 7), (13, 4, 33, 31), (12, 1, 1, 9)])
def test_core_training_node(vb, D, N, H, W):
    """The native node against the separate statements (fp32, which `oflex=False` still runs through)."""
    from vmamba_b200 import fused
    c = _core_case(2, D, H, W, N=N, seed=D * H, Cmodel=20)
    g = dev(np.random.default_rng(1).standard_normal(c["x"].shape, dtype=np.float32))
    res = []
    for oflex in (True, False):
        leaves = [dev(c[k]).requires_grad_(True) for k in ("x", "wx", "wdt", "bias", "A_logs", "Ds", "lw", "lb")]
        y = fused.ss2d_core_autograd(*leaves, d_state=N, dt_rank=c["R"], oflex=oflex)
        res.append([y.detach(), *torch.autograd.grad(y, leaves, g)])
    for a, b in zip(*res):
        assert a.shape == b.shape and O.max_rel_err(host(a), host(b)) <= 1e-4


@pytest.mark.parametrize("B,D,L", [(1, 8, 1), (3, 96, 49), (2, 97, 64), (40, 96, 784), (2, 300, 33), (1, 1000, 130)])
@pytest.mark.parametrize("dt", ["f32", "bf16"])
def test_layer_norm_backward(B, D, L, dt):
    from vmamba_b200 import _lib
    y, w = torch.randn(B, D, L, device="cuda"), torch.randn(D, device="cuda")
    g = torch.randn(B, D, L, device="cuda").to(TD[dt])
    dy, dw, db = torch.empty_like(y), torch.empty_like(w), torch.empty_like(w)
    p = _lib.NormBwdParams(y.data_ptr(), g.data_ptr(), w.data_ptr(), dy.data_ptr(), dw.data_ptr(), db.data_ptr(), B, D, L,
                           {"f32": _lib.SS2D_F32, "bf16": _lib.SS2D_BF16}[dt], 1e-5)
    ws = torch.empty(_lib.lib().ss2d_layer_norm_cf_bwd_workspace_bytes(p), device="cuda", dtype=torch.uint8)
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    assert _lib.lib().ss2d_layer_norm_cf_bwd(p, torch.cuda.current_stream().cuda_stream) == _lib.SS2D_OK
    yd, wd, bd = (t.double().requires_grad_(True) for t in (y, w, torch.zeros_like(w)))
    z = torch.nn.functional.layer_norm(yd.transpose(1, 2), (D,), wd, bd, 1e-5).transpose(1, 2)
    for got, want in zip((dy, dw, db), torch.autograd.grad(z, (yd, wd, bd), g.double())):
        scale = want.abs().max().item()
        assert (got.double() - want).abs().max().item() <= 1e-4 * max(scale, 1e-3)


@pytest.mark.parametrize("M,K,N", [(8, 32, 8), (32, 96, 64), (104, 384, 200), (200, 384, 2160), (40, 768, 72), (56, 192, 9472)])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
def test_linear_few_pixels(M, K, N, dt):
    from vmamba_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = (torch.randn(s, device="cuda", generator=g).to(TD[dt]) for s in ((K, N), (M, K)))
    b = torch.randn(M, device="cuda", generator=g)
    assert ops.linear_supported(M, K, N, TD[dt])
    want = w.double() @ x.double() + b.double()[:, None]
    got = ops.linear_cf(x, w, bias=b)
    assert O.max_rel_err(host(got), want.float().cpu().numpy()) <= TOL_BF16


@pytest.mark.parametrize("M,K,N", [(8, 32, 8), (40, 64, 72), (1536, 384, 200), (768, 192, 784), (96, 768, 56)])
@pytest.mark.parametrize("dt", ["bf16", "f16"])
def test_linear_few_pixels_gelu(M, K, N, dt):
    """Projection, bias and GELU in one launch: tiles of 32 rows and 64 pixels, whole and ragged."""
    from vmamba_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w, x = (torch.randn(s, device="cuda", generator=g).mul_(k).to(TD[dt]) for s, k in (((M, K), K ** -0.5), ((K, N), 1.0)))
    bias, out = torch.randn(M, device="cuda", generator=g), torch.empty(M, N, device="cuda", dtype=TD[dt])
    p = _lib.LinearParams(x.data_ptr(), w.data_ptr(), bias.data_ptr(), out.data_ptr(), M, K, N, 0, 0, {"bf16": _lib.SS2D_BF16, "f16": _lib.SS2D_F16}[dt], 1)
    assert _lib.lib().ss2d_linear_fwd(p, torch.cuda.current_stream().cuda_stream) == _lib.SS2D_OK
    ref = torch.nn.functional.gelu(w.double() @ x.double() + bias.double()[:, None])
    assert (out.double() - ref).abs().max() <= (2e-2 if dt == "bf16" else 3e-3)


@pytest.mark.parametrize("at", [(0, 0, 0, 0), (1, 3, 5, 7), (6, 2, 1, 4)])
@pytest.mark.parametrize("N,K,Cd,L,dt", [(1, 3, 3, 5, "bf16"), (1, 1, 1, 1, "f32"), (1, 3, 5, 49, "f16"), (1, 1, 3, 131, "f32"), (1, 3, 7, 1001, "bf16"),
                                         (1, 1, 9, 4099, "bf16"), (1, 3, 1100, 33, "f32"), (2, 3, 5, 67, "f32"), (4, 1, 33, 131, "bf16"), (16, 3, 3, 35, "f16")])
def test_scan_tensors_off_16_byte_boundaries(vb, N, K, Cd, L, dt, at):
    """Tensors that do not start or end on 16-byte boundaries, of odd row lengths and counts, in the middle of NaN: forward, states and
    gradients."""
    u, delta, A, B, C, D, bias, dout = _random_case(1, K, Cd, N, L, seed=L + N)
    td = TD[dt]

    def put(a, offset, type=td):
        flat = torch.full((a.size + 32,), float("nan"), device="cuda", dtype=type)
        view = flat[8 + offset:8 + offset + a.size].view(a.shape)
        view.copy_(dev(a, type))
        return view
    if dt != "f32":
        u, delta, B, C = (O._round_to(a, dt) for a in (u, delta, B, C))
    ts = [put(a, o) for a, o in zip((u, delta, B, C), at)]
    y, states = vb.selective_scan_fwd(ts[0], ts[1], dev(A), ts[2], ts[3], dev(D), dev(bias), True, True, return_checkpoints="grad")
    assert O.max_rel_err(host(y), CO.selective_scan(u, delta, A, B, C, D, bias, True)) <= TOL_F32
    ref = O.selective_scan_bwd(u, delta, A, B, C, D, bias, dout, True, dt)
    for ck in (states, None):
        got = vb.selective_scan_bwd(ts[0], ts[1], dev(A), ts[2], ts[3], dev(D), dev(bias), put(dout, at[0], torch.float32), True, ck)
        for name, x, r in zip(NAMES, got, ref):
            assert O.max_rel_err(host(x), r) <= TOL[dt], name


@pytest.mark.parametrize("dt", ["f32", "bf16"])
@pytest.mark.parametrize("scans", [0, 1, 2, 3])
@pytest.mark.parametrize("shape,offset", [((1, 1, 1, 1), 0), ((2, 3, 1, 9), 1), ((2, 3, 9, 1), 0), ((3, 50, 7, 7), 3), ((2, 37, 5, 6), 2), ((5, 61, 16, 32), 0),
                                          ((1, 3, 64, 32), 4), ((1, 3, 56, 58), 1), ((1, 2, 96, 96), 0), ((1, 2, 109, 113), 1), ((1, 2, 192, 192), 0),
                                          ((1, 2, 33, 161), 1), ((1, 2, 200, 190), 0), ((1, 1, 2, 9001), 0), ((1, 1, 20000, 3), 1), ((2, 2, 247, 231), 5)])
def test_cross_of_any_plane_and_alignment(vb, shape, offset, scans, dt):
    """CrossScan and CrossMerge at the edges of their kernels: single pixels and lines, planes that share a CTA, lines in one bank, pairs, the
    largest planes taken whole and the smallest in tiles, tensors that start anywhere.  The merge is rounded after every addition."""
    Bt, Cc, H, W = shape
    rng, td = np.random.default_rng(H * W + scans), TD[dt]

    def at_offset(a):
        room = torch.full((a.size + offset,), float("nan"), device="cuda", dtype=td)
        room[offset:] = dev(a.reshape(-1), td)
        return room[offset:].view(a.shape)
    rnd = (lambda a: a) if dt == "f32" else O.round_bf16
    x, ys = rnd(rng.standard_normal(shape, dtype=np.float32)), rnd(rng.standard_normal((Bt, 4, Cc, H, W), dtype=np.float32))
    assert np.array_equal(host(vb.cross_scan_fn(at_offset(x), scans=scans)), O.cross_scan(x, scans).reshape(Bt, 4, Cc, H * W))
    place = O.cross_scan(np.arange(H * W, dtype=np.float32).reshape(1, 1, H, W), scans).reshape(4, H * W).astype(np.int64)
    y = [torch.empty(Bt, Cc, H * W, dtype=td) for _ in range(4)]
    for k in range(4):
        y[k][..., torch.from_numpy(place[k])] = torch.from_numpy(ys[:, k].reshape(Bt, Cc, H * W)).to(td)
    if scans == 1:
        want = (((y[0].float() + y[1].float()) + y[2].float()) + y[3].float()).to(td)
    else:
        want = ((y[0] + y[1]) + y[2]) + y[3] if scans == 3 else (y[0] + y[2]) + (y[1] + y[3])
    assert torch.equal(vb.cross_merge_fn(at_offset(ys), scans=scans).cpu().view(Bt, Cc, H * W), want)


def test_cross_of_single_pixels_of_very_many_images(vb):
    """The number of a route, four times the image's, is beyond 32 bits."""
    n = (1 << 29) + 3
    x = torch.arange(n, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16).view(n, 1, 1, 1)
    ys = vb.cross_scan_fn(x)
    assert ys.shape == (n, 4, 1, 1) and all(torch.equal(ys[:, k, 0, 0].view(torch.int16), x.view(-1).view(torch.int16)) for k in range(4))
    ys = torch.ones(n, 4, 1, 1, 1, device="cuda", dtype=torch.bfloat16)
    del x
    ys[-2:] = 2
    y = vb.cross_merge_fn(ys)
    assert bool((y[:-2] == 4).all()) and bool((y[-2:] == 8).all())
