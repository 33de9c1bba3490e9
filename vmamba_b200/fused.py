"""Fused SS2D core: host side of `ss2d_core_fwd` and the hook that installs it into SS2D modules.

`ss2d_core(x, weights)` computes what SS2Dv2.forward_corev2 computes for scan mode "cross2d" on a
channel-first map (vmamba.py:1504-1571): CrossScan -> x_proj -> dt_projs -> selective scan ->
CrossMerge -> out_norm -> cast, without ever materialising the (B, 4, D, L) scan copy or the
per-route outputs.

Because a 1x1 projection commutes with a permutation of the pixels, the x_proj contraction is done
once on x in its native layout (one library GEMM, (4(R+2N) x D) . (D x L) per image); the rows of
the two column-major routes are then transposed (they are (R+2N)/D of the size of x), the step
sizes are expanded per route (R -> D, a batched library GEMM) and the CUDA kernel consumes x plus
the per-route (delta, B, C) streams in the orientation order of each route.
"""
from __future__ import annotations

import ctypes
import math
from dataclasses import dataclass
from typing import Optional

import torch

from . import _host, _lib, ops
from ._lib import CoreParams, check, lib

K = 4


@dataclass
class CoreWeights:
    """Inference-time constants of one SS2D core, laid out for the fused path."""
    wx: torch.Tensor            # (K*(R+2N), D) activation dtype
    wdt: torch.Tensor           # (K, D, R) activation dtype
    A: torch.Tensor             # (K*D, N) fp32, = -exp(A_logs)
    Ds: torch.Tensor            # (K*D,) fp32
    dt_bias: torch.Tensor       # (K*D,) fp32
    ln_weight: Optional[torch.Tensor]
    ln_bias: Optional[torch.Tensor]
    d_state: int
    dt_rank: int
    d_inner: int
    eps: float = 1e-5

    @staticmethod
    def build(x_proj_weight, dt_projs_weight, dt_projs_bias, A_logs, Ds, ln_weight, ln_bias, *,
              d_state: int, dt_rank: int, dtype: torch.dtype, eps: float = 1e-5) -> "CoreWeights":
        N, R = int(d_state), int(dt_rank)
        KD = A_logs.shape[0]
        D = KD // K
        wx = x_proj_weight.detach().reshape(K * (R + 2 * N), D).to(dtype).contiguous()
        wdt = dt_projs_weight.detach().reshape(K, D, R).to(dtype).contiguous()
        f32 = lambda t: None if t is None else t.detach().float().contiguous()
        return CoreWeights(wx, wdt,
                           (-torch.exp(A_logs.detach().float())).reshape(KD, N).contiguous(),
                           f32(Ds.reshape(-1)), f32(dt_projs_bias.reshape(-1)), f32(ln_weight), f32(ln_bias),
                           N, R, D, float(eps))


def project(x: torch.Tensor, w: CoreWeights, channel_major: bool = False):
    """x (B, D, H, W), or (D, B, H, W) with `channel_major` -> per-orientation projections.

    Returns (bc_even, bc_odd, delta_even, delta_odd):
      bc_even  (B, 2, 2N, L): B then C rows of routes 0 and 2, row-major pixel order
      bc_odd   (B, 2, 2N, L): routes 1 and 3, column-major pixel order
      delta_*  (B, 2, D, L) raw step sizes in the same orders
    all in the activation dtype (the dtype the projection produced them in, as in the reference under
    autocast).  One library GEMM (x_proj on the un-scanned map) and one `ss2d_route_expand` launch.
    """
    if channel_major:
        D, B, H, W = x.shape
    else:
        B, D, H, W = x.shape
    L, R, N = H * W, w.dt_rank, w.d_state
    C = R + 2 * N
    p = _lib.ExpandParams()
    if channel_major:
        # one GEMM over the whole batch: (4C x D) . (D x B*L) -> rows (route, c), columns (b, l); the route
        # streams keep that shape: delta (orientation, pair, D, B, L), B/C rows (orientation, pair, 2N, B, L)
        if ops.linear_supported(K * C, D, B * L, x.dtype):
            xd = ops.linear_cf(x.reshape(D, B * L), w.wx)             # x_proj on the tensor cores (ss2d_linear_fwd)
        else:
            xd = torch.matmul(w.wx, x.reshape(D, B * L))              # fp32 maps, odd widths: the library GEMM
        p.x_dbl_batch_stride, p.x_dbl_route_stride, p.x_dbl_row_stride = L, C * B * L, B * L
        delta = torch.empty((2, 2, D, B, L), device=x.device, dtype=x.dtype)
        bc = torch.empty((2, 2, 2 * N, B, L), device=x.device, dtype=x.dtype)
        for k in range(K):
            j, i = k % 2, k // 2
            p.delta[k], p.delta_batch_stride[k], p.delta_channel_stride[k] = delta[j, i].data_ptr(), L, B * L
            p.bc[k], p.bc_batch_stride[k], p.bc_row_stride[k] = bc[j, i].data_ptr(), L, B * L
    else:
        xd = torch.matmul(w.wx, x.reshape(B, D, L))                   # (B, 4*C, L), route-major rows
        p.x_dbl_batch_stride, p.x_dbl_route_stride, p.x_dbl_row_stride = xd.stride(0), C * L, L
        delta = torch.empty((2, B, 2, D, L), device=x.device, dtype=x.dtype)   # [orientation][b][pair index]
        bc = torch.empty((2, B, 2, 2 * N, L), device=x.device, dtype=x.dtype)
        for k in range(K):
            j, i = k % 2, k // 2
            p.delta[k], p.delta_batch_stride[k] = delta[j, :, i].data_ptr(), delta.stride(1)
            p.bc[k], p.bc_batch_stride[k] = bc[j, :, i].data_ptr(), bc.stride(1)
    p.x_dbl, p.dt_weight = xd.data_ptr(), w.wdt.data_ptr()
    p.B, p.D, p.R, p.N, p.H, p.W = B, D, R, N, H, W
    p.act_dtype = ops.dtype_code(x)
    need = int(lib().ss2d_route_expand_workspace_bytes(p))      # room for the transposed rows of the column-major routes
    if need > 0:
        ws = torch.empty(need, device=x.device, dtype=torch.uint8)
        p.workspace, p.workspace_bytes = ws.data_ptr(), need
    with torch.cuda.device(x.device):
        check(lib().ss2d_route_expand(p, torch.cuda.current_stream(x.device).cuda_stream), "ss2d_route_expand")
    if channel_major:       # (pair, rows, B, L) per orientation
        return RouteStreams(bc[0], bc[1], delta[0], delta[1], True)
    return RouteStreams(bc[0], bc[1], delta[0], delta[1], False)


class RouteStreams(tuple):
    """(bc_even, bc_odd, delta_even, delta_odd) plus the layout flag of the four tensors:
    batch-major (B, pair, rows, L) or channel-major (pair, rows, B, L)."""
    def __new__(cls, bc_even, bc_odd, delta_even, delta_odd, channel_major=False):
        self = super().__new__(cls, (bc_even, bc_odd, delta_even, delta_odd))
        self.channel_major = channel_major
        return self


def scan_merge_norm(x: torch.Tensor, proj, w: CoreWeights, *, with_norm: bool = True, out_dtype=None,
                    workspace: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
                    channel_major: bool = False) -> torch.Tensor:
    """The CUDA part of the fused core (`ss2d_core_fwd`): x plus the projections returned by
    `project` -> merged (and normalised) map.  Launches one scan+merge kernel and, with
    `with_norm`, one LayerNorm kernel; allocates the output and the fp32 workspace unless given."""
    bc_even, bc_odd, delta_even, delta_odd = proj
    if channel_major:
        D, B, H, W = x.shape
    else:
        B, D, H, W = x.shape
    R, N = w.dt_rank, w.d_state
    out_dtype = out_dtype or (x.dtype if with_norm else torch.float32)
    y = out if out is not None else torch.empty(x.shape, device=x.device, dtype=out_dtype)
    p = CoreParams()
    p.x = x.data_ptr()
    srcs = (bc_even, bc_odd)
    deltas = (delta_even, delta_odd)
    esz = x.element_size()
    streams_cm = getattr(proj, "channel_major", False)
    for k in range(K):
        j, i = k % 2, k // 2          # j: orientation (0 row, 1 column); i: index inside the pair
        bc, dl = srcs[j], deltas[j]
        if streams_cm:                # delta (pair, D, B, L), B/C rows (pair, 2N, B, L)
            p.delta[k] = dl[i].data_ptr()
            p.delta_batch_stride[k], p.delta_channel_stride[k] = dl.stride(2), dl.stride(1)
            p.Bm[k] = bc[i].data_ptr()
            p.Cm[k] = bc[i, N].data_ptr()
            p.bc_batch_stride[k] = bc.stride(2)
        else:                         # delta (B, pair, D, L), B/C rows (B, pair, 2N, L)
            p.delta[k] = dl.data_ptr() + i * dl.stride(1) * esz
            p.delta_batch_stride[k], p.delta_channel_stride[k] = dl.stride(0), dl.stride(2)
            base = bc.data_ptr() + i * bc.stride(1) * esz
            p.Bm[k] = base
            p.Cm[k] = base + N * bc.stride(2) * esz
            p.bc_batch_stride[k] = bc.stride(0)
    p.A, p.Dskip, p.delta_bias = w.A.data_ptr(), w.Ds.data_ptr(), w.dt_bias.data_ptr()
    p.ln_weight = None if w.ln_weight is None else w.ln_weight.data_ptr()
    p.ln_bias = None if w.ln_bias is None else w.ln_bias.data_ptr()
    p.y = y.data_ptr()
    p.B, p.D, p.H, p.W, p.N = B, D, H, W, N
    p.act_dtype, p.y_dtype = ops.dtype_code(x), ops.dtype_code(y)
    p.with_norm, p.ln_eps = int(with_norm), w.eps
    if channel_major:
        p.x_batch_stride, p.x_channel_stride = H * W, B * H * W
        p.y_batch_stride, p.y_channel_stride = H * W, B * H * W
    need = int(lib().ss2d_core_workspace_bytes(p))
    if need < 0:
        raise RuntimeError("ss2d_core_workspace_bytes: invalid arguments")
    if need > 0:
        if workspace is None or workspace.numel() * workspace.element_size() < need:
            workspace = torch.empty(need, device=x.device, dtype=torch.uint8)
        p.workspace, p.workspace_bytes = workspace.data_ptr(), workspace.numel() * workspace.element_size()
    with torch.cuda.device(x.device):
        check(lib().ss2d_core_fwd(p, torch.cuda.current_stream(x.device).cuda_stream), "ss2d_core_fwd")
    return y


def fused_supported(x_shape, d_state: int, dtype: torch.dtype = torch.bfloat16, channel_major: bool = False) -> bool:
    """True when `ss2d_core_fwd` takes the case itself.  Asks the library (`ss2d_core_supported`), which applies
    the rules of its launch planner to dense, 16-byte aligned streams of this shape, so the answer cannot drift
    from what the call will do."""
    if channel_major:
        D, B, H, W = x_shape
    else:
        B, D, H, W = x_shape
    L = H * W
    p = CoreParams()
    fake = 4096                                   # an aligned address; the query dereferences nothing
    p.x = p.A = p.Dskip = p.delta_bias = p.y = fake
    for k in range(K):
        p.delta[k] = p.Bm[k] = p.Cm[k] = fake
        if channel_major:
            p.delta_batch_stride[k], p.delta_channel_stride[k], p.bc_batch_stride[k] = L, B * L, L
        else:
            p.delta_batch_stride[k], p.delta_channel_stride[k], p.bc_batch_stride[k] = 2 * D * L, L, 4 * int(d_state) * L
    p.B, p.D, p.H, p.W, p.N = B, D, H, W, int(d_state)
    code = {torch.float32: _lib.SS2D_F32, torch.float16: _lib.SS2D_F16, torch.bfloat16: _lib.SS2D_BF16}[dtype]
    p.act_dtype = p.y_dtype = code
    p.with_norm = 1
    if channel_major:
        p.x_batch_stride = p.y_batch_stride = L
        p.x_channel_stride = p.y_channel_stride = B * L
    return int(lib().ss2d_core_supported(p)) == _lib.SS2D_OK


def ss2d_core(x: torch.Tensor, w: CoreWeights, *, with_norm: bool = True, out_dtype=None,
              workspace: Optional[torch.Tensor] = None, channel_major: bool = False) -> torch.Tensor:
    """Fused forward of the SS2D core.  x: (B, D, H, W) CUDA tensor, or (D, B, H, W) with
    `channel_major`; returns a map of the same layout in `out_dtype` (default x.dtype; fp32
    required when `with_norm` is False).  Falls back to the operator-surface kernels (still CUDA,
    never CPU) for d_state > 1 or planes too long for one CTA."""
    if not x.is_cuda:
        raise RuntimeError("vmamba_b200.ss2d_core runs on CUDA tensors only (no CPU fallback)")
    x = x.contiguous()
    if x.shape[0 if channel_major else 1] != w.d_inner:
        raise RuntimeError(f"x has {x.shape[0 if channel_major else 1]} channels, weights were built for {w.d_inner}")
    out_dtype = out_dtype or (x.dtype if with_norm else torch.float32)
    with torch.autocast("cuda", enabled=False):
        def unfused():
            if channel_major:
                return _ss2d_core_unfused_cm(x, w, with_norm, out_dtype)
            return _ss2d_core_unfused(x, w, with_norm, out_dtype)

        if not fused_supported(x.shape, w.d_state, x.dtype, channel_major) or (channel_major and not with_norm):
            return unfused()
        try:
            return scan_merge_norm(x, project(x, w, channel_major), w, with_norm=with_norm, out_dtype=out_dtype,
                                   workspace=workspace, channel_major=channel_major)
        except _lib.Ss2dError as e:        # refused before any launch (an alignment the query could not see)
            if e.status != _lib.SS2D_ENOTSUP:
                raise
            return unfused()


def _ss2d_core_unfused(x, w: CoreWeights, with_norm: bool, out_dtype, out_channel_major: bool = False):
    """Same mathematics through the operator-surface kernels (cross scan -> projections ->
    selective scan -> cross merge -> LayerNorm), the order of vmamba.py:1536-1571."""
    B, D, H, W = x.shape
    L, R, N = H * W, w.dt_rank, w.d_state
    C = R + 2 * N
    xs = ops.cross_scan_fwd(x, 0)                                        # (B, K, D, L)
    x_dbl = torch.matmul(w.wx.view(K, C, D), xs)                         # (B, K, C, L)
    dts = torch.matmul(w.wdt, x_dbl[:, :, :R]).reshape(B, K * D, L)
    Bs = x_dbl[:, :, R:R + N]                                            # strided views: the scan takes batch / group / state strides
    Cs = x_dbl[:, :, R + N:]
    ys = ops.selective_scan_fwd(xs.view(B, K * D, L), dts, w.A, Bs, Cs, w.Ds, w.dt_bias, True, True)
    y = ops.cross_merge_fwd(ys.view(B, K, D, H, W), 0).view(B, D, H, W)
    if with_norm:
        return ops.layer_norm_cf(y, w.ln_weight, w.ln_bias, w.eps, out_dtype, out_channel_major=out_channel_major)
    return y.to(out_dtype)


def _ss2d_core_unfused_cm(x, w: CoreWeights, with_norm: bool, out_dtype):
    """The same chain on a channel-major map (D, B, H, W) without a layout copy: the batch is folded into the
    plane count of CrossScan / CrossMerge (their routes stay per plane), each projection is one GEMM per route
    over all images, and the selective scan reads and writes (route, channel, image) rows through its strides."""
    D, B, H, W = x.shape
    L, R, N = H * W, w.dt_rank, w.d_state
    C = R + 2 * N
    xs = ops.cross_scan_fwd(x.view(1, D * B, H, W), 0).view(K, D, B * L)         # route k: (D, B, L)
    x_dbl = torch.bmm(w.wx.view(K, C, D), xs)                                    # (K, C, B*L)
    dts = torch.bmm(w.wdt, x_dbl[:, :R])                                         # (K, D, B*L)
    rows = lambda t: t.view(K * D, B, L).permute(1, 0, 2)                        # (B, K*D, L) view of (K, D, B, L)
    bc = x_dbl.view(K, C, B, L).permute(2, 0, 1, 3)                              # (B, K, C, L) view
    ys = torch.empty((K * D, B, L), device=x.device, dtype=torch.float32)
    ops.selective_scan_fwd(rows(xs), rows(dts), w.A, bc[:, :, R:R + N], bc[:, :, R + N:], w.Ds, w.dt_bias, True, True,
                           out=ys.permute(1, 0, 2))
    y = ops.cross_merge_fwd(ys.view(1, K, D * B, H, W), 0).view(D, B, H, W)
    if with_norm:
        return ops.layer_norm_cf(y, w.ln_weight, w.ln_bias, w.eps, out_dtype, channel_major=True)
    return y.to(out_dtype)


def ss2d_core_autograd(x, x_proj_weight, dt_projs_weight, dt_projs_bias, A_logs, Ds, ln_weight, ln_bias, *,
                       d_state: int, dt_rank: int, eps: float = 1e-5, oflex: bool = True):
    """Differentiable SS2D core for training: the statements of SS2Dv2.forward_corev2
    (vmamba.py:1536-1571) with this package's autograd Functions for CrossScan, the selective scan and
    CrossMerge, and torch for the projections and the LayerNorm.  Gradients flow to x and to every
    parameter; this is what a reference module computes after `vmamba_b200.install()`.
    x: (B, D, H, W); x_proj_weight: (K*(R+2N), D) or (K, R+2N, D); dt_projs_weight: (K*D, R) or (K, D, R)."""
    params = (x_proj_weight, dt_projs_weight, dt_projs_bias, A_logs, Ds, ln_weight, ln_bias)
    if oflex and x.is_cuda and x.dtype in ops._DTYPES and not torch.is_autocast_enabled("cuda") \
            and all(t is not None and t.is_cuda for t in params) and int(d_state) <= 16 and int(dt_rank) <= 1024:
        return _host.ss2d_core_autograd(x, *params, int(d_state), int(dt_rank), float(eps))     # the same statements as one node
    B, D, H, W = x.shape
    L, N, R = H * W, int(d_state), int(dt_rank)
    xs = ops.cross_scan_fn(x, True, True, False, 0)                                     # (B, K, D, L)
    wx = x_proj_weight.reshape(K, R + 2 * N, D).to(x.dtype)
    x_dbl = torch.einsum("bkdl,kcd->bkcl", xs.view(B, K, D, L), wx)
    dts, Bs, Cs = torch.split(x_dbl, [R, N, N], dim=2)
    wdt = dt_projs_weight.reshape(K, D, R).to(x.dtype)
    dts = torch.einsum("bkrl,kdr->bkdl", dts, wdt).reshape(B, K * D, L)
    As = -torch.exp(A_logs.float())
    ys = ops.selective_scan_fn(xs.reshape(B, K * D, L), dts.contiguous(), As, Bs.contiguous(), Cs.contiguous(),
                               Ds.float(), dt_projs_bias.reshape(-1).float(), True, oflex)
    y = ops.cross_merge_fn(ys.view(B, K, D, H, W), True, True, False, 0).view(B, D, H, W)
    y = torch.nn.functional.layer_norm(y.permute(0, 2, 3, 1), (D,), ln_weight, ln_bias, eps).permute(0, 3, 1, 2)
    return y.to(x.dtype)


# --------------------------------------------------------------------------------------------
# installing the fused core into reference SS2D modules without touching their source
# --------------------------------------------------------------------------------------------
def _supported(m) -> bool:
    fc = getattr(m, "forward_core", None)
    kw = getattr(fc, "keywords", None)
    if fc is None or kw is None:
        return False
    if kw.get("scan_mode", "cross2d") not in ("cross2d", 0):
        return False
    if kw.get("force_fp32", False):
        return False
    if not getattr(m, "channel_first", False):
        return False
    if not isinstance(getattr(m, "out_norm", None), torch.nn.LayerNorm):
        return False
    return all(hasattr(m, n) for n in ("x_proj", "dt_projs", "A_logs", "Ds", "dt_projs_bias"))


def enable_fused(model: torch.nn.Module, verbose: bool = False) -> int:
    """Rebind `forward_core` (an instance attribute set in SS2Dv2.__initv2__, vmamba.py:1448) of
    every supported SS2D module to the fused path.  Weights are snapshotted per activation dtype at
    first use, so call it on a model in eval mode; `disable_fused` restores the original."""
    n = 0
    for mod in model.modules():
        if not _supported(mod):
            continue
        cache = {}
        orig = mod.forward_core

        def fused_core(x, _m=mod, _cache=cache, _orig=orig, **kwargs):
            if getattr(_m, "__DEBUG__", False) or _m.training or not x.is_cuda:
                return _orig(x, **kwargs)
            # the fused call builds no autograd graph: whenever a gradient could be asked for through this
            # module (input gradients in eval mode, un-frozen parameters), the differentiable original runs
            if torch.is_grad_enabled() and (x.requires_grad or any(q.requires_grad for q in _m.parameters())):
                return _orig(x, **kwargs)
            w = _cache.get(x.dtype)
            if w is None:
                w = CoreWeights.build(_m.x_proj.weight, _m.dt_projs.weight, _m.dt_projs_bias, _m.A_logs, _m.Ds,
                                      _m.out_norm.weight, _m.out_norm.bias, d_state=_m.d_state,
                                      dt_rank=_m.dt_rank, dtype=x.dtype, eps=_m.out_norm.eps)
                _cache[x.dtype] = w
            return ss2d_core(x, w)

        fused_core._vmamba_b200_original = orig
        mod.forward_core = fused_core
        n += 1
    if verbose:
        print(f"vmamba_b200: fused SS2D core enabled on {n} modules")
    return n


def disable_fused(model: torch.nn.Module) -> int:
    n = 0
    for mod in model.modules():
        fc = getattr(mod, "forward_core", None)
        orig = getattr(fc, "_vmamba_b200_original", None)
        if orig is not None:
            mod.forward_core = orig
            n += 1
    return n
