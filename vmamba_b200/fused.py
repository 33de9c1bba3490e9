"""Fused SS2D core: host side of `ss2d_core_fwd` and the hook that installs it into SS2D modules.

`ss2d_core(x, weights)` computes what SS2Dv2.forward_corev2 computes for scan mode "cross2d" on a
channel-first map (vmamba.py:1504-1571): CrossScan -> x_proj -> dt_projs -> selective scan ->
CrossMerge -> out_norm -> cast, without ever materialising the (B, 4, D, L) scan copy or the
per-route outputs.

Because a 1x1 projection commutes with a permutation of the pixels, the x_proj contraction is done
once on x in its native layout ((4(R+2N) x D) . (D x L) per image); the rows of
the two column-major routes are then transposed (they are (R+2N)/D of the size of x), the step
sizes are expanded per route (R -> D, `ss2d_route_expand`) and the CUDA kernel consumes x plus
the per-route (delta, B, C) streams in the orientation order of each route.
"""
from __future__ import annotations

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

    _native = None              # no field: what `native` made of the fields above

    def __getstate__(self):     # copies and pickles hold the tensors; a copy makes its own `native`
        return {**self.__dict__, "_native": None}

    def __setattr__(self, name, value):
        super().__setattr__(name, value)
        if name != "_native":
            super().__setattr__("_native", None)

    @property
    def native(self):
        """The same weights as the host extension holds them."""
        if self._native is None:
            self._native = _host.CoreWeights(self.wx, self.wdt, self.A, self.Ds, self.dt_bias, self.ln_weight, self.ln_bias,
                                             self.d_state, self.dt_rank, self.eps)
        return self._native

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
    bc, delta = _host.project(x.contiguous(), w.native, channel_major)
    if channel_major:       # (pair, rows, B, L) per orientation
        D, B, H, W = x.shape
        delta, bc = delta.view(2, 2, D, B, H * W), bc.view(2, 2, 2 * w.d_state, B, H * W)
    return RouteStreams(bc[0], bc[1], delta[0], delta[1], channel_major)


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
    return _host.core_takes(list(x_shape), int(d_state), dtype, channel_major)


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
    return _host.ss2d_core(x, w.native, with_norm, out_dtype, workspace, channel_major)


def _ss2d_core_unfused(x, w: CoreWeights, with_norm: bool, out_dtype):
    """Same mathematics through the operator-surface kernels (cross scan -> projections ->
    selective scan -> cross merge -> LayerNorm), the order of vmamba.py:1536-1571."""
    return _host.ss2d_core_by_operators(x.contiguous(), w.native, with_norm, out_dtype, False)


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
