"""What the state of the calling program must not change: autocast regions, copies of a model, what a training step keeps.
Needs a GPU."""
import copy
import math

import pytest
import torch
import torch.utils.checkpoint

from vmamba_b200.backbone import AcceleratedVSSM

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vb():
    import vmamba_b200
    return vmamba_b200


def state_dict(dims=(32, 64, 128, 256), depths=(1, 1, 1, 1), classes=10, seed=0):
    """Random weights of a small backbone with a classifier and the feature norms, in the key layout of its checkpoints."""
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g) * math.prod(s[1:]) ** -0.5      # noqa: E731
    sd = {}

    def norm(name, n):
        sd[name + ".weight"], sd[name + ".bias"] = torch.ones(n), torch.zeros(n)

    def conv(name, out, inn):
        sd[name + ".weight"], sd[name + ".bias"] = rnd(out, inn, 3, 3), torch.zeros(out)

    conv("patch_embed.0", dims[0] // 2, 3)
    norm("patch_embed.2", dims[0] // 2)
    conv("patch_embed.5", dims[0], dims[0] // 2)
    norm("patch_embed.7", dims[0])
    for i, d in enumerate(dims):
        R = math.ceil(d / 16)
        for j in range(depths[i]):
            p = f"layers.{i}.blocks.{j}."
            norm(p + "norm", d)
            norm(p + "norm2", d)
            norm(p + "op.out_norm", d)
            for name, shape in (("op.in_proj", (d, d)), ("op.out_proj", (d, d)), ("mlp.fc1", (4 * d, d)), ("mlp.fc2", (d, 4 * d)),
                                ("op.conv2d", (d, 1, 3, 3)), ("op.x_proj", (4 * (R + 2), d)), ("op.dt_projs", (4 * d, R))):
                sd[p + name + ".weight"] = rnd(*shape)
            sd[p + "mlp.fc1.bias"], sd[p + "mlp.fc2.bias"] = torch.zeros(4 * d), torch.zeros(d)
            sd[p + "op.dt_projs_bias"], sd[p + "op.A_logs"], sd[p + "op.Ds"] = torch.full((4, d), -3.0), torch.zeros(4 * d, 1), torch.ones(4 * d)
        norm(f"outnorm{i}", d)
        if i + 1 < len(dims):
            conv(f"layers.{i}.downsample.1", dims[i + 1], d)
            norm(f"layers.{i}.downsample.3", dims[i + 1])
    norm("classifier.norm", dims[-1])
    sd["classifier.head.weight"], sd["classifier.head.bias"] = rnd(classes, dims[-1]), torch.zeros(classes)
    return sd


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("region", [torch.float16, torch.bfloat16])
def test_backbone_under_autocast(vb, dtype, region):
    """A model computes in its own type, inside an autocast region as outside: same bits."""
    m = vb.VSSMInfer.from_state_dict(state_dict(), dtype=dtype)
    x = torch.randn(2, 3, 64, 96, device="cuda").to(dtype)
    want, maps = m(x), m.features(x)
    with torch.autocast("cuda", dtype=region):
        got, inside = m(x), m.features(x)
    assert got.dtype == want.dtype and torch.equal(got, want)
    for a, b in zip(inside, maps):
        assert a.dtype == b.dtype and torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_core_under_autocast(vb, dtype):
    """The core, its projections and the gradients of a step whose backward pass alone lies in the region."""
    from vmamba_b200 import fused
    D, R = 32, 2
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)      # noqa: E731
    par = [rnd(4 * (R + 2), D) * D ** -0.5, rnd(4 * D, R) * R ** -0.5, torch.full((4, D), -3.0, device="cuda"), torch.zeros(4 * D, 1, device="cuda"),
           torch.ones(4 * D, device="cuda"), torch.ones(D, device="cuda"), torch.zeros(D, device="cuda")]
    x, gy = rnd(2, D, 9, 10).to(dtype), rnd(2, D, 9, 10).to(dtype)
    w = vb.CoreWeights.build(*par, d_state=1, dt_rank=R, dtype=dtype)
    leaves = [t.requires_grad_(True) for t in [x, *par]]

    def step(region):
        with torch.no_grad(), torch.autocast("cuda", enabled=region):
            outs = [vb.ss2d_core(x, w), *fused.project(x, w)]
        y = vb.ss2d_core_autograd(*leaves, d_state=1, dt_rank=R)
        with torch.autocast("cuda", enabled=region):
            return [*outs, y, *torch.autograd.grad(y, leaves, gy)]
    for a, b in zip(step(False), step(True)):
        assert a.dtype == b.dtype and torch.equal(a, b)


def test_parts_replaced_after_the_first_call(vb):
    """A model whose parts are replaced gives what one built with them gives, and a copy is a model of its own."""
    sd, x = state_dict(), torch.randn(2, 3, 64, 64, device="cuda").bfloat16()
    m = vb.VSSMInfer.from_state_dict(sd)
    first = m(x)
    twin = copy.deepcopy(m)
    sd["classifier.head.bias"], sd["layers.2.blocks.0.op.Ds"] = torch.ones(10), sd["layers.2.blocks.0.op.Ds"] * 2
    other = vb.VSSMInfer.from_state_dict(sd)
    m.head["b"], m.blocks[2][0].core.Ds = other.head["b"], other.blocks[2][0].core.Ds
    assert torch.equal(m(x), other(x)) and not torch.equal(m(x), first)
    assert torch.equal(twin(x), first)
    w = vb.CoreWeights(*(getattr(m.blocks[0][0].core, k) for k in ("wx", "wdt", "A", "Ds", "dt_bias", "ln_weight", "ln_bias", "d_state", "dt_rank", "d_inner")))
    y = torch.randn(1, w.d_inner, 8, 8, device="cuda").bfloat16()
    one = vb.ss2d_core(y, w)
    w.ln_bias = w.ln_bias + 1
    assert ((vb.ss2d_core(y, w) - one).float() - 1).abs().max() < 0.05      # bf16: half a unit in the last place of values below 8


def _core_step(vb, dtype=torch.bfloat16):
    D, R = 64, 4
    g = torch.Generator(device="cuda").manual_seed(2)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)      # noqa: E731
    leaves = [rnd(2, D, 24, 24).to(dtype), rnd(4 * (R + 2), D) * D ** -0.5, rnd(4 * D, R) * R ** -0.5, torch.full((4, D), -3.0, device="cuda"),
              torch.zeros(4 * D, 1, device="cuda"), torch.ones(4 * D, device="cuda"), torch.ones(D, device="cuda"), torch.zeros(D, device="cuda")]
    return [t.requires_grad_(True) for t in leaves], lambda *t: vb.ss2d_core_autograd(*t, d_state=1, dt_rank=R)


def _scan_step(vb):
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)      # noqa: E731
    leaves = [rnd(2, 64, 600), rnd(2, 64, 600) - 3, -torch.ones(64, 1, device="cuda"), rnd(2, 4, 1, 600), rnd(2, 4, 1, 600)]
    return [t.requires_grad_(True) for t in leaves], vb.selective_scan_fn


# what a step keeps between its passes, in units of its largest input: the core four routes of x and of the step sizes, the states
# (four routes, fp32, one of eight elements) and the merged map (fp32); the scan u, delta and the states
@pytest.mark.parametrize("step,kept", [(_core_step, 4 + 4 + 1 + 2), (_scan_step, 2 + 1 / 8)])
def test_what_a_training_step_keeps(vb, step, kept):
    """Tensors kept for the backward pass go through saved-tensor hooks and are freed by it, though the result lives on."""
    leaves, fn = step(vb)
    size = leaves[0].numel() * leaves[0].element_size()
    seen = []

    def pack(t):
        seen.append(t.numel() * t.element_size())
        return t.cpu()
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        y = fn(*leaves)
    assert sum(seen) >= kept * size
    gy = torch.ones_like(y)
    from_host = torch.autograd.grad(y, leaves, gy)
    y = fn(*leaves)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    grads = torch.autograd.grad(y, leaves, gy)
    torch.cuda.synchronize()
    held = sum(t.numel() * t.element_size() for t in grads)
    own = 0 if step is _core_step else 2             # the scan keeps its caller's u and delta
    assert torch.cuda.memory_allocated() <= before + held - 0.9 * (kept - own) * size
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(y, leaves, gy)
    again = torch.autograd.grad(torch.utils.checkpoint.checkpoint(fn, *leaves, use_reentrant=False), leaves, gy)
    for a, b, c in zip(grads, from_host, again):
        assert torch.equal(a, b) and torch.equal(a, c)


def test_core_refuses_what_does_not_fit(vb):
    """Types and sizes that a library product or layer_norm refused are still refused where kernels take their place."""
    from vmamba_b200 import fused
    D, R = 32, 2
    par = [torch.randn(4 * (R + 2), D), torch.randn(4 * D, R), torch.zeros(4, D), torch.zeros(4 * D, 1), torch.ones(4 * D), torch.ones(D), torch.zeros(D)]
    par = [t.cuda() for t in par]
    w = vb.CoreWeights.build(*par, d_state=1, dt_rank=R, dtype=torch.bfloat16)
    for shape, cm in (((2, D, 8, 8), False), ((2, D, 7, 7), False), ((D, 2, 8, 8), True)):
        for other in (torch.float16, torch.float32):
            with pytest.raises(RuntimeError):
                vb.ss2d_core(torch.randn(shape, device="cuda", dtype=other), w, channel_major=cm)
            with pytest.raises(RuntimeError):
                fused.project(torch.randn(shape, device="cuda", dtype=other), w, cm)
    with pytest.raises(RuntimeError):
        fused.project(torch.randn(2, D + 8, 8, 8, device="cuda", dtype=torch.bfloat16), w)
    x = torch.randn(2, D, 8, 8, device="cuda")
    for i in (5, 6):                                     # the LayerNorm's weight and bias
        wrong = list(par)
        wrong[i] = wrong[i][:D // 2]
        with pytest.raises(RuntimeError):
            vb.ss2d_core_autograd(x, *wrong, d_state=1, dt_rank=R)


def test_a_captured_graph_keeps_its_weights(vb):
    """Parts replaced after the capture count in eager calls; the graph goes on with those it was captured with, which stay allocated."""
    m = vb.VSSMInfer.from_state_dict(state_dict())
    x = torch.randn(2, 3, 64, 64, device="cuda").bfloat16()
    for model in (m, AcceleratedVSSM(m, False, ())):
        runner = vb.GraphedBackbone(model, tuple(x.shape), dtype=torch.bfloat16)
        first = runner(x).clone()
        torch.cuda.synchronize()
        for stage in m.blocks:
            for b in stage:
                for name in ("w_in", "w_dw", "w_out", "w1", "w2"):
                    setattr(b, name, getattr(b, name) * 2)
        assert not torch.equal(m(x), first)              # the model's own object is made anew, and the old one let go
        junk = [torch.full_like(t, float("nan")) for stage in m.blocks for b in stage for t in (b.w_in, b.w_dw, b.w_out, b.w1, b.w2)]
        assert torch.equal(runner(x), first) and len(junk) == 20


def test_threads_with_planes_of_other_sizes(vb):
    """The limit of a kernel's shared memory belongs to all threads: calls on planes of 51 KB and of 71 KB of routes, which take the same kernel, in two
    threads at once."""
    import threading

    from vmamba_b200 import _lib
    done = {}

    def calls(H, W):
        stream = torch.cuda.Stream()
        ys = torch.randn(1, 4, 8, H, W, device="cuda")
        out = torch.empty(1, 8, H, W, device="cuda")
        torch.cuda.synchronize()
        p = _lib.CrossParams(in_=ys.data_ptr(), out=out.data_ptr(), dtype=_lib.SS2D_F32, scans=1, B=1, C=8, H=H, W=W)
        done[H, W] = {_lib.lib().ss2d_cross_merge(p, stream.cuda_stream) for _ in range(4000)}
        stream.synchronize()
        done[H, W].add(torch.equal(out, ((ys[:, 0] + ys[:, 1]) + ys[:, 2]) + ys[:, 3]))

    threads = [threading.Thread(target=calls, args=(56, 57 + 14 * i)) for i in (0, 1, 0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert done == {(56, 57): {_lib.SS2D_OK, True}, (56, 71): {_lib.SS2D_OK, True}}


def test_results_of_kernels_in_front(vb):
    """Library kernels write what the next call reads, and it what they read, call behind call on one stream: as with a wait for the GPU between them."""
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(4, 96, 28, 28, device="cuda", generator=g).bfloat16()
    w = torch.randn(96, 96, device="cuda", generator=g).mul(96 ** -0.5).bfloat16()
    A, D = -torch.rand(384, 1, device="cuda", generator=g), torch.ones(384, device="cuda")

    def chain(between):
        h, out = x, []
        for i in range(24):
            h = torch.matmul(w, h.flatten(2)).view_as(x)
            between()
            xs = vb.cross_scan_fn(h)
            between()
            s = torch.matmul(w[:4], h.flatten(2)).repeat(1, 4, 1).view(4, 4, 4, 784)
            y = vb.selective_scan_fn(xs.view(4, 384, 784), xs.view(4, 384, 784), A, s[:, :, :1], s[:, :, 1:2], D, None, True, True)
            between()
            h = vb.cross_merge_fn(y.view(4, 4, 96, 28, 28)).view_as(x)
            between()
            h = (h / h.std()).bfloat16()
            out.append(h)
        return torch.stack(out)

    want = chain(torch.cuda.synchronize)
    for _ in range(8):
        assert torch.equal(chain(lambda: None), want)
