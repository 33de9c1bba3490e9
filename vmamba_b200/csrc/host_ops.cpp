// Selective scan, CrossScan and CrossMerge: argument checks, results, workspaces and autograd nodes.
#include "host_common.h"

namespace host {

int64_t scan_ratio(const Tensor& u, const Tensor& delta) { return u.size(1) / delta.size(1); }

std::pair<Tensor, Tensor> scan_fwd(Tensor u, Tensor delta, Tensor A, Tensor B, Tensor C, Tensor D, Tensor bias, bool softplus, bool out_float,
                                   int64_t every, Tensor out) {
    require_cuda({&u, &delta, &A, &B, &C, &D, &bias});
    TORCH_CHECK(u.dim() == 3 && delta.dim() == 3 && delta.size(0) == u.size(0) && delta.size(2) == u.size(2) && delta.size(1) != 0 &&
                    u.size(1) % delta.size(1) == 0,
                "u must be (batch, dim, L) and delta (batch, dim / r, L), got ", u.sizes(), " ", delta.sizes());
    TORCH_CHECK(B.dim() == 4 && C.sizes() == B.sizes(), "B and C must be (batch, n_groups, dstate, L) with equal shapes");
    const int64_t batch = u.size(0), dim = u.size(1), L = u.size(2), K = B.size(1), N = B.size(2);
    TORCH_CHECK(B.size(0) == batch && B.size(3) == L && K > 0 && dim % K == 0, "B/C shape does not match u");
    TORCH_CHECK(A.dim() == 2 && A.size(0) == dim && A.size(1) == N, "A must be (dim, dstate) = (", dim, ", ", N, "), got ", A.sizes());
    TORCH_CHECK(delta.scalar_type() == u.scalar_type() && B.scalar_type() == u.scalar_type() && C.scalar_type() == u.scalar_type(),
                "u, delta, B, C must share one dtype");
    u = rows(u); delta = rows(delta); B = rows(B); C = rows(C);
    A = f32(A); D = f32(D); bias = f32(bias);
    TORCH_CHECK(!D.defined() || D.numel() == dim, "D must have dim elements");
    const int64_t ratio = scan_ratio(u, delta);          // channels sharing one delta row (selective_scan_oflex.cpp:59)
    TORCH_CHECK(!bias.defined() || bias.numel() == delta.size(1), "delta_bias must have one element per delta row");
    const auto out_type = out_float ? at::kFloat : u.scalar_type();
    const int in_code = dtype_code(u);
    if (!out.defined()) out = at::empty({batch, dim, L}, u.options().dtype(out_type));
    else
        TORCH_CHECK(out.dim() == 3 && out.size(0) == batch && out.size(1) == dim && out.size(2) == L && out.scalar_type() == out_type &&
                        out.stride(-1) == 1 && out.device() == u.device(),
                    "out must be (batch, dim, L) of the result type on u's device with contiguous rows");
    ss2d_scan_params p = {};
    p.u = u.data_ptr(); p.delta = delta.data_ptr(); p.A = A.data_ptr(); p.B = B.data_ptr(); p.C = C.data_ptr();
    p.D = ptr(D); p.delta_bias = ptr(bias); p.out = out.data_ptr();
    p.in_dtype = in_code; p.out_dtype = dtype_code(out);
    p.delta_softplus = softplus; p.delta_ratio = (int32_t)ratio;
    p.batch = batch; p.dim = dim; p.dstate = N; p.seqlen = L; p.n_groups = K;
    p.u_batch_stride = u.stride(0); p.u_dim_stride = u.stride(1);
    p.delta_batch_stride = delta.stride(0); p.delta_dim_stride = delta.stride(1);
    p.out_batch_stride = out.stride(0); p.out_dim_stride = out.stride(1);
    p.B_batch_stride = B.stride(0); p.B_group_stride = B.stride(1); p.B_state_stride = B.stride(2);
    p.C_batch_stride = C.stride(0); p.C_group_stride = C.stride(1); p.C_state_stride = C.stride(2);
    Tensor ckpt, ws;
    if (every) {
        ckpt = at::empty({batch, dim, (L + every - 1) / every, N}, u.options().dtype(at::kFloat));
        p.checkpoints = ckpt.data_ptr(); p.checkpoint_every = every;
    }
    if (N > 1) {            // rows too few to fill the GPU are walked in segments
        const int64_t need = ss2d_selective_scan_fwd_workspace_bytes(&p);
        if (need > 0) { ws = bytes(need, u); p.workspace = ws.data_ptr(); p.workspace_bytes = need; }
    }
    const c10::cuda::OptionalCUDAGuard guard(u.device());
    check(ss2d_selective_scan_fwd(&p, stream_of(u)), "ss2d_selective_scan_fwd");
    return {out, ckpt};
}

std::vector<Tensor> scan_bwd(Tensor u, Tensor delta, Tensor A, Tensor B, Tensor C, Tensor D, Tensor bias, Tensor dout, bool softplus, Tensor ckpt) {
    return scan_bwd_into(u, delta, A, B, C, D, bias, dout, softplus, ckpt, Tensor(), Tensor());
}

std::vector<Tensor> scan_bwd_into(Tensor u, Tensor delta, Tensor A, Tensor B, Tensor C, Tensor D, Tensor bias, Tensor dout, bool softplus, Tensor ckpt,
                                  Tensor dB, Tensor dC) {
    require_cuda({&u, &delta, &A, &B, &C, &D, &bias, &dout});
    TORCH_CHECK(dout.sizes() == u.sizes(), "dout must have the shape of u, got ", dout.sizes());
    TORCH_CHECK(dout.scalar_type() == at::kFloat || dout.scalar_type() == u.scalar_type(), "dout must be fp32 or of u's dtype");
    const int64_t batch = u.size(0), dim = u.size(1), L = u.size(2), K = B.size(1), N = B.size(2);
    u = rows(u); delta = rows(delta); B = rows(B); C = rows(C); dout = rows(dout);
    A = f32(A); D = f32(D); bias = f32(bias);
    const auto of = u.options(), of32 = of.dtype(at::kFloat);
    Tensor du = at::empty({batch, dim, L}, of), ddelta = at::empty({batch, dim, L}, of), dA = at::empty({dim, N}, of32);
    if (!dB.defined()) { dB = at::empty({batch, K, N, L}, of); dC = at::empty({batch, K, N, L}, of); }
    Tensor dD = D.defined() ? at::empty({dim}, of32) : Tensor(), dbias = bias.defined() ? at::empty({dim}, of32) : Tensor();
    ss2d_scan_bwd_params p = {};
    p.u = u.data_ptr(); p.delta = delta.data_ptr(); p.A = A.data_ptr(); p.B = B.data_ptr(); p.C = C.data_ptr(); p.D = ptr(D);
    p.delta_bias = ptr(bias); p.dout = dout.data_ptr();
    p.du = du.data_ptr(); p.ddelta = ddelta.data_ptr(); p.dA = dA.data_ptr(); p.dB = dB.data_ptr(); p.dC = dC.data_ptr();
    p.dD = ptr(dD); p.ddelta_bias = ptr(dbias);
    p.in_dtype = dtype_code(u); p.dout_dtype = dtype_code(dout);
    const int64_t ratio = scan_ratio(u, delta);
    p.delta_softplus = softplus; p.delta_ratio = (int32_t)ratio;
    p.batch = batch; p.dim = dim; p.dstate = N; p.seqlen = L; p.n_groups = K;
    p.u_batch_stride = u.stride(0); p.u_dim_stride = u.stride(1);
    p.delta_batch_stride = delta.stride(0); p.delta_dim_stride = delta.stride(1);
    p.dout_batch_stride = dout.stride(0); p.dout_dim_stride = dout.stride(1);
    p.B_batch_stride = B.stride(0); p.B_group_stride = B.stride(1); p.B_state_stride = B.stride(2);
    p.C_batch_stride = C.stride(0); p.C_group_stride = C.stride(1); p.C_state_stride = C.stride(2);
    p.bc_out_group_stride = dB.stride(1);
    const int64_t every = ss2d_selective_scan_checkpoint_every(N, ratio);
    p.checkpoint_every = every;
    if (ckpt.defined()) {
        const int64_t far = (L + 127) / 128, near = (L + every - 1) / every;
        TORCH_CHECK(ckpt.scalar_type() == at::kFloat && ckpt.dim() == 4 && ckpt.size(0) == batch && ckpt.size(1) == dim &&
                        (ckpt.size(2) == far || ckpt.size(2) == near) && ckpt.size(3) == N && ckpt.is_contiguous() && ckpt.device() == u.device(),
                    "checkpoints must be the fp32 (batch, dim, ceil(L/128), dstate) tensor of the forward call");
        if (ckpt.size(2) == near) p.checkpoints = ckpt.data_ptr();      // the kernels form their own where these are too far apart
    }
    const int64_t need = ss2d_selective_scan_bwd_workspace_bytes(&p);
    TORCH_CHECK(need >= 0, "ss2d_selective_scan_bwd_workspace_bytes: invalid or unsupported arguments");
    Tensor ws = bytes(std::max<int64_t>(need, 16), u);
    p.workspace = ws.data_ptr(); p.workspace_bytes = ws.numel();
    const c10::cuda::OptionalCUDAGuard guard(u.device());
    check(ss2d_selective_scan_bwd(&p, stream_of(u)), "ss2d_selective_scan_bwd");
    if (ratio > 1) {        // rows that shared a delta row: their gradients add up (selective_scan_oflex.cpp:348-352)
        ddelta = ddelta.view({batch, dim / ratio, ratio, L}).to(at::kFloat).sum(2).to(u.scalar_type());
        if (dbias.defined()) dbias = dbias.view({dim / ratio, ratio}).sum(1);
    }
    return {du, ddelta, dA, dB, dC, dD, dbias};
}

// The node that selective_scan_fn leaves in the graph (SelectiveScanCuda, csms6s.py:71-109): saves the inputs and the states
// that the gradient kernels read.
struct ScanNode : public torch::autograd::Function<ScanNode> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& u, const Tensor& delta, const Tensor& A, const Tensor& B,
                          const Tensor& C, const OptT& D_, const OptT& bias_, bool softplus, bool out_float) {
        const Tensor D = opt(D_), bias = opt(bias_);
        const int64_t ratio = u.dim() == 3 && delta.dim() == 3 && delta.size(1) ? scan_ratio(u, delta) : 1;
        auto [out, ckpt] = scan_fwd(u, delta, A, B, C, D, bias, softplus, out_float, ss2d_selective_scan_checkpoint_every(A.size(-1), ratio), Tensor());
        ctx->save_for_backward({u, delta, A, B, C, D, bias, ckpt});
        ctx->saved_data["softplus"] = softplus;
        return out;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list g) {
        const auto s = ctx->get_saved_variables();
        auto r = scan_bwd(s[0], s[1], s[2], s[3], s[4], s[5], s[6], g[0], ctx->saved_data["softplus"].toBool(), s[7]);
        auto as = [](const Tensor& x, const Tensor& like) { return x.defined() && x.scalar_type() != like.scalar_type() ? x.to(like.scalar_type()) : x; };
        return {r[0], r[1], as(r[2], s[2]), r[3], r[4], as(r[5], s[5]), as(r[6], s[6]), Tensor(), Tensor()};
    }
};

static bool wants_grad(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t->defined() && t->requires_grad()) return true;
    return false;
}

static Tensor scan_fn(const Tensor& u, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C, const OptT& D_, const OptT& bias_,
                      bool softplus, bool oflex) {
    const Tensor D = opt(D_), bias = opt(bias_);
    if (wants_grad({&u, &delta, &A, &B, &C, &D, &bias})) return ScanNode::apply(u, delta, A, B, C, D_, bias_, softplus, oflex);
    return scan_fwd(u, delta, A, B, C, D, bias, softplus, oflex, 0, Tensor()).first;
}

Tensor cross_scan(const Tensor& x_, int64_t scans) {
    require_cuda({&x_});
    TORCH_CHECK(x_.dim() == 4, "cross_scan expects a (B, C, H, W) tensor");
    const Tensor x = x_.contiguous();
    const int64_t B = x.size(0), C = x.size(1), H = x.size(2), W = x.size(3);
    Tensor y = at::empty({B, 4, C, H * W}, x.options());
    ss2d_cross_params p = {x.data_ptr(), y.data_ptr(), dtype_code(x), (int32_t)scans, B, C, H, W};
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    check(ss2d_cross_scan(&p, stream_of(x)), "ss2d_cross_scan");
    return y;
}

Tensor cross_merge(const Tensor& ys_, int64_t scans) {
    require_cuda({&ys_});
    TORCH_CHECK(ys_.dim() == 5, "cross_merge expects a 5-d tensor of four routes");
    const Tensor ys = ys_.contiguous();
    const int64_t B = ys.size(0), C = ys.size(2), H = ys.size(3), W = ys.size(4);
    TORCH_CHECK(ys.size(1) == 4, "cross_merge expects (B, 4, C, H, W)");
    Tensor y = at::empty({B, C, H * W}, ys.options());
    ss2d_cross_params p = {ys.data_ptr(), y.data_ptr(), dtype_code(ys), (int32_t)scans, B, C, H, W};
    const c10::cuda::OptionalCUDAGuard guard(ys.device());
    check(ss2d_cross_merge(&p, stream_of(ys)), "ss2d_cross_merge");
    return y;
}

// The adjoint of the four-route copy is the four-route sum and the reverse (csm_triton.py:182-273).
struct CrossScanNode : public torch::autograd::Function<CrossScanNode> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, int64_t scans) {
        Tensor y = cross_scan(x, scans);
        ctx->saved_data["scans"] = scans;
        ctx->saved_data["shape"] = x.sizes().vec();
        return y;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list g) {
        const auto s = ctx->saved_data["shape"].toIntVector();
        return {cross_merge(g[0].contiguous().view({s[0], 4, s[1], s[2], s[3]}), ctx->saved_data["scans"].toInt()).view(s), Tensor()};
    }
};
struct CrossMergeNode : public torch::autograd::Function<CrossMergeNode> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& ys, int64_t scans) {
        Tensor y = cross_merge(ys, scans);
        ctx->saved_data["scans"] = scans;
        ctx->saved_data["shape"] = ys.sizes().vec();
        return y;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list g) {
        const auto s = ctx->saved_data["shape"].toIntVector();
        return {cross_scan(g[0].contiguous().view({s[0], s[2], s[3], s[4]}), ctx->saved_data["scans"].toInt()).view(s), Tensor()};
    }
};

static Tensor cross_scan_fn(const Tensor& x, int64_t scans) {
    return wants_grad({&x}) ? CrossScanNode::apply(x, scans) : cross_scan(x, scans);
}
static Tensor cross_merge_fn(const Tensor& ys, int64_t scans) {
    return wants_grad({&ys}) ? CrossMergeNode::apply(ys, scans) : cross_merge(ys, scans);
}

void bind_ops(pybind11::module_& m) {
    namespace py = pybind11;
    using release = py::call_guard<py::gil_scoped_release>;
    m.def("selective_scan_fn", &scan_fn, release());
    m.def("selective_scan_fwd",
          [](const Tensor& u, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C, const OptT& D, const OptT& bias, bool softplus,
             bool out_float, int64_t every, const OptT& out) {
              return scan_fwd(u, delta, A, B, C, opt(D), opt(bias), softplus, out_float, every, opt(out));
          }, release());
    m.def("selective_scan_bwd",
          [](const Tensor& u, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C, const OptT& D, const OptT& bias,
             const Tensor& dout, bool softplus, const OptT& ckpt) {
              return scan_bwd(u, delta, A, B, C, opt(D), opt(bias), dout, softplus, opt(ckpt));
          }, release());
    m.def("cross_scan", &cross_scan, release());
    m.def("cross_merge", &cross_merge, release());
    m.def("cross_scan_fn", &cross_scan_fn, release());
    m.def("cross_merge_fn", &cross_merge_fn, release());
}

}  // namespace host
