// The differentiable SS2D core (fused.ss2d_core_autograd) as one autograd node.
//
// Forward: CrossScan of x; x_proj ONCE on the un-scanned map (a 1 x 1 projection commutes with the permutation: a quarter of
// the reads), its rows permuted into route order; dt_projs; selective scan; CrossMerge; LayerNorm.  Backward: LayerNorm,
// the scan of its gradient, the selective-scan gradients (dB, dC written in place into the rows of x_dbl's gradient), the
// four small contractions, CrossMerge.  Rows are padded to a multiple of eight elements where the map's pixel count is
// none, so that the scan and the library's GEMMs see aligned rows whatever H and W are.
#include "host_common.h"

namespace host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

Tensor cross(const Tensor& in, Tensor out, int64_t B, int64_t C, int64_t H, int64_t W, int64_t stride, int op) {
    ss2d_cross_params p = {in.data_ptr(), out.data_ptr(), dtype_code(in), 0, B, C, H, W, stride};
    void* st = stream_of(in);
    if (op == 0) check(ss2d_cross_scan(&p, st), "ss2d_cross_scan");
    else if (op == 1) check(ss2d_cross_merge(&p, st), "ss2d_cross_merge");
    else check(ss2d_cross_rows(&p, op == 3, st), "ss2d_cross_rows");
    return out;
}

// Row stride of the core's route tensors: H * W, or that rounded up to a multiple of eight where the kernels take padded rows.
int64_t padded_row(int64_t B, int64_t C, int64_t H, int64_t W) {
    const int64_t L = H * W, Lp = (L + 7) / 8 * 8;
    if (Lp == L) return L;
    ss2d_cross_params p = {nullptr, nullptr, SS2D_F32, 0, B, C, H, W, Lp};
    return ss2d_cross_padding_supported(&p) ? Lp : L;
}
// cross_rows keeps whole planes in shared memory: 200 KB
bool rows_fit(int64_t H, int64_t W, int64_t esize) { return H * (W | 1) * esize <= 200 * 1024 && H * W <= 65536; }

// (b, k) weights of a batched product: the four routes' matrices, repeated over the images
static Tensor per_image(const Tensor& w, int64_t B) {
    return w.unsqueeze(0).expand({B, 4, w.size(1), w.size(2)}).reshape({B * 4, w.size(1), w.size(2)});
}

// sum over the images of a . b^T (rows of equal length), in fp32; a, b: (images * groups, rows, elements)
static Tensor row_products(const Tensor& a, const Tensor& b, int64_t groups) {
    const bool turned = b.size(1) > a.size(1);                        // the shorter one is the kernel's b
    const Tensor &x = turned ? b : a, &y = turned ? a : b;
    if (a.scalar_type() != at::kFloat && x.stride(2) == 1 && y.stride(2) == 1) {
        ss2d_row_products_params p = {};
        p.a = x.data_ptr(); p.b = y.data_ptr(); p.dtype = dtype_code(a); p.turned = turned;
        p.outer = a.size(0) / groups; p.groups = groups; p.M = x.size(1); p.N = y.size(1); p.L = a.size(2);
        p.a_outer_stride = groups * x.stride(0); p.a_group_stride = x.stride(0); p.a_row_stride = x.stride(1);
        p.b_outer_stride = groups * y.stride(0); p.b_group_stride = y.stride(0); p.b_row_stride = y.stride(1);
        const int64_t need = ss2d_row_products_workspace_bytes(&p);
        if (need > 0 && (uintptr_t)p.a % 16 == 0 && (uintptr_t)p.b % 16 == 0) {
            Tensor out = at::empty({groups, a.size(1), b.size(1)}, a.options().dtype(at::kFloat)), ws = bytes(need, a);
            p.out = out.data_ptr(); p.workspace = ws.data_ptr(); p.workspace_bytes = need;
            check(ss2d_row_products(&p, stream_of(a)), "ss2d_row_products");
            return out;
        }
    }
    const Tensor bt = b.transpose(1, 2);
    const Tensor p = a.scalar_type() == at::kFloat ? at::bmm(a, bt) : at::bmm(a, bt, at::kFloat);
    return p.view({-1, groups, p.size(1), p.size(2)}).sum(0);
}

Tensor expand_rows(const Tensor& xd, const Tensor& wdt, Tensor dts, int64_t B, int64_t D, int64_t R, int64_t N, int64_t S) {
    const int64_t C = R + 2 * N;
    Tensor bc = at::empty({B, 4, 2 * N, S}, xd.options());
    ss2d_expand_params p = {};
    p.x_dbl = xd.data_ptr(); p.dt_weight = wdt.data_ptr();
    p.x_dbl_batch_stride = 4 * C * S; p.x_dbl_route_stride = C * S; p.x_dbl_row_stride = S;
    const int64_t e = xd.element_size();
    for (int64_t k = 0; k < 4; ++k) {
        p.delta[k] = (char*)dts.data_ptr() + k * D * S * e; p.delta_batch_stride[k] = 4 * D * S; p.delta_channel_stride[k] = S;
        p.bc[k] = (char*)bc.data_ptr() + k * 2 * N * S * e; p.bc_batch_stride[k] = 8 * N * S; p.bc_row_stride[k] = S;
    }
    p.B = B; p.D = D; p.R = R; p.N = N; p.H = 1; p.W = S;      // the rows are in route order already: one long row each
    p.act_dtype = dtype_code(xd);
    check(ss2d_route_expand(&p, stream_of(xd)), "ss2d_route_expand");
    return bc;
}

struct CoreNode : public torch::autograd::Function<CoreNode> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& x_proj, const Tensor& dt_projs, const Tensor& dt_bias,
                          const Tensor& A_logs, const Tensor& Ds, const Tensor& ln_w, const Tensor& ln_b, int64_t N, int64_t R, double eps) {
        require_on(x_, {&x_proj, &dt_projs, &dt_bias, &A_logs, &Ds, &ln_w, &ln_b});
        const Tensor x = x_.contiguous();
        const CallGuard guard(x);
        const int64_t B = x.size(0), D = x.size(1), H = x.size(2), W = x.size(3), L = H * W, C = R + 2 * N, S = padded_row(B, D, H, W);
        TORCH_CHECK(ln_w.numel() == D && ln_b.numel() == D, "the LayerNorm's weight and bias must have ", D, " elements, got ", ln_w.numel(), " and ",
                    ln_b.numel());
        const auto of = x.options();
        const Tensor wx = x_proj.reshape({4 * C, D}).to(x.scalar_type()), wdt = dt_projs.reshape({4, D, R}).to(x.scalar_type()).contiguous();
        const Tensor A = A_logs.to(at::kFloat).exp().neg().contiguous(), bias = f32(dt_bias.reshape(-1)), Dp = f32(Ds.reshape(-1));
        const Tensor xs = cross(x, at::empty({B, 4, D, S}, of), B, D, H, W, S, 0);
        Tensor xd = at::empty({B, 4, C, S}, of);
        if (rows_fit(H, W, x.element_size())) {
            const Tensor nat = at::bmm(wx.unsqueeze(0).expand({B, 4 * C, D}), S == L ? x.view({B, D, L}) : xs.select(1, 0));
            cross(nat, xd, B, C, H, W, S, 2);
        } else {
            Tensor out = xd.view({B * 4, C, S});
            at::bmm_out(out, per_image(wx.view({4, C, D}), B), xs.view({B * 4, D, S}));
        }
        Tensor dts = at::empty({B, 4, D, S}, of);
        const Tensor bc = expand_rows(xd, wdt, dts, B, D, R, N, S);
        auto [ys, states] = scan_fwd(xs.view({B, 4 * D, S}), dts.view({B, 4 * D, S}), A, bc.narrow(2, 0, N), bc.narrow(2, N, N), Dp, bias, true, true,
                                     ss2d_selective_scan_checkpoint_every(N, 1), Tensor());
        const Tensor y = cross(ys, at::empty({B, D, L}, of.dtype(at::kFloat)), B, D, H, W, S, 1);
        Tensor out = at::empty({B, D, H, W}, of);
        const Tensor lw = f32(ln_w), lb = f32(ln_b);
        ss2d_norm_params n = {};
        n.in = y.data_ptr(); n.weight = lw.data_ptr(); n.bias = lb.data_ptr(); n.out = out.data_ptr();
        n.B = B; n.D = D; n.L = L; n.io_dtype = dtype_code(x); n.eps = (float)eps;
        check(ss2d_layer_norm_cf(&n, stream_of(x)), "ss2d_layer_norm_cf");
        // all tensors as saved variables: saved-tensor hooks see them, and they are freed as the backward pass advances
        ctx->save_for_backward({x_, x_proj, dt_projs, dt_bias, A_logs, Ds, ln_w, ln_b, xs, xd, dts, bc, states, y, wx, wdt, A});
        ctx->saved_data["n"] = std::vector<int64_t>{B, D, H, W, N, R, S};
        ctx->saved_data["eps"] = eps;
        return out;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const auto in = ctx->get_saved_variables();
        const auto sz = ctx->saved_data["n"].toIntVector();
        const Tensor &xs = in[8], &xd = in[9], &dts = in[10], &bc = in[11], &states = in[12], &y = in[13], &wx = in[14], &wdt = in[15], &A = in[16];
        const int64_t B = sz[0], D = sz[1], H = sz[2], W = sz[3], N = sz[4], R = sz[5], S = sz[6], L = H * W, C = R + 2 * N;
        const CallGuard guard(xs);                // backward() may be called inside an autocast region that the forward was not in
        const auto of = xs.options(), of32 = of.dtype(at::kFloat);
        const Tensor g = grads[0].contiguous(), lw = f32(in[6]);
        Tensor dy = at::empty({B, D, L}, of32), dlw = at::empty({D}, of32), dlb = at::empty({D}, of32);
        {
            ss2d_norm_bwd_params p = {};
            p.y = y.data_ptr(); p.g = g.data_ptr(); p.weight = lw.data_ptr(); p.dy = dy.data_ptr(); p.dweight = dlw.data_ptr(); p.dbias = dlb.data_ptr();
            p.B = B; p.D = D; p.L = L; p.g_dtype = dtype_code(g); p.eps = (float)ctx->saved_data["eps"].toDouble();
            const Tensor ws = bytes(ss2d_layer_norm_cf_bwd_workspace_bytes(&p), xs);
            p.workspace = ws.data_ptr(); p.workspace_bytes = ws.numel();
            check(ss2d_layer_norm_cf_bwd(&p, stream_of(xs)), "ss2d_layer_norm_cf_bwd");
        }
        Tensor dys = cross(dy, at::empty({B, 4, D, S}, of32), B, D, H, W, S, 0);
        dy = Tensor();
        // gradient of x_dbl in route order: rows 0 .. R from the step sizes, the others are dB and dC
        Tensor dxd = at::empty({B, 4, C, S}, of);
        const Tensor bias = f32(in[3].reshape(-1)), Dp = f32(in[5].reshape(-1));
        auto r = scan_bwd_into(xs.view({B, 4 * D, S}), dts.view({B, 4 * D, S}), A, bc.narrow(2, 0, N), bc.narrow(2, N, N), Dp, bias,
                               dys.view({B, 4 * D, S}), true, states, dxd.narrow(2, R, N), dxd.narrow(2, R + N, N));
        dys = Tensor();
        Tensor du = r[0].view({B * 4, D, S});
        const Tensor dd = r[1].view({B * 4, D, S});
        Tensor low = dxd.view({B * 4, C, S}).narrow(1, 0, R);
        at::bmm_out(low, per_image(wdt.transpose(1, 2), B), dd);
        const Tensor dwdt = row_products(dd, xd.view({B * 4, C, S}).narrow(1, 0, R), 4);        // (4, D, R)
        Tensor dwx;
        if (rows_fit(H, W, xs.element_size())) {
            const Tensor nat = cross(dxd, at::empty({B, 4 * C, S}, of), B, C, H, W, S, 3), x0 = xs.select(1, 0);
            dwx = row_products(nat, x0, 1).view({4 * C, D});
            Tensor du0 = du.view({B, 4, D, S}).select(1, 0);                                    // route 0 is the pixel order
            at::baddbmm_out(du0, du0, wx.t().unsqueeze(0).expand({B, D, 4 * C}), nat);
        } else {
            dwx = row_products(dxd.view({B * 4, C, S}), xs.view({B * 4, D, S}), 4).view({4 * C, D});
            at::baddbmm_out(du, du, per_image(wx.view({4, C, D}).transpose(1, 2), B), dxd.view({B * 4, C, S}));
        }
        const Tensor dx = cross(du, at::empty({B, D, H, W}, of), B, D, H, W, S, 1);
        auto as = [](const Tensor& v, const Tensor& like) { return v.reshape(like.sizes()).to(like.scalar_type()); };
        return {dx, as(dwx, in[1]), as(dwdt, in[2]), as(r[6], in[3]), as(r[2].mul(A), in[4]), as(r[5], in[5]), as(dlw, in[6]), as(dlb, in[7]),
                Tensor(), Tensor(), Tensor()};
    }
};

void bind_core(pybind11::module_& m) {
    namespace py = pybind11;
    m.def("ss2d_core_autograd",
          [](const Tensor& x, const Tensor& x_proj, const Tensor& dt_projs, const Tensor& dt_bias, const Tensor& A_logs, const Tensor& Ds,
             const Tensor& ln_w, const Tensor& ln_b, int64_t N, int64_t R, double eps) {
              return CoreNode::apply(x, x_proj, dt_projs, dt_bias, A_logs, Ds, ln_w, ln_b, N, R, eps);
          }, py::call_guard<py::gil_scoped_release>());
}

}  // namespace host
