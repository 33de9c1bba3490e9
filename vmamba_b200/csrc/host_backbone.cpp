// The fused SS2D core and the inference backbone around it, host side (fused.py, backbone.py).
//
// Between the stem and the head every map is channel-major: (C, S) with a channel's B * H * W pixels in a row, S that rounded up
// to a multiple of eight elements, so that every projection is ONE GEMM with aligned rows for any batch and map size (14 x 14
// and 7 x 7 maps of one image: 196 and 49 pixels per row sent the library to its unaligned kernels).  The padding takes
// part in the projections and the elementwise kernels and is never looked at.
#include <map>

#include "host_common.h"

namespace host {

static int64_t round8(int64_t n) { return (n + 7) / 8 * 8; }

struct CoreW {
    Tensor wx, wdt, A, Ds, bias, lnw, lnb;       // (4 (R + 2N), D), (4, D, R), (4 D, N), (4 D), (4 D), (D), (D)
    int64_t N = 0, R = 0, D = 0;
    double eps = 1e-5;
};
struct Map {                                      // channel-major
    Tensor t;                                     // (C, S), or anything whose data is that
    int64_t C, B, H, W, S;
    int64_t L() const { return H * W; }
    Map like(int64_t channels, at::ScalarType type) const { return {at::empty({channels, S}, t.options().dtype(type)), channels, B, H, W, S}; }
    Map like(int64_t channels) const { return like(channels, t.scalar_type()); }
};

static Tensor linear_cm(const Tensor& w, const Tensor& x, int64_t S) {      // x: (K, S)
    ss2d_linear_params p = {};
    p.x = x.data_ptr(); p.w = w.data_ptr(); p.M = w.size(0); p.K = w.size(1); p.N = S; p.dtype = dtype_code(x);
    if (x.scalar_type() != at::kFloat) {
        Tensor y = at::empty({p.M, S}, x.options());
        p.out = y.data_ptr();
        if (ss2d_linear_supported(&p) == SS2D_OK) {
            check(ss2d_linear_fwd(&p, stream_of(x)), "ss2d_linear_fwd");
            return y;
        }
    }
    return at::mm(w, x);
}

// -------------------------------------------------------------------------------------------- the core
// Route streams: delta and B / C rows of the two orientations (even: routes 0, 2; odd: 1, 3) and two routes each.
struct Streams { Tensor bc, delta; bool cm, x_cm; int64_t S, pad; };      // x_cm: x's own layout; pad: elements per image row, 0: dense

// Whether the streams' rows are better padded (the library's planner decides).
static bool prefers_padded(const CoreW& w, at::ScalarType type, bool cm, int64_t B, int64_t H, int64_t W, int64_t S) {
    ss2d_core_params q = {};
    q.x = (void*)(intptr_t)4096;                 // an aligned address: the query dereferences nothing
    q.B = B; q.D = w.D; q.H = H; q.W = W; q.N = w.N; q.act_dtype = dtype_code(type);
    q.x_batch_stride = cm ? H * W : w.D * H * W; q.x_channel_stride = cm ? S : H * W;
    return ss2d_core_prefers_padded_rows(&q) != 0;
}

// x: channel-major, or (B, D, L) with S = L
static Streams project(const Tensor& x, bool cm, int64_t B, int64_t H, int64_t W, int64_t S, const CoreW& w, bool padding) {
    const int64_t D = w.D, R = w.R, N = w.N, C = R + 2 * N, L = H * W;
    ss2d_expand_params p = {};
    Streams s;
    s.x_cm = cm;
    s.pad = padding && prefers_padded(w, x.scalar_type(), cm, B, H, W, S) ? round8(L) : 0;
    // 16-bit (B, D, L) maps whose planes are no whole vectors: a channel-major copy, so that the images of a row are one run and
    // projection and expansion take the tensor-core kernels (whole core, 128 x 768 planes of 7 x 7 269 -> 109 us,
    // 1 x 384 of 14 x 14 32 -> 25 us of kernels)
    Tensor xc = x;
    if (!cm && padding && !s.pad && L % 8 != 0 && R <= 64 && x.scalar_type() != at::kFloat) {
        cm = true;
        S = round8(B * L);
        xc = at::empty({D, S}, x.options());
        Tensor from = x.view({B, D, L}), to = xc.narrow(1, 0, B * L).view({D, B, L});
        const int64_t e = L % 4 == 0 ? 4 : L % 2 == 0 ? 2 : 1;        // elements moved as one word
        if (e > 1 && x.storage_offset() % e == 0 && (uintptr_t)x.data_ptr() % (2 * e) == 0) {
            const auto word = e == 4 ? at::kLong : at::kInt;
            from = from.view(word); to = to.view(word);
        }
        to.copy_(from.transpose(0, 1));
    }
    s.cm = cm;
    s.S = S;
    Tensor xd;
    auto at_el = [](const Tensor& t, int64_t i) { return (char*)t.data_ptr() + i * t.element_size(); };
    if (cm) {
        xd = linear_cm(w.wx, xc.view({D, S}), S);
        p.x_dbl_batch_stride = L; p.x_dbl_route_stride = C * S; p.x_dbl_row_stride = S;
        if (!s.pad) {
            s.delta = at::empty({2, 2, D, S}, x.options());
            s.bc = at::empty({2, 2, 2 * N, S}, x.options());
            for (int k = 0; k < 4; ++k) {
                const int64_t i = (k % 2) * 2 + k / 2;
                p.delta[k] = at_el(s.delta, i * D * S); p.delta_batch_stride[k] = L; p.delta_channel_stride[k] = S;
                p.bc[k] = at_el(s.bc, i * 2 * N * S); p.bc_batch_stride[k] = L; p.bc_row_stride[k] = S;
            }
            p.padded_rows = S > B * L;
        }
    } else {
        xd = at::matmul(w.wx, x.view({B, D, L}));
        p.x_dbl_batch_stride = 4 * C * L; p.x_dbl_route_stride = C * L; p.x_dbl_row_stride = L;
        if (!s.pad) {
            s.delta = at::empty({2, B, 2, D, L}, x.options());
            s.bc = at::empty({2, B, 2, 2 * N, L}, x.options());
            for (int k = 0; k < 4; ++k) {
                const int64_t j = k % 2, i = k / 2;
                p.delta[k] = at_el(s.delta, (j * B * 2 + i) * D * L); p.delta_batch_stride[k] = 2 * D * L;
                p.bc[k] = at_el(s.bc, (j * B * 2 + i) * 2 * N * L); p.bc_batch_stride[k] = 4 * N * L;
            }
        }
    }
    if (s.pad) {            // rows of an image padded: one (route, channel, image, row) layout for either layout of x
        const int64_t n = B * s.pad;
        s.delta = at::empty({4, D, n}, x.options());
        s.bc = at::empty({4, 2 * N, n}, x.options());
        for (int k = 0; k < 4; ++k) {
            p.delta[k] = at_el(s.delta, k * D * n); p.delta_batch_stride[k] = s.pad; p.delta_channel_stride[k] = n;
            p.bc[k] = at_el(s.bc, k * 2 * N * n); p.bc_batch_stride[k] = s.pad; p.bc_row_stride[k] = n;
        }
        p.image_row = s.pad;
    }
    p.x_dbl = xd.data_ptr(); p.dt_weight = w.wdt.data_ptr();
    p.B = B; p.D = D; p.R = R; p.N = N; p.H = H; p.W = W; p.act_dtype = dtype_code(x);
    const int64_t need = ss2d_route_expand_workspace_bytes(&p);      // room for the transposed rows of the column-major routes
    Tensor ws;
    if (need > 0) { ws = bytes(need, x); p.workspace = ws.data_ptr(); p.workspace_bytes = need; }
    check(ss2d_route_expand(&p, stream_of(x)), "ss2d_route_expand");
    return s;
}

static ss2d_core_params core_params(const Tensor& x, const Streams& s, const CoreW& w, int64_t B, int64_t H, int64_t W) {
    const int64_t L = H * W, S = s.S, D = w.D, N = w.N, e = x.element_size();
    ss2d_core_params p = {};
    p.x = x.data_ptr();
    for (int k = 0; k < 4; ++k) {
        const int64_t j = k % 2, i = k / 2;
        if (s.pad) {
            const int64_t n = B * s.pad;
            p.delta[k] = (char*)s.delta.data_ptr() + k * D * n * e; p.delta_batch_stride[k] = s.pad; p.delta_channel_stride[k] = n;
            p.Bm[k] = (char*)s.bc.data_ptr() + k * 2 * N * n * e; p.Cm[k] = (char*)p.Bm[k] + N * n * e; p.bc_batch_stride[k] = s.pad;
        } else if (s.cm) {
            p.delta[k] = (char*)s.delta.data_ptr() + (j * 2 + i) * D * S * e; p.delta_batch_stride[k] = L; p.delta_channel_stride[k] = S;
            p.Bm[k] = (char*)s.bc.data_ptr() + (j * 2 + i) * 2 * N * S * e; p.Cm[k] = (char*)p.Bm[k] + N * S * e; p.bc_batch_stride[k] = L;
        } else {
            p.delta[k] = (char*)s.delta.data_ptr() + (j * B * 2 + i) * D * L * e; p.delta_batch_stride[k] = 2 * D * L; p.delta_channel_stride[k] = L;
            p.Bm[k] = (char*)s.bc.data_ptr() + (j * B * 2 + i) * 2 * N * L * e; p.Cm[k] = (char*)p.Bm[k] + N * L * e; p.bc_batch_stride[k] = 4 * N * L;
        }
    }
    p.A = w.A.data_ptr(); p.Dskip = w.Ds.data_ptr(); p.delta_bias = w.bias.data_ptr(); p.ln_weight = ptr(w.lnw); p.ln_bias = ptr(w.lnb);
    p.B = B; p.D = D; p.H = H; p.W = W; p.N = N; p.act_dtype = dtype_code(x); p.ln_eps = (float)w.eps;
    p.stream_row = s.pad;
    if (s.x_cm) { p.x_batch_stride = p.y_batch_stride = L; p.x_channel_stride = p.y_channel_stride = S; }
    return p;
}

// Whether ss2d_core_fwd takes the map (its planner decides from sizes, strides and types); `padding`: with padded rows too.
static bool core_takes(const CoreW& w, at::ScalarType type, bool cm, int64_t B, int64_t H, int64_t W, int64_t S, bool padding) {
    if (padding && prefers_padded(w, type, cm, B, H, W, S)) return true;
    const int64_t L = H * W;
    ss2d_core_params p = {};
    void* some = (void*)(intptr_t)4096;          // an aligned address: the query dereferences nothing
    p.x = p.A = p.Dskip = p.delta_bias = some; p.y = some;
    for (int k = 0; k < 4; ++k) {
        p.delta[k] = p.Bm[k] = p.Cm[k] = some;
        p.delta_batch_stride[k] = cm ? L : 2 * w.D * L; p.delta_channel_stride[k] = cm ? S : L; p.bc_batch_stride[k] = cm ? L : 4 * w.N * L;
    }
    p.B = B; p.D = w.D; p.H = H; p.W = W; p.N = w.N; p.act_dtype = p.y_dtype = dtype_code(type); p.with_norm = 1;
    if (cm) { p.x_batch_stride = p.y_batch_stride = L; p.x_channel_stride = p.y_channel_stride = S; }
    return ss2d_core_supported(&p) == SS2D_OK;
}

static void norm_cf(const Tensor& in, const Tensor& out, const CoreW& w, int64_t B, int64_t L, int64_t bs, int64_t cs, int64_t obs, int64_t ocs) {
    ss2d_norm_params n = {};
    n.in = in.data_ptr(); n.weight = ptr(w.lnw); n.bias = ptr(w.lnb); n.out = out.data_ptr();
    n.B = B; n.D = w.D; n.L = L; n.batch_stride = bs; n.channel_stride = cs; n.out_batch_stride = obs; n.out_channel_stride = ocs;
    n.io_dtype = dtype_code(out); n.eps = (float)w.eps;
    check(ss2d_layer_norm_cf(&n, stream_of(in)), "ss2d_layer_norm_cf");
}

// The same mathematics through the operator kernels, for what the fused kernel does not take: CrossScan, projections, scan,
// CrossMerge, LayerNorm (vmamba.py:1536-1571).  Channel-major maps: the images of a channel are planes of one big image.
static Tensor core_by_operators(const Tensor& x, bool cm, int64_t B, int64_t H, int64_t W, int64_t S, const CoreW& w, bool with_norm,
                                at::ScalarType out_type, Tensor out) {
    const int64_t D = w.D, N = w.N, R = w.R, C = R + 2 * N, L = H * W, Bi = cm ? 1 : B, planes = cm ? D * B : D;
    const auto of = x.options(), of32 = of.dtype(at::kFloat);
    const int64_t P = padded_row(Bi, planes, H, W);                   // elements per row of a route
    const bool dense = !cm || S == B * L;
    const Tensor xin = dense ? x : x.view({D, S}).narrow(1, 0, B * L).contiguous();
    const int64_t n = cm ? B * P : P;                                 // a channel's elements in one route (of one image)
    Tensor xs = at::empty({Bi, 4, D, n}, of);
    cross(xin, xs, Bi, planes, H, W, P, 0);
    Tensor xd = at::empty({Bi, 4, C, n}, of);
    if (rows_fit(H, W, x.element_size())) {                           // x_proj once, on the pixel order; its rows permuted
        const Tensor x0 = P == L ? xin.view({Bi, D, n}) : xs.select(1, 0);
        const Tensor nat = cm ? linear_cm(w.wx, x0.view({D, n}), n) : at::bmm(w.wx.unsqueeze(0).expand({Bi, 4 * C, D}), x0);
        cross(nat, xd, Bi, cm ? C * B : C, H, W, P, 2);
    } else {
        for (int64_t k = 0; k < 4; ++k) {
            Tensor o = xd.select(1, k);
            at::bmm_out(o, w.wx.view({4, C, D})[k].unsqueeze(0).expand({Bi, C, D}), xs.select(1, k));
        }
    }
    Tensor dts = at::empty({Bi, 4, D, n}, of);
    const Tensor bc = expand_rows(xd, w.wdt, dts, Bi, D, R, N, n);
    // rows (b, k d) and groups (b, k, n) of the scan as views
    auto rows_of = [&](const Tensor& t) { return cm ? t.view({4 * D, B, P}).permute({1, 0, 2}) : t.view({B, 4 * D, P}); };
    auto group = [&](int64_t first) {
        return cm ? bc.view({4, 2 * N, B, P}).narrow(1, first, N).permute({2, 0, 1, 3}) : bc.view({B, 4, 2 * N, P}).narrow(2, first, N);
    };
    Tensor ys = at::empty({Bi, 4, D, n}, of32);
    scan_fwd(rows_of(xs), rows_of(dts), w.A, group(0), group(N), w.Ds, w.bias, true, true, 0, rows_of(ys));
    const Tensor y = cross(ys, at::empty({Bi, planes, L}, of32), Bi, planes, H, W, P, 1);
    if (!with_norm) {
        TORCH_CHECK(dense, "an un-normalised padded map is not provided");
        return y.view(x.sizes()).to(out_type);
    }
    if (!out.defined()) out = at::empty_like(x, of.dtype(out_type));
    if (cm) norm_cf(y, out, w, B, L, L, B * L, L, S);
    else norm_cf(y, out, w, B, L, D * L, L, D * L, L);
    return out;
}

static Tensor core_run(const Tensor& x, bool cm, int64_t B, int64_t H, int64_t W, int64_t S, const CoreW& w, bool with_norm, at::ScalarType out_type,
                       Tensor workspace, Tensor out) {
    if (!core_takes(w, x.scalar_type(), cm, B, H, W, S, true) || (cm && !with_norm))
        return core_by_operators(x, cm, B, H, W, S, w, with_norm, out_type, out);
    const Streams s = project(x, cm, B, H, W, S, w, true);
    if (!out.defined()) out = at::empty_like(x, x.options().dtype(out_type));
    ss2d_core_params p = core_params(x, s, w, B, H, W);
    p.y = out.data_ptr(); p.y_dtype = dtype_code(out); p.with_norm = with_norm;
    const int64_t need = ss2d_core_workspace_bytes(&p);
    TORCH_CHECK(need >= 0, "ss2d_core_workspace_bytes: invalid arguments");
    if (need > 0) {
        if (!workspace.defined() || (int64_t)workspace.nbytes() < need) workspace = bytes(need, x);
        p.workspace = workspace.data_ptr(); p.workspace_bytes = workspace.nbytes();
    }
    const int rc = ss2d_core_fwd(&p, stream_of(x));
    if (rc == SS2D_ENOTSUP) return core_by_operators(x, cm, B, H, W, S, w, with_norm, out_type, out);   // an alignment the query could not see
    check(rc, "ss2d_core_fwd");
    return out;
}

// Weights whose data the kernels read by address: of the stated size and type, in one piece.
static void expect(const char* name, const Tensor& t, std::vector<int64_t> sizes, at::ScalarType type) {
    TORCH_CHECK(t.defined() && t.sizes() == at::IntArrayRef(sizes), name, " must be ", at::IntArrayRef(sizes), ", got ", t.sizes());
    TORCH_CHECK(t.scalar_type() == type, name, " must be ", type, ", got ", t.scalar_type());
    TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
}

static CoreW core_weights(const Tensor& wx, const Tensor& wdt, const Tensor& A, const Tensor& Ds, const Tensor& bias, const OptT& lnw, const OptT& lnb,
                          int64_t N, int64_t R, double eps) {
    CoreW w;
    w.wx = wx; w.wdt = wdt; w.A = A; w.Ds = Ds; w.bias = bias; w.lnw = opt(lnw); w.lnb = opt(lnb);
    w.N = N; w.R = R; w.D = wx.size(-1); w.eps = eps;
    const int64_t K = 4;
    expect("wx", wx, {K * (R + 2 * N), w.D}, wx.scalar_type());
    expect("wdt", wdt, {K, w.D, R}, wx.scalar_type());
    expect("A", A, {K * w.D, N}, at::kFloat);
    expect("Ds", Ds, {K * w.D}, at::kFloat);
    expect("dt_bias", bias, {K * w.D}, at::kFloat);
    for (const Tensor* t : {&w.lnw, &w.lnb})
        if (t->defined()) expect("ln_weight / ln_bias", *t, {w.D}, at::kFloat);
    return w;
}

static void check_core(const Tensor& x, const CoreW& w, bool cm) {
    require_on(x, {&w.wx, &w.wdt, &w.A, &w.Ds, &w.bias, &w.lnw, &w.lnb});
    TORCH_CHECK(x.dim() == 4 && x.size(cm ? 0 : 1) == w.D, "x must be a 4-d map of ", w.D, " channels, got ", x.sizes());
    TORCH_CHECK(x.scalar_type() == w.wx.scalar_type() && x.scalar_type() == w.wdt.scalar_type(), "x is ", x.scalar_type(),
                ", the weights were built for ", w.wx.scalar_type(), " and ", w.wdt.scalar_type());
}

// -------------------------------------------------------------------------------------------- the backbone
struct Norm { Tensor w, b; };
struct Block {
    Norm n1, n2;
    Tensor w_in, w_dw, w_out, w1, b1, w2, b2;
    CoreW core;
};
struct Down { bool there = false; Tensor w, b; Norm n; };

class Backbone {
public:
    // stem: w0, b0, norm0 (w, b), w1, b1, norm1 (w, b)
    std::vector<Tensor> stem;
    std::vector<std::vector<Block>> stages;
    std::vector<Down> downs;
    std::vector<Tensor> head;                     // norm (w, b), weight, bias; empty without a classifier
    std::map<int64_t, Norm> outnorm;
    at::ScalarType type = at::kBFloat16;

    void add_block(bool first, std::vector<Tensor> t, const CoreW& core) {
        Block b;
        b.n1 = {t[0], t[1]}; b.n2 = {t[2], t[3]};
        b.w_in = t[4]; b.w_dw = t[5]; b.w_out = t[6]; b.w1 = t[7]; b.b1 = t[8]; b.w2 = t[9]; b.b2 = t[10];
        b.core = core;
        if (first) stages.emplace_back();
        stages.back().push_back(std::move(b));
    }
    void add_down(std::vector<Tensor> t) {        // w, b, norm (w, b), or nothing
        Down d;
        if (!t.empty()) { d.there = true; d.w = t[0]; d.b = t[1]; d.n = {t[2], t[3]}; }
        downs.push_back(d);
    }

    // every part of the size that the parts around it ask for, once per model
    void validate() const {
        auto norm_of = [](const char* name, const Norm& n, int64_t C) {
            expect(name, n.w, {C}, at::kFloat);
            expect(name, n.b, {C}, at::kFloat);
        };
        TORCH_CHECK(stem.size() == 8 && stages.size() == downs.size() && !stages.empty(), "a backbone needs a stem and stages");
        const int64_t C0 = stem[0].size(0);
        int64_t C = stem[4].size(0);
        expect("patch_embed.0.weight", stem[0], {C0, stem[0].size(1), 3, 3}, type);
        expect("patch_embed.0.bias", stem[1], {C0}, at::kFloat);
        norm_of("patch_embed.2", {stem[2], stem[3]}, C0);
        expect("patch_embed.5.bias", stem[5], {C}, at::kFloat);
        norm_of("patch_embed.7", {stem[6], stem[7]}, C);
        for (size_t i = 0; i < stages.size(); ++i) {
            for (const Block& b : stages[i]) {
                const int64_t D = b.w_in.size(0), hidden = b.w1.size(0);
                norm_of("norm", b.n1, C);
                norm_of("norm2", b.n2, C);
                expect("op.in_proj", b.w_in, {D, C}, type);
                TORCH_CHECK(b.w_dw.numel() == 9 * D, "op.conv2d must have 3 x 3 weights for ", D, " channels, got ", b.w_dw.sizes());
                expect("op.conv2d", b.w_dw.view({D, 9}), {D, 9}, type);
                expect("op.out_proj", b.w_out, {C, D}, type);
                expect("mlp.fc1", b.w1, {hidden, C}, type);
                expect("mlp.fc1.bias", b.b1, {hidden}, at::kFloat);
                expect("mlp.fc2", b.w2, {C, hidden}, type);
                expect("mlp.fc2.bias", b.b2, {C}, at::kFloat);
                TORCH_CHECK(b.core.D == D && b.core.wx.scalar_type() == type, "the core must have ", D, " channels of ", type);
                TORCH_CHECK(b.core.lnw.defined() && b.core.lnb.defined(), "the core needs its LayerNorm");
            }
            const auto it = outnorm.find((int64_t)i);
            if (it != outnorm.end()) norm_of("outnorm", it->second, C);
            if (downs[i].there) {
                C = downs[i].w.size(0);
                expect("downsample bias", downs[i].b, {C}, at::kFloat);
                norm_of("downsample norm", downs[i].n, C);
            }
        }
        if (!head.empty()) norm_of("classifier.norm", {head[0], head[1]}, C);
    }
    Tensor forward(const Tensor& img) {
        TORCH_CHECK(!head.empty(), "this model was built without a classifier");
        at::NoGradGuard no_grad;
        require_on(img, {&stem.at(0)});
        const CallGuard guard(img);
        const Tensor x = run(img, nullptr);
        return at::linear(x.mean({2, 3}).to(type), head[2], head[3]);
    }
    std::vector<Tensor> features(const Tensor& img, const std::vector<int64_t>& which) {
        at::NoGradGuard no_grad;
        require_on(img, {&stem.at(0)});
        const CallGuard guard(img);
        std::vector<Map> maps;
        run(img, &maps);
        std::vector<Tensor> out;
        for (int64_t i : which) {
            const auto it = outnorm.find(i);
            if (it == outnorm.end()) throw pybind11::key_error(std::to_string(i));
            const Map& m = maps.at(i);
            Tensor y = at::empty({m.B, m.C, m.H, m.W}, m.t.options());
            norm(m, Map{}, Tensor(), it->second, y, m.B, false, m.L(), m.C * m.L(), m.L());
            out.push_back(y);
        }
        return out;
    }

private:
    // LayerNorm over channels of x (+ add + add_bias, written back with `update`) into `out`; images: how many runs the pixels
    // are taken as (1: one row of S pixels per channel, the output laid out like the input)
    static void norm(const Map& x, const Map& add, const Tensor& add_bias, const Norm& n, const Tensor& out, int64_t images, bool update,
                     int64_t run, int64_t obs, int64_t ocs, bool normalize = true) {
        ss2d_norm_params p = {};
        p.in = x.t.data_ptr(); p.add = ptr(add.t); p.add_bias = ptr(add_bias); p.sum_out = update ? x.t.data_ptr() : nullptr;
        p.weight = ptr(n.w); p.bias = ptr(n.b); p.out = out.data_ptr();
        p.B = images; p.D = x.C; p.L = run; p.batch_stride = images > 1 ? run : x.S * x.C; p.channel_stride = x.S;
        p.out_batch_stride = obs; p.out_channel_stride = ocs;
        p.io_dtype = dtype_code(out); p.eps = 1e-5f; p.skip_norm = !normalize;
        check(ss2d_layer_norm_cf(&p, stream_of(x.t)), "ss2d_layer_norm_cf");
    }
    Map norm_run(const Map& x, const Map& add, const Tensor& add_bias, const Norm& n, bool update) const {
        Map y = x.like(x.C, type);
        norm(x, add, add_bias, n, y.t, 1, update, x.S, x.S * x.C, x.S);
        return y;
    }
    static Map pw(const Tensor& w, const Map& x) {                    // 1 x 1 projection (vmamba.py:1060-1064)
        Map y = x;
        y.C = w.size(0);
        y.t = at::mm(w, x.t);
        return y;
    }
    Map dwconv(const Map& x, const Tensor& w) const {
        Map y = x.like(x.C);
        ss2d_pointwise_params p = {};
        p.x = x.t.data_ptr(); p.weight = w.data_ptr(); p.y = y.t.data_ptr();
        p.B = x.B; p.D = x.C; p.H = x.H; p.W = x.W; p.dtype = dtype_code(x.t); p.act = 2; p.channel_major = 1; p.channel_stride = x.S;
        check(ss2d_dwconv3x3_act(&p, stream_of(x.t)), "ss2d_dwconv3x3_act");
        return y;
    }
    Map mlp(const Map& x, const Block& b) const {                     // without the bias of fc2 (vmamba.py:1151-1167)
        if (type != at::kFloat) {
            Map y = x.like(x.C);
            ss2d_mlp_params p = {};
            p.x = x.t.data_ptr(); p.w1 = b.w1.data_ptr(); p.b1 = b.b1.data_ptr(); p.w2 = b.w2.data_ptr(); p.y = y.t.data_ptr();
            p.C = x.C; p.hidden = b.w1.size(0); p.N = x.S; p.dtype = dtype_code(x.t);
            if (ss2d_mlp_supported(&p) == SS2D_OK) {
                check(ss2d_mlp_fwd(&p, stream_of(x.t)), "ss2d_mlp_fwd");
                return y;
            }
        }
        if (type != at::kFloat) {                                     // few pixels: bias and GELU in the projection's epilogue
            ss2d_linear_params p = {};
            Map h = x.like(b.w1.size(0));
            p.x = x.t.data_ptr(); p.w = b.w1.data_ptr(); p.bias = b.b1.data_ptr(); p.out = h.t.data_ptr();
            p.M = h.C; p.K = x.C; p.N = x.S; p.dtype = dtype_code(x.t); p.act = 1;
            if (ss2d_linear_supported(&p) == SS2D_OK) {
                check(ss2d_linear_fwd(&p, stream_of(x.t)), "ss2d_linear_fwd");
                return pw(b.w2, h);
            }
        }
        const Map h = pw(b.w1, x);
        ss2d_pointwise_params p = {};
        p.x = p.y = h.t.data_ptr(); p.bias = b.b1.data_ptr();
        p.B = 1; p.D = h.C; p.H = 1; p.W = h.S; p.dtype = dtype_code(h.t); p.act = 1; p.channel_major = 1;
        check(ss2d_bias_act(&p, stream_of(h.t)), "ss2d_bias_act");
        return pw(b.w2, h);
    }
    // 3 x 3 stride-2 convolution (library) of a pixel-major map
    static Tensor conv_s2(const Tensor& rows, const Tensor& w) {
        return at::conv2d(rows.permute({0, 3, 1, 2}), w, {}, {2, 2}, {1, 1}).permute({0, 2, 3, 1}).contiguous();
    }
    static Map planes(const Tensor& rows, const Tensor& bias, const Norm& n) {       // + bias, LayerNorm, pixel-major -> channel-major fp32
        Map m;
        m.B = rows.size(0); m.H = rows.size(1); m.W = rows.size(2); m.C = rows.size(3); m.S = round8(m.B * m.L());
        m.t = at::empty({m.C, m.S}, rows.options().dtype(at::kFloat));
        ss2d_relayout_params p = {};
        p.rows = rows.data_ptr(); p.planes = m.t.data_ptr(); p.bias = ptr(bias); p.ln_weight = ptr(n.w); p.ln_bias = ptr(n.b);
        p.N = m.B * m.L(); p.C = m.C; p.plane_stride = m.S; p.rows_dtype = dtype_code(rows); p.planes_dtype = SS2D_F32; p.eps = 1e-5f;
        check(ss2d_pixels_norm_to_planes(&p, stream_of(rows)), "ss2d_pixels_norm_to_planes");
        return m;
    }
    Tensor pixels(const Map& x, const Map& add, const Tensor& bias, bool update) const {
        Tensor rows = at::empty({x.B, x.H, x.W, x.C}, x.t.options().dtype(type));
        ss2d_relayout_params p = {};
        p.rows = rows.data_ptr(); p.planes = x.t.data_ptr(); p.add = add.t.data_ptr(); p.bias = ptr(bias); p.sum_out = update ? x.t.data_ptr() : nullptr;
        p.N = x.B * x.L(); p.C = x.C; p.plane_stride = x.S; p.rows_dtype = dtype_code(rows); p.planes_dtype = SS2D_F32;
        check(ss2d_planes_to_pixels(&p, stream_of(x.t)), "ss2d_planes_to_pixels");
        return rows;
    }
    // patch embed v2 (vmamba.py:1928-1942)
    Map embed(const Tensor& image) const {
        const Tensor img = image.to(type).contiguous();
        const int64_t C0 = stem[0].size(0), B = img.size(0), H = img.size(2), W = img.size(3);
        Tensor x;
        if (img.size(1) == 3 && (C0 == 32 || C0 == 48 || C0 == 64)) {
            x = at::empty({B, (H + 1) / 2, (W + 1) / 2, C0}, img.options());
            ss2d_stem_params p = {};
            p.x = img.data_ptr(); p.weight = stem[0].data_ptr(); p.conv_bias = stem[1].data_ptr(); p.ln_weight = stem[2].data_ptr();
            p.ln_bias = stem[3].data_ptr(); p.y = x.data_ptr();
            p.B = B; p.H = H; p.W = W; p.C0 = C0; p.in_channels = 3; p.dtype = dtype_code(img); p.act = 1; p.eps = 1e-5f;
            check(ss2d_stem_conv_norm_act(&p, stream_of(img)), "ss2d_stem_conv_norm_act");
        } else {
            const Tensor c = at::conv2d(img, stem[0], {}, {2, 2}, {1, 1}).contiguous();
            Tensor y = at::empty_like(c);
            ss2d_norm_params p = {};
            p.add = c.data_ptr(); p.add_bias = stem[1].data_ptr(); p.weight = stem[2].data_ptr(); p.bias = stem[3].data_ptr(); p.out = y.data_ptr();
            p.B = B; p.D = C0; p.L = c.size(2) * c.size(3); p.io_dtype = dtype_code(y); p.eps = 1e-5f;
            check(ss2d_layer_norm_cf(&p, stream_of(c)), "ss2d_layer_norm_cf");
            x = at::gelu(y).permute({0, 2, 3, 1}).contiguous();
        }
        return planes(conv_s2(x, stem[4]), stem[5], {stem[6], stem[7]});
    }
    // The stages.  With `maps` the residual maps behind every stage; else returns the normalised last map for the classifier.
    Tensor run(const Tensor& img, std::vector<Map>* maps) const {
        Map x = embed(img);
        const Norm none;
        for (size_t i = 0; i < stages.size(); ++i) {
            const auto& stage = stages[i];
            Map h = norm_run(x, Map{}, Tensor(), stage[0].n1, false), m;
            for (size_t j = 0; j < stage.size(); ++j) {               // VSSBlock._forward, eval mode (vmamba.py:1766-1778)
                const Block& b = stage[j];
                h = dwconv(pw(b.w_in, h), b.w_dw);
                Map c = h.like(b.core.D);
                core_run(h.t, true, h.B, h.H, h.W, h.S, b.core, true, type, Tensor(), c.t);
                const Map o = pw(b.w_out, c);
                h = norm_run(x, o, Tensor(), b.n2, true);             // residual update fused with the norm that follows it
                m = mlp(h, b);
                if (j + 1 < stage.size()) h = norm_run(x, m, b.b2, stage[j + 1].n1, true);
            }
            const Tensor& mb = stage.back().b2;
            const Down& d = downs[i];
            if (d.there) {
                // downsample v3 (vmamba.py:1964-1971): x + m + bias as the pixel-major 16-bit input of the strided convolution in one
                // pass (written back into x only when the stage's map is asked for)
                const Tensor rows = pixels(x, m, mb, maps != nullptr);
                if (maps) maps->push_back(x);
                x = planes(conv_s2(rows, d.w), d.b, d.n);
            } else if (maps) {
                Map y = x.like(x.C, type);
                norm(x, m, mb, none, y.t, 1, true, x.S, x.S * x.C, x.S, false);
                maps->push_back(x);
            } else {                                                  // classifier norm fused with the last residual update
                Tensor last = at::empty({x.B, x.C, x.H, x.W}, x.t.options());
                m.t = m.t.to(at::kFloat);
                norm(x, m, mb, {head[0], head[1]}, last, x.B, true, x.L(), x.C * x.L(), x.L());
                return last;
            }
        }
        return Tensor();
    }
};

void bind_backbone(pybind11::module_& m) {
    namespace py = pybind11;
    using release = py::call_guard<py::gil_scoped_release>;
    py::class_<CoreW>(m, "CoreWeights")
        .def(py::init(&core_weights), py::arg("wx"), py::arg("wdt"), py::arg("A"), py::arg("Ds"), py::arg("bias"), py::arg("ln_weight"),
             py::arg("ln_bias"), py::arg("d_state"), py::arg("dt_rank"), py::arg("eps"));
    // x: contiguous (D, B, H, W) with channel_major, else (B, D, H, W)
    m.def("ss2d_core",
          [](const Tensor& x, const CoreW& w, bool with_norm, at::ScalarType out_type, const OptT& workspace, bool cm) {
              check_core(x, w, cm);
              const int64_t B = x.size(cm ? 1 : 0), H = x.size(2), W = x.size(3);
              const CallGuard guard(x);
              at::NoGradGuard no_grad;
              return core_run(x, cm, B, H, W, cm ? B * H * W : H * W, w, with_norm, out_type, opt(workspace), Tensor());
          }, release());
    m.def("ss2d_core_by_operators",
          [](const Tensor& x, const CoreW& w, bool with_norm, at::ScalarType out_type, bool cm) {
              check_core(x, w, cm);
              const int64_t B = x.size(cm ? 1 : 0), H = x.size(2), W = x.size(3);
              const CallGuard guard(x);
              return core_by_operators(x, cm, B, H, W, cm ? B * H * W : H * W, w, with_norm, out_type, Tensor());
          }, release());
    m.def("project",
          [](const Tensor& x, const CoreW& w, bool cm) {
              check_core(x, w, cm);
              const int64_t B = x.size(cm ? 1 : 0), H = x.size(2), W = x.size(3);
              const CallGuard guard(x);
              const Streams s = project(x, cm, B, H, W, cm ? B * H * W : H * W, w, false);
              return std::make_pair(s.bc, s.delta);
          }, release());
    m.def("core_takes",
          [](std::vector<int64_t> shape, int64_t d_state, at::ScalarType type, bool cm) {
              CoreW w;
              w.D = shape[cm ? 0 : 1]; w.N = d_state;
              const int64_t B = shape[cm ? 1 : 0], L = shape[2] * shape[3];
              return core_takes(w, type, cm, B, shape[2], shape[3], cm ? B * L : L, false);      // of dense streams
          });
    py::class_<Backbone>(m, "Backbone")
        .def(py::init<>())
        .def_readwrite("stem", &Backbone::stem)
        .def_readwrite("head", &Backbone::head)
        .def_readwrite("dtype", &Backbone::type)
        .def("add_block", &Backbone::add_block)
        .def("add_down", &Backbone::add_down)
        .def("validate", &Backbone::validate)
        .def("add_outnorm", [](Backbone& b, int64_t i, const Tensor& w, const Tensor& bias) { b.outnorm[i] = {w, bias}; })
        .def("forward", &Backbone::forward, release())
        .def("features", &Backbone::features, release());
}

}  // namespace host
