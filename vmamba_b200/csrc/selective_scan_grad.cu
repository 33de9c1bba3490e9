// Planner and launches of the selective-scan gradients for 1 .. 16 states (scan_n1_bwd.cuh, scan_states_bwd.cuh).
#include "scan_states_bwd.cuh"
#include "selective_scan_grad.cuh"

namespace ss2d {

int selective_scan_fwd(const ss2d_scan_params* p, cudaStream_t st);
long long selective_scan_fwd_workspace_bytes(const ss2d_scan_params* p);
long long selective_scan_checkpoint_every(int64_t dstate, int64_t delta_ratio);

// Workspace, in floats, in this order (every part a multiple of 4): per-row sums, dB / dC partials, reverse end states and
// their sums (segments), the states where the forward call did not leave them, the workspace of the call that forms them.
struct GradPlan {
    int NS, vw, parts, sets, S, seg_len, Lp;     // sets: rows per warp (one state), sets of 32 rows (more)
    bool recompute;
    int64_t rowred, bcpart, ends, sums, ckpt, fwd, total;
};

static int64_t pad4(int64_t n) { return (n + 3) / 4 * 4; }

static ss2d_scan_params forward_of(const ss2d_scan_bwd_params* p, int every) {
    ss2d_scan_params f = {};
    f.u = p->u; f.delta = p->delta; f.A = p->A; f.B = p->B; f.C = p->C; f.D = nullptr; f.delta_bias = p->delta_bias;
    f.out = p->du;                      // not written: the states alone are asked for
    f.in_dtype = f.out_dtype = p->in_dtype;
    f.delta_softplus = p->delta_softplus; f.delta_ratio = p->delta_ratio;
    f.batch = p->batch; f.dim = p->dim; f.dstate = p->dstate; f.seqlen = p->seqlen; f.n_groups = p->n_groups;
    f.u_batch_stride = p->u_batch_stride; f.u_dim_stride = p->u_dim_stride;
    f.delta_batch_stride = p->delta_batch_stride; f.delta_dim_stride = p->delta_dim_stride;
    f.out_batch_stride = p->dim * p->seqlen; f.out_dim_stride = p->seqlen;
    f.B_batch_stride = p->B_batch_stride; f.B_group_stride = p->B_group_stride; f.B_state_stride = p->B_state_stride;
    f.C_batch_stride = p->C_batch_stride; f.C_group_stride = p->C_group_stride; f.C_state_stride = p->C_state_stride;
    f.checkpoints = p->du;              // replaced before the call is made
    f.checkpoint_every = every;
    f.states_only = 1;
    return f;
}

bool selective_scan_grad_takes(const ss2d_scan_bwd_params* p) {
    return p->checkpoint_every > 0 && selective_scan_checkpoint_every(p->dstate, p->delta_ratio) != 128;
}

static int n1_lanes(int64_t L) { return L <= 64 ? 8 : L <= 128 ? 16 : 32; }      // lanes per row

static int plan_grad(const ss2d_scan_bwd_params* p, GradPlan& c) {
    const int64_t L = p->seqlen, gs = p->dim / p->n_groups, rows = p->batch * p->dim, N = p->dstate;
    const size_t si = dtype_size(p->in_dtype), sg = dtype_size(p->dout_dtype);
    auto ptr_el = [](const void* q, size_t s) { return (int64_t)(reinterpret_cast<uintptr_t>(q) / s); };
    int v = 8;
    for (int64_t x : {L, p->u_batch_stride, p->u_dim_stride, p->delta_batch_stride, p->delta_dim_stride, p->dout_batch_stride, p->dout_dim_stride,
                      p->B_batch_stride, p->B_group_stride, p->B_state_stride, p->C_batch_stride, p->C_group_stride, p->C_state_stride,
                      ptr_el(p->u, si), ptr_el(p->delta, si), ptr_el(p->B, si), ptr_el(p->C, si), ptr_el(p->dout, sg), ptr_el(p->du, si), ptr_el(p->ddelta, si)})
        while (v > 1 && x % v != 0) v >>= 1;
    c.vw = v >= 8 ? 8 : v >= 4 ? 4 : 1;
    c.Lp = (int)((L + 31) / 32 * 32);
    const int64_t every = selective_scan_checkpoint_every(N, p->delta_ratio);
    c.recompute = !p->checkpoints || p->checkpoint_every != every;
    const int64_t groups = p->batch * p->n_groups;
    if (N == 1) {
        c.NS = 1;
        // rows per warp: as many as leave two CTAs per SM (the sums over rows of a chunk are then formed once for all of them; three
        // CTAs are resident, 153 to 168 registers).  us with one, two, three, four and six left, bf16: 32 x 384 rows of 3 136 elements
        // 170, 167, 177, 181, 199; 8 x 384 of 3 136 81, 61, 75, 75, 75; 8 x 768 of 784 50, 38, 45, 53, 54; 16 x 768 of 784 63, 63,
        // 65, 65, 73; 4 x 384 of 3 136 54, 44, 44, 44, 44
        const int64_t step = kN1Warps * (32 / n1_lanes(L));
        auto parts_of = [&](int64_t R) { return (gs + step * R - 1) / (step * R); };
        c.sets = 1;
        while (c.sets < kN1MaxR && step * c.sets < gs && groups * parts_of(c.sets * 2) >= 148 * 2) c.sets *= 2;
        c.parts = (int)parts_of(c.sets);
        const int64_t ctas = groups * c.parts;
        c.S = 1; c.seg_len = (int)((L + kN1Chunk - 1) / kN1Chunk * kN1Chunk);
        if (ctas * 2 <= 148 * 4 && L >= 4 * kN1Chunk) {
            const int64_t s = std::min<int64_t>((148 * 4 + ctas - 1) / ctas, L / (2 * kN1Chunk));
            c.seg_len = (int)(((L + s - 1) / s + kN1Chunk - 1) / kN1Chunk * kN1Chunk);
            c.S = (int)((L + c.seg_len - 1) / c.seg_len);
        }
    } else {
        c.NS = st_pad_states(N);
        // Eight warps fit an SM (240 registers).  Row sets and segments are chosen for the shortest schedule, in units of a
        // hundredth of a row set's walk: a CTA costs 100 per set and 29 for the sums over its rows, a wave takes as long
        // as a CTA, and cutting rows adds a pass of 25 per row set.
        const int64_t parts1 = (gs + kStRows - 1) / kStRows, slots = 148 * 8 / (c.NS / 4);
        double best = 0;
        c.S = 0;
        for (int sets = 1; sets <= kStMaxSets && sets <= parts1; sets *= 2) {
            const int64_t parts = (parts1 + sets - 1) / sets, ctas = groups * parts;
            for (int64_t s = 1; s <= 64 && (s == 1 || L >= s * 64); ++s) {
                const int64_t len = ((L + s - 1) / s + 63) / 64 * 64, S = (L + len - 1) / len, waves = (ctas * S + slots - 1) / slots;
                const double cost = (double)waves * (100 * sets + 29) * (double)len / (double)L + (S > 1 ? 25.0 * (double)(groups * parts1) / (double)slots : 0.0);
                if (c.S == 0 || cost < 0.97 * best) { best = cost; c.sets = sets; c.parts = (int)parts; c.S = (int)S; c.seg_len = (int)len; }
            }
        }
    }
    c.rowred = pad4(c.S * rows * (N + 2));
    c.bcpart = groups * c.parts * 2 * N * c.Lp;
    c.ends = c.S > 1 ? pad4(rows * c.S * c.NS) : 0;
    c.sums = c.S > 1 ? pad4(rows * c.S) : 0;
    c.ckpt = c.recompute ? pad4(rows * ((L + every - 1) / every) * N) : 0;
    c.fwd = 0;
    if (c.recompute) {
        const ss2d_scan_params f = forward_of(p, (int)every);
        const long long b = selective_scan_fwd_workspace_bytes(&f);
        if (b < 0) return SS2D_EINVAL_SHAPE;
        c.fwd = pad4(b / 4);
    }
    c.total = c.rowred + c.bcpart + c.ends + c.sums + c.ckpt + c.fwd;
    return SS2D_OK;
}

long long selective_scan_grad_workspace_bytes(const ss2d_scan_bwd_params* p) {
    GradPlan c;
    return plan_grad(p, c) == SS2D_OK ? (long long)c.total * 4 : -1;
}

template <typename Tin, typename Tg, int AL, int BC>
static int launch_n1_bwd(const N1BwdArgs& a, cudaStream_t st) {
    const size_t smem = sizeof(float) * (2 * kN1Warps * 2 * kN1Chunk + (size_t)kN1Warps * a.R * (4 * (32 / n1_lanes(a.L)) + 96) + (AL ? 0 : kN1Warps * 264));
    const int lpr = n1_lanes(a.L);
    auto kern = lpr == 8 ? n1_bwd_kernel<Tin, Tg, AL, 8, BC> : lpr == 16 ? n1_bwd_kernel<Tin, Tg, AL, 16, BC> : n1_bwd_kernel<Tin, Tg, AL, 32, BC>;
    if (const int rc = allow_dynamic_smem(kern, smem)) return rc;
    const int64_t ctas = a.batch * a.n_groups * a.parts * a.S, seg_ctas = (a.batch * a.dim * (a.S - 1) + kN1Warps - 1) / kN1Warps;
    if (ctas > 0x7fffffffLL || seg_ctas > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
    if (a.S > 1) {
        launch(n1_bwd_segments_kernel<Tin, Tg, AL, BC>, (unsigned)seg_ctas, kN1Warps * 32, 0, st, a);
        count_launch();
    }
    launch(kern, (unsigned)ctas, kN1Warps * 32, smem, st, a);
    count_launch();
    return check_launch();
}

template <typename Tin, typename Tg, int NS, int VW>
static int launch_st_bwd(const StBwdArgs& a, cudaStream_t st) {
    using Y = StLayout<NS>;
    const size_t smem = StBwdSmem<NS>::bytes(a.sets);
    auto kern = st_bwd_kernel<Tin, Tg, NS, VW>;
    if (const int rc = allow_dynamic_smem(kern, smem)) return rc;
    const int64_t ctas = a.batch * a.n_groups * a.parts * a.S;
    const int64_t seg_ctas = a.batch * a.n_groups * ((a.group_size + kStRows - 1) / kStRows) * (a.S - 1);
    if (ctas > 0x7fffffffLL || seg_ctas > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
    if (a.S > 1) {
        const size_t s2 = sizeof(float) * (2 * kStRows * kStPitch + kStChunk * Y::BCP);
        launch(st_bwd_segments_kernel<Tin, Tg, NS, VW>, (unsigned)seg_ctas, Y::kWarps * 32, s2, st, a);
        count_launch();
    }
    launch(kern, (unsigned)ctas, Y::kWarps * 32, smem, st, a);
    count_launch();
    return check_launch();
}

template <typename Tin, typename Tg>
static int dispatch_grad(const ss2d_scan_bwd_params* p, const GradPlan& c, float* ws, const float* ckpt, cudaStream_t st) {
    if (c.NS == 1) {
        N1BwdArgs a = {};
        a.u = p->u; a.delta = p->delta; a.B = p->B; a.C = p->C; a.dout = p->dout;
        a.A = (const float*)p->A; a.D = (const float*)p->D; a.bias = (const float*)p->delta_bias;
        a.du = p->du; a.ddelta = p->ddelta;
        a.rowred = ws; a.bcpart = ws + c.rowred; a.eagg = a.bcpart + c.bcpart; a.esum = a.eagg + c.ends; a.ckpt = ckpt;
        a.dim = p->dim; a.group_size = p->dim / p->n_groups; a.batch = p->batch; a.dratio = p->delta_ratio > 1 ? p->delta_ratio : 1;
        a.u_bs = p->u_batch_stride; a.u_ds = p->u_dim_stride; a.d_bs = p->delta_batch_stride; a.d_ds = p->delta_dim_stride;
        a.g_bs = p->dout_batch_stride; a.g_ds = p->dout_dim_stride;
        a.B_bs = p->B_batch_stride; a.B_gs = p->B_group_stride; a.C_bs = p->C_batch_stride; a.C_gs = p->C_group_stride;
        const ScanSpans s = scan_spans(*p, dtype_size(p->in_dtype));
        a.L = (int)p->seqlen; a.Lp = c.Lp; a.n_groups = (int)p->n_groups; a.parts = c.parts; a.R = c.sets; a.S = c.S; a.seg_len = c.seg_len;
        a.softplus = p->delta_softplus;
        // rows without vectors: pieces of the tensors that start and end on 16-byte boundaries; else single elements
        const Span g = span_of(p->dout, dtype_size(p->dout_dtype), (p->batch - 1) * p->dout_batch_stride + (p->dim - 1) * p->dout_dim_stride + p->seqlen);
        const bool pieces = whole_pieces(s.u) && whole_pieces(s.delta) && whole_pieces(g);
        return c.vw == 8                                        ? launch_n1_bwd<Tin, Tg, 8, 8>(a, st)
               : c.vw == 4                                      ? launch_n1_bwd<Tin, Tg, 4, 4>(a, st)
               : !pieces                                        ? launch_n1_bwd<Tin, Tg, 1, 1>(a, st)
               : whole_pieces(s.B) && whole_pieces(s.C)         ? launch_n1_bwd<Tin, Tg, 0, 0>(a, st)
                                                                : launch_n1_bwd<Tin, Tg, 0, 1>(a, st);
    }
    StBwdArgs a = {};
    a.u = p->u; a.delta = p->delta; a.B = p->B; a.C = p->C; a.dout = p->dout;
    a.A = (const float*)p->A; a.D = (const float*)p->D; a.bias = (const float*)p->delta_bias;
    a.du = p->du; a.ddelta = p->ddelta;
    a.rowred = ws; a.bcpart = ws + c.rowred; a.ends = a.bcpart + c.bcpart; a.sums = a.ends + c.ends; a.ckpt = ckpt;
    a.dim = p->dim; a.group_size = p->dim / p->n_groups; a.batch = p->batch;
    a.u_bs = p->u_batch_stride; a.u_ds = p->u_dim_stride; a.d_bs = p->delta_batch_stride; a.d_ds = p->delta_dim_stride;
    a.g_bs = p->dout_batch_stride; a.g_ds = p->dout_dim_stride;
    a.B_bs = p->B_batch_stride; a.B_gs = p->B_group_stride; a.B_ss = p->B_state_stride;
    a.C_bs = p->C_batch_stride; a.C_gs = p->C_group_stride; a.C_ss = p->C_state_stride;
    a.L = (int)p->seqlen; a.Lp = c.Lp; a.N = (int)p->dstate; a.n_groups = (int)p->n_groups; a.parts = c.parts; a.sets = c.sets;
    a.softplus = p->delta_softplus; a.S = c.S; a.seg_len = c.seg_len;
#define SS2D_ST(NS_)                                                                                       \
    if (c.NS == NS_)                                                                                       \
        return c.vw == 8   ? launch_st_bwd<Tin, Tg, NS_, 8>(a, st)                                         \
               : c.vw == 4 ? launch_st_bwd<Tin, Tg, NS_, 4>(a, st)                                         \
                           : launch_st_bwd<Tin, Tg, NS_, 1>(a, st);
    SS2D_ST(4)
    SS2D_ST(8)
    SS2D_ST(16)
#undef SS2D_ST
    return SS2D_ENOTSUP;
}

int selective_scan_grad(const ss2d_scan_bwd_params* p, BwdFold& fold, cudaStream_t st) {
    GradPlan c;
    const int rc = plan_grad(p, c);
    if (rc != SS2D_OK) return rc;
    if (!p->workspace || p->workspace_bytes < (long long)c.total * 4) return SS2D_EWORKSPACE;
    if (!aligned_to(p->workspace, 16)) return SS2D_EINVAL_ALIGN;
    float* ws = (float*)p->workspace;
    const float* ckpt = (const float*)p->checkpoints;
    if (c.recompute) {
        float* at = ws + c.rowred + c.bcpart + c.ends + c.sums;
        ss2d_scan_params f = forward_of(p, (int)selective_scan_checkpoint_every(p->dstate, p->delta_ratio));
        f.checkpoints = at;
        f.workspace = c.fwd ? at + c.ckpt : nullptr; f.workspace_bytes = c.fwd * 4;
        const int r = selective_scan_fwd(&f, st);
        if (r != SS2D_OK) return r;
        ckpt = at;
    }
    if (c.NS > 1 && p->dstate == c.NS && !aligned_to(ckpt, 16)) return SS2D_EINVAL_ALIGN;
    fold.rowred = ws; fold.bcpart = ws + c.rowred; fold.images = (int64_t)c.S * p->batch; fold.parts = c.parts; fold.Lp = c.Lp;
    const bool gf32 = p->dout_dtype == SS2D_F32;
    if (p->in_dtype == SS2D_F32) return dispatch_grad<float, float>(p, c, ws, ckpt, st);
    if (p->in_dtype == SS2D_BF16)
        return gf32 ? dispatch_grad<__nv_bfloat16, float>(p, c, ws, ckpt, st) : dispatch_grad<__nv_bfloat16, __nv_bfloat16>(p, c, ws, ckpt, st);
    return gf32 ? dispatch_grad<__half, float>(p, c, ws, ckpt, st) : dispatch_grad<__half, __half>(p, c, ws, ckpt, st);
}

}  // namespace ss2d
