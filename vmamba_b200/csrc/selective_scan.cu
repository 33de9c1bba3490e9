// Selective-scan forward, the operator surface: planner, launches, and the kernels for one state and for many.
//
// One state (every VMamba backbone): selscan_fwd_n1_kernel.  2 .. 16 states: scan_states_fwd.cuh.  More than 16 states, and more than
// one where channels share a row of step sizes: selscan_fwd_nx_kernel, a warp per row, the carry of every state in shared memory.
// In all of them u and delta are read once and the result is written once; the B / C rows, shared by the channels of a
// group, come from the caches.
#include <type_traits>

#include "scan_row.cuh"
#include "scan_states_fwd.cuh"

namespace ss2d {

struct ScanArgs {
    const void *u, *delta, *B, *C;
    const float *A, *D, *bias;
    void* out;
    int64_t rows, dim, dstate, seqlen, group_size;
    int64_t u_bs, u_ds, d_bs, d_ds, o_bs, o_ds;
    int64_t B_bs, B_gs, B_ss, C_bs, C_gs, C_ss;
    ScanSpans span;
    int softplus;
    int64_t dratio;   // channels per delta row
    float* ckpt;      // (rows, nck, dstate) or null
    int64_t nck;
    int every;        // elements between the states kept in ckpt
    bool states_only; // no result, the states alone
};

constexpr int kWarpsPerCta = 4;

// d_state 1: W warps per row (1: four rows per CTA; 2 .. 8: the CTA is one row).  Per step a warp takes 256 elements, eight
// per lane, and scans its lanes' (a, b) pairs by shuffle; with several warps per row their totals meet in shared memory
// (one barrier per step) and every warp folds the ones in front of it.  How many: n1_warps.  The next step's vectors are
// fetched in front of this one's arithmetic.
// Bound, 1 024 rows of 16 385 elements (four warps each, 45 us, 20 % of the DRAM rate): instruction issue, 72 % of the slots of an SM
// that has work, and 1 024 CTAs on the 740 places that 91 registers leave, so that the second wave is a third full.  32 x 384 rows of
// 3 136 with the states kept, 66 us: issue (79 %) and HBM (330 MB, 50 us at the copy rate).  Arithmetic in pairs, 50 and 70 us before.
// AL is the vector width of every access (8 or 4 elements), or 0 for rows of any alignment: a row is then walked from
// the 16-byte boundary in front of its result, so that the results leave as vectors, and the inputs are cut out of the
// aligned pieces around them.  Elements of the tensors' first and last rows whose pieces would reach beyond a tensor (at most
// seven at either end) are taken one by one in front of the walk and behind it.
// `every` (a multiple of 8): spacing of the states kept for the backward pass.
// Rows of at most 128 (64) elements share a warp, two (four) at a time, LPR = 16 (8) lanes each.
// fp32 rows of any alignment are held to 128 registers, four CTAs per SM (12 288 rows of 3 137 elements: 170 -> 132 us).
template <typename Tin, typename Tout, int AL, int W, int LPR>
__global__ void __launch_bounds__(W == 1 ? kWarpsPerCta * 32 : W * 32, W == 1 && AL == 0 && sizeof(Tin) == 4 ? 4 : 0) selscan_fwd_n1_kernel(const ScanArgs a) {
    follow_previous();
    static_assert(W == 1 || LPR == 32, "rows of several warps take whole warps");
    // Elementwise arithmetic in pairs, but where it measured slower.  fp32 pieces are at their 128 registers and would spill (12 288 rows of 3 137
    // elements 124 -> 136 us).  Whole vectors, in pairs / one by one: two warps of 16-bit rows, 2 048 rows of 65 536 elements bf16 215 / 194 us, f16 211 / 189,
    // of 16 384 56 / 51 and 55 / 50; four warps of bf16 rows, 1 024 of 65 536 110 / 98 (f16 110 / 117); one warp of fp32 rows, 3 584 of
    // 65 536 572 / 551.  Else 16-bit rows gain: 3 584 of 65 536 bf16 325 / 354, 256 of 65 536 35.0 / 37.3.
    // (Vectors of four, single warps, in pairs: bf16, 3 584 rows of 65 540 413, 385 before the pairs; of 3 140 20.1 and 22.6.)
    constexpr bool kOneByOne = (AL == 0 && sizeof(Tin) == 4) ||
                               (AL == 8 && (sizeof(Tin) == 4 ? W == 1 : W == 2 || (W == 4 && std::is_same<Tin, __nv_bfloat16>::value)));
    constexpr bool kPacked = !kOneByOne;
    constexpr int VEC = 8, WSTEP = LPR * VEC, STEP = W * WSTEP;
    __shared__ AB agg[2][W];
    const int lane = threadIdx.x & (LPR - 1), wi = W == 1 ? 0 : threadIdx.x >> 5;
    int64_t row = W == 1 ? ((int64_t)blockIdx.x * (kWarpsPerCta * 32) + threadIdx.x) / LPR : (int64_t)blockIdx.x;
    if (row - (threadIdx.x & 31) / LPR >= a.rows) return;      // whole warps (whole CTAs where W > 1)
    const bool real = LPR == 32 || row < a.rows;               // the last warp's spare lanes repeat its last row, unseen
    if (!real) row = a.rows - 1;
    const int64_t b = row / a.dim, r = row - b * a.dim, k = r / a.group_size;
    const int64_t rd_ = a.dratio == 1 ? r : r / a.dratio;
    const Tin* __restrict__ u = (const Tin*)a.u + b * a.u_bs + r * a.u_ds;
    const Tin* __restrict__ dt = (const Tin*)a.delta + b * a.d_bs + rd_ * a.d_ds;
    const Tin* __restrict__ Bm = (const Tin*)a.B + b * a.B_bs + k * a.B_gs;
    const Tin* __restrict__ Cm = (const Tin*)a.C + b * a.C_bs + k * a.C_gs;
    Tout* __restrict__ out = (Tout*)a.out + b * a.o_bs + r * a.o_ds;
    const float A2 = a.A[r] * kLog2e;
    const float Dv = a.D ? a.D[r] : 0.f;
    const float bias = a.bias ? a.bias[rd_] : 0.f;
    const bool sp = a.softplus != 0;
    const int L = (int)a.seqlen;
    constexpr int OV = 16 / (int)sizeof(Tout);       // elements per 16-byte store
    const int ph = AL ? 0 : (int)((reinterpret_cast<uintptr_t>(out) / sizeof(Tout)) & (OV - 1));
    constexpr int ph_max = AL ? 0 : OV - 1;
    Inner in = {0, L};
    if constexpr (AL == 0)
        in = both(both(inner_of(u, L, a.span.u), inner_of(dt, L, a.span.delta), L), both(inner_of(Bm, L, a.span.B), inner_of(Cm, L, a.span.C), L), L);
    const int l0 = in.from, l1 = in.to;              // the elements of the walk
    Row8<Tin, AL> ru, rd, rb, rc;
    auto fetch = [&](int at) { ru.load(u, at, l0, l1); rd.load(dt, at, l0, l1); rb.load(Bm, at, l0, l1); rc.load(Cm, at, l0, l1); };
    int pos = wi * WSTEP + lane * VEC - ph;
    fetch(pos);
    float hc = 0.f;                                  // state entering this step
    auto one_by_one = [&](int l, int to) {           // by all lanes of the row alike
        for (; l < to; ++l) {
            const float ul = to_f<Tin>(u[l]);
            float dl = to_f<Tin>(dt[l]) + bias;
            if (sp) dl = softplus_fast(dl);
            const bool writes = real && lane == 0 && wi == 0;
            if (a.ckpt && writes && l % a.every == 0) a.ckpt[row * a.nck + l / a.every] = hc;
            hc = fmaf(decay_fast(dl, A2), hc, dl * to_f<Tin>(Bm[l]) * ul);
            if (!a.states_only && writes) out[l] = from_f<Tout>(fmaf(Dv, ul, to_f<Tin>(Cm[l]) * hc));
        }
    };
    if constexpr (AL == 0) one_by_one(0, l0);
    // rows that share a warp may start at different phases and end at different elements: they take the same number of steps
    for (int base = LPR < 32 ? -ph_max : -ph, it = 0; base < (LPR < 32 ? L : l1); base += STEP, ++it) {
        float uv[VEC], dv[VEC], bv[VEC], cv[VEC], P[VEC], hl[VEC];
        ru.get(u, pos, l0, l1, uv); rd.get(dt, pos, l0, l1, dv); rb.get(Bm, pos, l0, l1, bv); rc.get(Cm, pos, l0, l1, cv);
        fetch(pos + STEP);
        float p = 1.f, h = 0.f;
        if constexpr (!kPacked) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                float dl = dv[i] + bias;
                if (sp) dl = softplus_fast(dl);
                if constexpr (AL == 0) dl = pos + i < l1 && pos + i >= l0 ? dl : 0.f;       // outside the row: a step of zero (below)
                const float aa = decay_fast(dl, A2);
                h = fmaf(aa, h, dl * bv[i] * uv[i]);
                p *= aa;
                P[i] = p; hl[i] = h;
            }
        } else {
#pragma unroll
            for (int i = 0; i < VEC; i += 2) {
                float2 dl = __fadd2_rn(make_float2(dv[i], dv[i + 1]), splat2(bias));
                if (sp) dl = softplus_fast2(dl);
                // outside the row: a step of zero leaves the state as it is (whole vectors are tested once below)
                if constexpr (AL != 8) {
                    dl.x = pos + (AL ? i / (AL ? AL : 1) * AL : i) < l1 && (AL || pos + i >= l0) ? dl.x : 0.f;
                    dl.y = pos + (AL ? (i + 1) / (AL ? AL : 1) * AL : i + 1) < l1 && (AL || pos + i + 1 >= l0) ? dl.y : 0.f;
                }
                const float2 t = __fmul2_rn(dl, splat2(A2));
                const float2 aa = make_float2(ex2_approx(t.x), ex2_approx(t.y));
                const float2 x = __fmul2_rn(__fmul2_rn(dl, make_float2(bv[i], bv[i + 1])), make_float2(uv[i], uv[i + 1]));
                h = fmaf(aa.x, h, x.x); p *= aa.x;
                P[i] = p; hl[i] = h;
                h = fmaf(aa.y, h, x.y); p *= aa.y;
                P[i + 1] = p; hl[i + 1] = h;
            }
        }
        float ia = p, ib = h;
        if constexpr (AL == 8) { const bool in = pos < L; ia = in ? p : 1.f; ib = in ? h : 0.f; }
        float hin;
        if constexpr (W == 1) {
            if (lane == 0) ib = fmaf(ia, hc, ib);
            scan_step_up<1, LPR>(ia, ib); scan_step_up<2, LPR>(ia, ib); scan_step_up<4, LPR>(ia, ib);
            if constexpr (LPR > 8) scan_step_up<8, LPR>(ia, ib);
            if constexpr (LPR > 16) scan_step_up<16, LPR>(ia, ib);
            hin = entering_state<false, LPR>(ib, hc);
            hc = __shfl_sync(0xffffffffu, ib, LPR - 1, LPR);
        } else {
            scan_step_up<1>(ia, ib); scan_step_up<2>(ia, ib); scan_step_up<4>(ia, ib); scan_step_up<8>(ia, ib); scan_step_up<16>(ia, ib);
            if (lane == 31) agg[it & 1][wi] = AB{ia, ib};
            float ea = __shfl_up_sync(0xffffffffu, ia, 1), eb = __shfl_up_sync(0xffffffffu, ib, 1);
            if (lane == 0) { ea = 1.f; eb = 0.f; }
            __syncthreads();        // the buffer of this step was last read two steps ago, in front of the barrier in between
            float hw = hc;
#pragma unroll
            for (int j = 0; j < W; ++j) {
                if (j == wi) hw = hc;
                const AB g = agg[it & 1][j];
                hc = fmaf(g.a, hc, g.b);
            }
            hin = fmaf(ea, hw, eb);
        }
        if (a.ckpt && real) {
            if constexpr (AL != 0) {
                if (pos < L && pos % a.every == 0) a.ckpt[row * a.nck + pos / a.every] = hin;
            } else {
#pragma unroll
                for (int i = 0; i < VEC; ++i)
                    if (pos + i >= l0 && pos + i < l1 && (pos + i) % a.every == 0)
                        a.ckpt[row * a.nck + (pos + i) / a.every] = i == 0 ? hin : fmaf(P[i > 0 ? i - 1 : 0], hin, hl[i > 0 ? i - 1 : 0]);
            }
        }
        if (!a.states_only && real) {
            float ov[VEC];
            if constexpr (!kPacked) {
#pragma unroll
                for (int i = 0; i < VEC; ++i) ov[i] = fmaf(Dv, uv[i], cv[i] * fmaf(P[i], hin, hl[i]));
            } else {
#pragma unroll
                for (int i = 0; i < VEC; i += 2) {
                    const float2 y = __ffma2_rn(splat2(Dv), make_float2(uv[i], uv[i + 1]),
                                                __fmul2_rn(make_float2(cv[i], cv[i + 1]),
                                                           __ffma2_rn(make_float2(P[i], P[i + 1]), splat2(hin), make_float2(hl[i], hl[i + 1]))));
                    ov[i] = y.x; ov[i + 1] = y.y;
                }
            }
            constexpr int SV = AL && AL < OV ? AL : OV;          // elements per store
#pragma unroll
            for (int j = 0; j < VEC; j += SV) {
                const int q = pos + j;
                if (AL != 0 ? q < L : (q >= l0 && q + SV <= l1)) {
                    float o[SV];
#pragma unroll
                    for (int e = 0; e < SV; ++e) o[e] = ov[j + e];
                    Vec<Tout, SV>::store(out + q, o);
                } else if (AL == 0) {
#pragma unroll
                    for (int e = 0; e < SV; ++e)
                        if (q + e >= l0 && q + e < l1) out[q + e] = from_f<Tout>(ov[j + e]);
                }
            }
        }
        pos += STEP;
    }
    if constexpr (AL == 0) one_by_one(max(l0, l1), L);
}

// d_state > 1: the carry of each state lives in shared memory (one slot per warp and state).
template <typename Tin, typename Tout, int VEC>
__global__ void __launch_bounds__(kWarpsPerCta * 32) selscan_fwd_nx_kernel(const ScanArgs a) {
    follow_previous();
    __shared__ float carry_s[kWarpsPerCta][SS2D_MAX_DSTATE];
    __shared__ float A2_s[kWarpsPerCta][SS2D_MAX_DSTATE];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row = (int64_t)blockIdx.x * kWarpsPerCta + warp;
    if (row >= a.rows) return;
    const int64_t b = row / a.dim, r = row % a.dim, k = r / a.group_size;
    const Tin* __restrict__ u = (const Tin*)a.u + b * a.u_bs + r * a.u_ds;
    const Tin* __restrict__ dt = (const Tin*)a.delta + b * a.d_bs + (r / a.dratio) * a.d_ds;
    const Tin* __restrict__ Bm = (const Tin*)a.B + b * a.B_bs + k * a.B_gs;
    const Tin* __restrict__ Cm = (const Tin*)a.C + b * a.C_bs + k * a.C_gs;
    Tout* __restrict__ out = (Tout*)a.out + b * a.o_bs + r * a.o_ds;
    const int N = (int)a.dstate;
    for (int n = lane; n < N; n += 32) {
        carry_s[warp][n] = 0.f;
        A2_s[warp][n] = a.A[r * N + n] * kLog2e;
    }
    __syncwarp();
    const bool has_D = a.D != nullptr;
    const float Dv = has_D ? a.D[r] : 0.f;
    const float bias = a.bias ? a.bias[r / a.dratio] : 0.f;
    const bool sp = a.softplus != 0;
    const int L = (int)a.seqlen;
    constexpr int STEP = 32 * VEC;
    using VI = Vec<Tin, VEC>;
    using VO = Vec<Tout, VEC>;

    for (int base = 0; base < L; base += STEP) {
        const int pos = base + lane * VEC;
        const bool in = pos < L;
        float uv[VEC], dl[VEC], du[VEC], y[VEC];
        if (in) { VI::load(u + pos, uv); VI::load(dt + pos, dl); }
        else {
#pragma unroll
            for (int i = 0; i < VEC; ++i) { uv[i] = 0.f; dl[i] = 0.f; }
        }
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            float d = dl[i] + bias;
            if (sp) d = softplus_fast(d);
            dl[i] = d; du[i] = d * uv[i];
            y[i] = has_D ? Dv * uv[i] : 0.f;
        }
        for (int n = 0; n < N; ++n) {
            float bv[VEC], cv[VEC], P[VEC], hl[VEC];
            if (in) { VI::load(Bm + n * a.B_ss + pos, bv); VI::load(Cm + n * a.C_ss + pos, cv); }
            else {
#pragma unroll
                for (int i = 0; i < VEC; ++i) { bv[i] = 0.f; cv[i] = 0.f; }
            }
            const float A2 = A2_s[warp][n];
            float p = 1.f, h = 0.f;
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                const float aa = decay_fast(dl[i], A2);
                h = fmaf(aa, h, du[i] * bv[i]);
                p *= aa;
                P[i] = p; hl[i] = h;
            }
            const AB inc = warp_scan_inclusive(AB{p, h}, lane);
            float ea = __shfl_up_sync(0xffffffffu, inc.a, 1);
            float eb = __shfl_up_sync(0xffffffffu, inc.b, 1);
            if (lane == 0) { ea = 1.f; eb = 0.f; }
            const float hc = carry_s[warp][n];
            const float hin = fmaf(ea, hc, eb);
            if (a.ckpt && pos % a.every == 0 && in) a.ckpt[(row * a.nck + pos / a.every) * N + n] = hin;
            __syncwarp();
            if (lane == 31) carry_s[warp][n] = fmaf(inc.a, hc, inc.b);
#pragma unroll
            for (int i = 0; i < VEC; ++i) y[i] = fmaf(cv[i], fmaf(P[i], hin, hl[i]), y[i]);
        }
        __syncwarp();
        if (in) VO::store(out + pos, y);
    }
}

// d_state 1: warps per row.  One where the rows alone are 24 warps for each of 148 SMs; fewer rows get more, as long as a step of
// all warps but half is shorter than the row.  The rule counts warps, not the CTAs that are resident at once (aligned rows: 4, 8
// and 16 CTAs per SM of eight, four and two warps; unaligned ones 2, 5 and 10), because long rows gain from more warps in a
// second wave too.  us with 1 / 2 / 4 / 8 warps, bf16, the rule's in brackets:
//   rows    L = 3 136 (aligned)        L = 3 137                  L = 16 385
//   256      7.2   6.5   6.2  [7.3]    11.7   8.0   6.7  [6.2]    47.3  27.3  18.1 [16.1]
//   740      8.6   7.3   6.3  [6.9]    13.7  11.3  10.8 [13.7]    55.2  38.4  31.2 [38.6]
//   1 024    8.6   8.5  [8.1]  8.9     13.6  13.3 [14.2] 17.8     59.2  47.2 [44.6] 54.1
//   1 536    9.9  11.2 [11.6] 13.0     16.7  19.2 [20.4] 26.7     70.4  74.1 [66.5] 81.9
//   2 048   11.8 [12.8] 14.4  16.5     20.4 [21.3] 24.9  33.6     85.2 [81.0] 80.9 103.7
//   3 072   16.1 [18.6] 20.4  24.1     30.2 [31.0] 36.1  49.5      134 [121]  119   153
//   3 584  [18.2] 21.4  23.8  28.1    [33.6] 35.3  42.0  57.6     [146]  136   139   179
// It is within 7 % of the best for rows of 16 385 and for 2 048 rows and more of 3 137, but where CTAs of eight warps do not fit at once (444 to 740
// rows, up to 27 %); it gives a warp too many to 256 rows of 3 136 (18 %) and from 1 536 rows of about 3 100 on (up to 22 %).
static int n1_warps(int64_t rows, int64_t L) {
    int w = 1;
    while (w < 8 && rows * w < 148 * 24 && (int64_t)w * 256 < L) w *= 2;
    return w;
}

template <typename Tin, typename Tout, int AL>
static int launch_n1(const ScanArgs& a, cudaStream_t st) {
    const int w = n1_warps(a.rows, a.seqlen), lpr = w > 1 ? 32 : a.seqlen <= 64 ? 8 : a.seqlen <= 128 ? 16 : 32;
    const int64_t per_cta = kWarpsPerCta * (32 / lpr), ctas = w == 1 ? (a.rows + per_cta - 1) / per_cta : a.rows;
    if (ctas > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
    const unsigned g = (unsigned)ctas;
    if (w == 8) launch(selscan_fwd_n1_kernel<Tin, Tout, AL, 8, 32>, g, 256, 0, st, a);
    else if (w == 4) launch(selscan_fwd_n1_kernel<Tin, Tout, AL, 4, 32>, g, 128, 0, st, a);
    else if (w == 2) launch(selscan_fwd_n1_kernel<Tin, Tout, AL, 2, 32>, g, 64, 0, st, a);
    else if (lpr == 8) launch(selscan_fwd_n1_kernel<Tin, Tout, AL, 1, 8>, g, kWarpsPerCta * 32, 0, st, a);
    else if (lpr == 16) launch(selscan_fwd_n1_kernel<Tin, Tout, AL, 1, 16>, g, kWarpsPerCta * 32, 0, st, a);
    else launch(selscan_fwd_n1_kernel<Tin, Tout, AL, 1, 32>, g, kWarpsPerCta * 32, 0, st, a);
    count_launch();
    return check_launch();
}

template <typename Tin, typename Tout, int VEC>
static int launch_nx(const ScanArgs& a, cudaStream_t st) {
    const int64_t ctas = (a.rows + kWarpsPerCta - 1) / kWarpsPerCta;
    if (ctas > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
    launch(selscan_fwd_nx_kernel<Tin, Tout, VEC>, (unsigned)ctas, kWarpsPerCta * 32, 0, st, a);
    count_launch();
    return check_launch();
}

// `vec`: widest vector, in elements and at most 8, that every row start of every tensor allows
template <typename Tin, typename Tout>
static int dispatch_vec(const ScanArgs& a, int vec, cudaStream_t st) {
    if (a.dstate == 1)
        return vec >= 8   ? launch_n1<Tin, Tout, 8>(a, st)
               : vec >= 4 ? launch_n1<Tin, Tout, 4>(a, st)
               : vec >= 2 && sizeof(Tin) == 4 ? launch_n1<Tin, Tout, sizeof(Tin) == 4 ? 2 : 0>(a, st)
                          : launch_n1<Tin, Tout, 0>(a, st);
    if constexpr (sizeof(Tin) == 2) {
        if (vec >= 8) return launch_nx<Tin, Tout, 8>(a, st);
    }
    if (vec >= 4) return launch_nx<Tin, Tout, 4>(a, st);
    if (vec >= 2) return launch_nx<Tin, Tout, 2>(a, st);
    return launch_nx<Tin, Tout, 1>(a, st);
}

// largest power of two v <= cap such that every listed quantity is a multiple of v
static int common_pow2(std::initializer_list<int64_t> xs, int cap) {
    int v = cap;
    for (int64_t x : xs) {
        if (x < 0) x = -x;
        while (v > 1 && (x % v) != 0) v >>= 1;
    }
    return v;
}

// What the kernels of scan_states.cuh take: 2 .. 16 states, a row of step sizes per row.
static bool st_states(const ss2d_scan_params* p) { return p->dstate >= 2 && p->dstate <= 16 && p->delta_ratio <= 1; }

static int validate_fwd(const ss2d_scan_params* p) {
    if (!p) return SS2D_EINVAL_NULL;
    if (!p->u || !p->delta || !p->A || !p->B || !p->C || !p->out) return SS2D_EINVAL_NULL;
    if (!dtype_ok(p->in_dtype) || !dtype_ok(p->out_dtype)) return SS2D_EINVAL_DTYPE;
    if (p->out_dtype != SS2D_F32 && p->out_dtype != p->in_dtype) return SS2D_EINVAL_DTYPE;
    if (p->batch <= 0 || p->dim <= 0 || p->dstate <= 0 || p->seqlen <= 0 || p->n_groups <= 0) return SS2D_EINVAL_SHAPE;
    if (p->dstate > SS2D_MAX_DSTATE) return SS2D_ENOTSUP;
    if (p->dim % p->n_groups != 0) return SS2D_EINVAL_SHAPE;
    if (p->delta_ratio < 0 || (p->delta_ratio > 1 && p->dim % p->delta_ratio != 0)) return SS2D_EINVAL_SHAPE;
    if (p->seqlen > 0x3fffffffLL) return SS2D_ENOTSUP;
    const int64_t L = p->seqlen;
    // rows must not overlap: |stride| >= extent of what it steps over
    if (p->u_dim_stride < L || p->delta_dim_stride < L || p->out_dim_stride < L) return SS2D_EINVAL_STRIDE;
    if (p->B_state_stride < L || p->C_state_stride < L) return SS2D_EINVAL_STRIDE;
    if (p->batch > 1 && (p->u_batch_stride < L || p->delta_batch_stride < L || p->out_batch_stride < L ||
                         p->B_batch_stride < L || p->C_batch_stride < L)) return SS2D_EINVAL_STRIDE;
    if (p->n_groups > 1 && (p->B_group_stride < L || p->C_group_stride < L)) return SS2D_EINVAL_STRIDE;
    const size_t si = dtype_size(p->in_dtype), so = dtype_size(p->out_dtype);
    if (!aligned_to(p->u, si) || !aligned_to(p->delta, si) || !aligned_to(p->B, si) || !aligned_to(p->C, si) ||
        !aligned_to(p->out, so) || !aligned_to(p->checkpoints, 4) || !aligned_to(p->A, 4) || !aligned_to(p->D, 4) || !aligned_to(p->delta_bias, 4))
        return SS2D_EINVAL_ALIGN;

    if (p->states_only && (!p->checkpoints || (p->dstate != 1 && !st_states(p)))) return SS2D_ENOTSUP;
    if (p->checkpoints && p->checkpoint_every < 0) return SS2D_EINVAL_SHAPE;
    if (p->checkpoint_every % (p->dstate == 1 ? 8 : st_states(p) ? 32 : 128) != 0) return SS2D_EINVAL_SHAPE;
    return SS2D_OK;
}

// Widest vector (in elements, at most 8) that keeps every row start aligned for every tensor.
static int fwd_vec(const ss2d_scan_params* p) {
    const size_t si = dtype_size(p->in_dtype), so = dtype_size(p->out_dtype);
    auto ptr_el = [](const void* q, size_t s) { return (int64_t)(reinterpret_cast<uintptr_t>(q) / s); };
    return common_pow2({p->seqlen, p->u_batch_stride, p->u_dim_stride, p->delta_batch_stride, p->delta_dim_stride, p->out_batch_stride,
                        p->out_dim_stride, p->B_batch_stride, p->B_group_stride, p->B_state_stride, p->C_batch_stride, p->C_group_stride,
                        p->C_state_stride, ptr_el(p->u, si), ptr_el(p->delta, si), ptr_el(p->B, si), ptr_el(p->C, si), ptr_el(p->out, so)}, 8);
}

// Vector width of the 2 .. 16 state kernels: 8, 4, 1, or 0 for pieces (st_dispatch_fwd).
static int states_vw(const ss2d_scan_params* p) {
    const int v = fwd_vec(p);
    if (v >= 4) return v >= 8 ? 8 : 4;
    const ScanSpans s = scan_spans(*p, dtype_size(p->in_dtype));
    const bool pieces = whole_pieces(s.u) && whole_pieces(s.delta) && whole_pieces(s.B) && whole_pieces(s.C);
    return pieces && st_takes_pieces(dtype_size(p->in_dtype), st_pad_states(p->dstate)) ? 0 : 1;
}

// How the rows of a 2 .. 16 state problem are cut, and the floats that the segments' end states and sums take.  The number of segments depends on
// where the tensors lie (`resident`, st_segments); the workspace that callers are asked for is of the larger number, so that one
// of this shape serves tensors of any alignment.
static StSegments fwd_segments(const ss2d_scan_params* p, bool resident) {
    return st_segments(p->batch * p->n_groups * st_parts(p->dim / p->n_groups) * (st_pad_states(p->dstate) / 4), p->seqlen, resident);
}
static int64_t segment_floats(const ss2d_scan_params* p, StSegments s) {
    return s.count > 1 ? p->batch * p->dim * s.count * (st_pad_states(p->dstate) + 1) : 0;
}

long long selective_scan_checkpoint_every(int64_t dstate, int64_t delta_ratio) {
    return dstate == 1 ? 8 : dstate >= 2 && dstate <= 16 && delta_ratio <= 1 ? 32 : 128;
}

long long selective_scan_fwd_workspace_bytes(const ss2d_scan_params* p) {
    if (validate_fwd(p) != SS2D_OK) return -1;
    if (!st_states(p)) return 0;
    return (long long)segment_floats(p, fwd_segments(p, false)) * 4;
}

template <typename Tin, typename Tout>
static int states_fwd(StFwdArgs& a, const ss2d_scan_params* p, int vw, cudaStream_t st) {
    if (a.S > 1) {
        a.fold = 0;
        float* ck = a.ckpt;
        a.ckpt = nullptr;
        const int rc = st_dispatch_fwd<Tin, Tin, false>(a, p->batch, vw, st);
        if (rc != SS2D_OK) return rc;
        a.ckpt = ck;
        a.fold = 1;
    }
    return p->states_only ? st_dispatch_fwd<Tin, Tin, false>(a, p->batch, vw, st) : st_dispatch_fwd<Tin, Tout, true>(a, p->batch, vw, st);
}

static int selective_scan_states(const ss2d_scan_params* p, cudaStream_t st) {
    StFwdArgs a = {};
    a.u = p->u; a.delta = p->delta; a.B = p->B; a.C = p->C; a.out = p->out;
    a.A = (const float*)p->A; a.D = (const float*)p->D; a.bias = (const float*)p->delta_bias;
    a.dim = p->dim; a.group_size = p->dim / p->n_groups;
    a.u_bs = p->u_batch_stride; a.u_ds = p->u_dim_stride; a.d_bs = p->delta_batch_stride; a.d_ds = p->delta_dim_stride;
    a.o_bs = p->out_batch_stride; a.o_ds = p->out_dim_stride;
    a.B_bs = p->B_batch_stride; a.B_gs = p->B_group_stride; a.B_ss = p->B_state_stride;
    a.C_bs = p->C_batch_stride; a.C_gs = p->C_group_stride; a.C_ss = p->C_state_stride;
    a.L = (int)p->seqlen; a.N = (int)p->dstate; a.n_groups = (int)p->n_groups; a.softplus = p->delta_softplus;
    a.parts = st_parts(a.group_size);
    a.every = p->checkpoint_every ? (int)p->checkpoint_every : 128;
    a.ckpt = (float*)p->checkpoints; a.nck = (p->seqlen + a.every - 1) / a.every;
    const int vw = states_vw(p);
    StSegments s = fwd_segments(p, vw != 0);
    int64_t floats = segment_floats(p, s);
    if (floats && (!p->workspace || p->workspace_bytes < floats * 4)) { s = {1, (a.L + 63) / 64 * 64}; floats = 0; }   // uncut: slower, same result
    if (floats && !aligned_to(p->workspace, 16)) return SS2D_EINVAL_ALIGN;
    a.S = s.count; a.seg_len = s.len;
    a.ends = floats ? (float*)p->workspace : nullptr;
    a.sums = floats ? a.ends + p->batch * p->dim * s.count * st_pad_states(p->dstate) : nullptr;
    const bool of32 = p->out_dtype == SS2D_F32;
    if (p->in_dtype == SS2D_F32) return states_fwd<float, float>(a, p, vw, st);
    if (p->in_dtype == SS2D_BF16) return of32 ? states_fwd<__nv_bfloat16, float>(a, p, vw, st) : states_fwd<__nv_bfloat16, __nv_bfloat16>(a, p, vw, st);
    return of32 ? states_fwd<__half, float>(a, p, vw, st) : states_fwd<__half, __half>(a, p, vw, st);
}

int selective_scan_fwd(const ss2d_scan_params* p, cudaStream_t st) {
    const int rc = validate_fwd(p);
    if (rc != SS2D_OK) return rc;
    if (st_states(p)) return selective_scan_states(p, st);
    const int64_t L = p->seqlen;
    ScanArgs a;
    a.u = p->u; a.delta = p->delta; a.B = p->B; a.C = p->C;
    a.A = (const float*)p->A; a.D = (const float*)p->D; a.bias = (const float*)p->delta_bias;
    a.out = p->out;
    a.rows = p->batch * p->dim; a.dim = p->dim; a.dstate = p->dstate; a.seqlen = L;
    a.group_size = p->dim / p->n_groups;
    a.u_bs = p->u_batch_stride; a.u_ds = p->u_dim_stride;
    a.d_bs = p->delta_batch_stride; a.d_ds = p->delta_dim_stride;
    a.o_bs = p->out_batch_stride; a.o_ds = p->out_dim_stride;
    a.B_bs = p->B_batch_stride; a.B_gs = p->B_group_stride; a.B_ss = p->B_state_stride;
    a.C_bs = p->C_batch_stride; a.C_gs = p->C_group_stride; a.C_ss = p->C_state_stride;
    a.span = scan_spans(*p, dtype_size(p->in_dtype));
    a.softplus = p->delta_softplus;
    a.dratio = p->delta_ratio > 1 ? p->delta_ratio : 1;
    a.ckpt = (float*)p->checkpoints;

    a.every = p->checkpoint_every ? (int)p->checkpoint_every : 128;
    a.nck = (L + a.every - 1) / a.every;
    a.states_only = p->states_only != 0;
    const int vec = fwd_vec(p);

    const int in = p->in_dtype;
    const bool of32 = p->out_dtype == SS2D_F32;
    if (in == SS2D_F32) return dispatch_vec<float, float>(a, vec, st);
    if (in == SS2D_BF16)
        return of32 ? dispatch_vec<__nv_bfloat16, float>(a, vec, st) : dispatch_vec<__nv_bfloat16, __nv_bfloat16>(a, vec, st);
    return of32 ? dispatch_vec<__half, float>(a, vec, st) : dispatch_vec<__half, __half>(a, vec, st);
}

}  // namespace ss2d
