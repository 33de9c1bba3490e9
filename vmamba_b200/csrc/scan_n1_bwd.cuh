// Selective-scan backward for one state (every VMamba backbone).
//
// A lane holds eight consecutive elements of a row, a warp a chunk of 256; the rows of an (image, group) are dealt to the
// warps of a CTA, R rows to each, and all of them walk their row from its end, chunk by chunk.  The state in front of
// every eighth element comes from the forward pass (half a byte per element, against the twelve to twenty that the pass moves
// anyway), so that the only scan of a chunk is the one of the reverse recurrence e_l = a_l (C_l g_l + e_{l+1}).  The dB / dC
// terms of a warp's R rows meet in registers and those of the CTA's warps in shared memory (double-buffered: one
// barrier per chunk); what crosses CTAs goes to an fp32 workspace and is folded in a fixed order.
//
// Segments: where the rows do not fill the chip they are cut into S segments; a first kernel leaves each segment's
// effect on e (its value from zero, and the sum of its step sizes), and a segment starts from the fold of those behind it.
//
// Bound: latency at three CTAs of four warps per SM (153 to 168 registers).  32 x 384 rows of 3 136 elements, bf16, 138 us (150 with the
// addresses of every row formed from its number): an SM issues in half of its cycles with 2.5 warps per scheduler, and of a warp's five
// cycles per instruction 1.4 wait for the one before it, 0.7 for shuffles and exponentials and 0.5 for memory; the bytes are 74 us at the copy
// rate.  Not faster: four elements per lane and twice the warps (190), rows through shared memory three deep (135; fp32 174 -> 228).
#pragma once
#include "scan_row.cuh"

namespace ss2d {

constexpr int kN1Warps = 4, kN1Chunk = 256, kN1MaxR = 8;

struct N1BwdArgs {
    const void *u, *delta, *B, *C, *dout;
    const float *A, *D, *bias;
    void *du, *ddelta;
    float* rowred;          // (segment, image, row, 3): dA, dD, dbias
    float* bcpart;          // (image, group, part, 2, Lp)
    const float* ckpt;      // (rows, ceil(L / 8)): the state in front of every eighth element
    float *eagg, *esum;     // (rows, S) each; null with S = 1
    int64_t dim, group_size, batch, dratio;
    int64_t u_bs, u_ds, d_bs, d_ds, g_bs, g_ds, B_bs, B_gs, C_bs, C_gs;
    int L, Lp, n_groups, parts, R, S, seg_len, softplus;
};

template <typename T, int AL>
__device__ __forceinline__ void row8_pairs(const Row8<T, AL>& w, const T* row, int pos, int L, float2 (&v)[4]) {
    float x[8];
    w.get(row, pos, 0, L, x);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = make_float2(x[2 * i], x[2 * i + 1]);
}
template <typename T, int AL, int LPR>
__device__ __forceinline__ void row8_store(T* row, int pos, int L, const float2 (&v)[4], float* stage, int lane) {
    const float x[8] = {v[0].x, v[0].y, v[1].x, v[1].y, v[2].x, v[2].y, v[3].x, v[3].y};
    if constexpr (AL != 0) {
#pragma unroll
        for (int j = 0; j < 8 / AL; ++j)
            if (pos + j * AL < L) {
                float y[AL];
#pragma unroll
                for (int e = 0; e < AL; ++e) y[e] = x[j * AL + e];
                Vec<T, AL>::store(row + pos + j * AL, y);
            }
    } else {
        // through the warp's 8 x 33 floats, so that neighbouring lanes write neighbouring elements
        const int ln = lane & (LPR - 1), c0 = pos - ln * 8, first = lane - ln;      // first lane of the row
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 8; ++e) stage[e * 33 + lane] = x[e];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int el = j * LPR + ln;
            if (c0 + el < L) row[c0 + el] = from_f<T>(stage[(el & 7) * 33 + first + (el >> 3)]);
        }
    }
}

__device__ __forceinline__ float2 pk(float x) { return make_float2(x, x); }

// Step size and its derivative with respect to the raw value, for a pair.  Above torch's threshold of 20 the step size is the
// raw value and the derivative 1 (to fp32 rounding: 1 - 2e-9).
__device__ __forceinline__ void softplus_pair(float2 x, float2& sp, float2& dsp) {
    const float2 xm = make_float2(fminf(x.x, 20.f), fminf(x.y, 20.f));
    const float2 t = __fmul2_rn(xm, pk(kLog2e));
    const float2 e = make_float2(ex2_approx(t.x), ex2_approx(t.y));
    const float2 w = __fadd2_rn(e, pk(1.f));
    const float2 series = __fmul2_rn(e, __ffma2_rn(e, __ffma2_rn(e, pk(0.33333334f), pk(-0.5f)), pk(1.f)));
    const float2 full = __fmul2_rn(make_float2(lg2_approx(w.x), lg2_approx(w.y)), pk(kLn2));
    float2 r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(w.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(w.y));
    dsp = __fmul2_rn(e, r);
    const float2 s = make_float2(e.x < 0.015625f ? series.x : full.x, e.y < 0.015625f ? series.y : full.y);
    sp = __fadd2_rn(s, __ffma2_rn(xm, pk(-1.f), x));
}

// LPR: lanes per row.  Rows of at most 128 (64) elements share a warp, two (four) at a time.
// BC: vectors of B and C; AL, or 1 with AL 0 where they do not start and end on 16-byte boundaries.  (32 x 384 rows of 3 137 elements,
// bf16, all gradients: 245 us with pieces; single elements cost 9 %, the choice inside one kernel 4 %.)
template <typename Tin, typename Tg, int AL, int LPR, int BC>
__global__ void __launch_bounds__(kN1Warps * 32, 3) n1_bwd_kernel(const N1BwdArgs a) {
    follow_previous();
    extern __shared__ __align__(16) float n1_sm[];
    constexpr int G = 32 / LPR, kChunk = LPR * 8, kStep = kN1Warps * G;     // kStep: rows of the CTA that are worked on at a time
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, R = a.R, L = a.L, ln = lane & (LPR - 1), wr = warp * G + lane / LPR;
    float* red = n1_sm;                                          // [2][warp][2][256]
    float4* par = reinterpret_cast<float4*>(red + 2 * kN1Warps * 2 * kChunk);   // [row of the CTA]: A, bias, D, e behind the chunk
    float* racc = reinterpret_cast<float*>(par + kStep * R);     // [warp's row set][3][32]: per-lane sums of dA, dD, dbias
    float* stage = racc + kN1Warps * R * 96 + warp * 264;        // AL = 0: the warp's way out
    int cta = blockIdx.x;
    const int seg = cta % a.S; cta /= a.S;
    const int part = cta % a.parts; cta /= a.parts;
    const int k = cta % a.n_groups;
    const int64_t b = cta / a.n_groups;
    const int first = part * kStep * R + wr;                     // this lane's rows of the group: first + i * kStep
    const int gs = (int)a.group_size;
    const int lo = seg * a.seg_len, hi = min(L, lo + a.seg_len);
    const Tin* __restrict__ u = (const Tin*)a.u + b * a.u_bs;
    const Tin* __restrict__ dt = (const Tin*)a.delta + b * a.d_bs;
    const Tg* __restrict__ gp = (const Tg*)a.dout + b * a.g_bs;
    const Tin* __restrict__ Bm = (const Tin*)a.B + b * a.B_bs + k * a.B_gs;
    const Tin* __restrict__ Cm = (const Tin*)a.C + b * a.C_bs + k * a.C_gs;
    const int64_t out0 = b * a.dim;
    const int nck = (L + 7) / 8;
    const bool sp = a.softplus != 0;

    for (int i = 0; i < R; ++i) {
        const int ig = first + i * kStep;
#pragma unroll
        for (int j = 0; j < 3; ++j) racc[((i * kN1Warps + warp) * 3 + j) * 32 + lane] = 0.f;
        if (ln == 0) {                                           // spare lanes of a shared warp: the group's last row
            const int64_t r = (int64_t)k * gs + min(ig, gs - 1);
            const float An = a.A[r];
            float e = 0.f;
            for (int j = a.S - 1; j > seg; --j)                  // what the segments behind leave
                e = fmaf(ex2_approx(a.esum[(out0 + r) * a.S + j] * An * kLog2e), e, a.eagg[(out0 + r) * a.S + j]);
            par[i * kStep + wr] = make_float4(An, a.bias ? a.bias[a.dratio == 1 ? r : r / a.dratio] : 0.f, a.D ? a.D[r] : 0.f, e);
        }
    }
    __syncwarp();

    // The rows of a set.  The next one's lie a fixed step behind, but for shared warps (their last set) and shared step sizes.  Stepping saves the
    // products of row number and stride, but holds ten registers: fp32 vectors (160 -> 163 us at 1 x 1 024 x 16 384) and pieces of 16-bit rows
    // (243 -> 247 at 32 x 384 x 3 137) are at their limit.
    constexpr bool kStepped = (AL != 0) == (sizeof(Tin) == 2);
    struct Rows { const Tin *u, *d; const Tg* g; const float* ck; int64_t out; };
    auto rows_of = [&](int i) {
        const int64_t r = (int64_t)k * gs + min(first + i * kStep, gs - 1);
        return Rows{u + r * a.u_ds, dt + (a.dratio == 1 ? r : r / a.dratio) * a.d_ds, gp + r * a.g_ds, a.ckpt + (out0 + r) * nck, (out0 + r) * L};
    };
    auto advance = [&](Rows& w, int i) {
        if (!kStepped || G > 1 || a.dratio != 1) w = rows_of(i);
        else { w.u += kStep * a.u_ds; w.d += kStep * a.d_ds; w.g += kStep * a.g_ds; w.ck += kStep * nck; w.out += (int64_t)kStep * L; }
    };
    Row8<Tin, AL> nu, nd;
    Row8<Tg, AL> ng;
    float nh = 0.f;
    auto fetch = [&](const Rows& w, int pos) {
        nu.load(w.u, pos, 0, L); nd.load(w.d, pos, 0, L); ng.load(w.g, pos, 0, L);
        nh = pos < L ? w.ck[pos >> 3] : 0.f;
    };
    int buf = 0;
    const int first_w = first - lane / LPR, mine = first_w < gs ? min(R, (gs - first_w + kStep - 1) / kStep) : 0;     // row sets of this warp
    const Rows row0 = rows_of(0);
    for (int c = (hi - 1) / kChunk; c * kChunk >= lo; --c, buf ^= 1) {
        const int pos = c * kChunk + ln * 8;
        float2 bv[4], cv[4], accB[4], accC[4];
        Rows row = row0;
        if (mine) fetch(row, pos);
        {
            Row8<Tin, BC> rb, rc;
            rb.load(Bm, pos, 0, L); rc.load(Cm, pos, 0, L);
            row8_pairs(rb, Bm, pos, L, bv); row8_pairs(rc, Cm, pos, L, cv);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) accB[i] = accC[i] = pk(0.f);
#pragma unroll 1
        for (int i = 0; i < mine; ++i) {
            float2 uv[4], d[4], g[4];
            row8_pairs(nu, row.u, pos, L, uv); row8_pairs(nd, row.d, pos, L, d); row8_pairs(ng, row.g, pos, L, g);
            float h = nh;
            const int64_t out = row.out;
            if (i + 1 < mine) { advance(row, i + 1); fetch(row, pos); }
            const float4 pr = par[i * kStep + wr];
            const float An = pr.x;
            const bool real = G == 1 || first + i * kStep < gs;   // spare lanes repeat the last row and take part in nothing
            if (!real) {
#pragma unroll
                for (int j = 0; j < 4; ++j) uv[j] = g[j] = pk(0.f);
            }
            float2 dsp[4], av[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 x = __fadd2_rn(d[j], pk(pr.y));
                if (sp) softplus_pair(x, d[j], dsp[j]);
                else { d[j] = x; dsp[j] = pk(1.f); }
            }
            if (pos + 8 > L) {                                   // beyond the row: a step of zero, which takes part in nothing
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (pos + 2 * j >= L) { d[j].x = 0.f; dsp[j].x = 0.f; }
                    if (pos + 2 * j + 1 >= L) { d[j].y = 0.f; dsp[j].y = 0.f; }
                }
            }
            float2 hp[4], cg[4], dhv[4], bu[4];                  // hp: state in front of the element
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 t = __fmul2_rn(d[j], pk(An * kLog2e));
                av[j] = make_float2(ex2_approx(t.x), ex2_approx(t.y));
                bu[j] = __fmul2_rn(bv[j], uv[j]);
                cg[j] = __fmul2_rn(cv[j], g[j]);
                const float2 in = __fmul2_rn(d[j], bu[j]);
                hp[j].x = h;
                h = fmaf(av[j].x, h, in.x);
                accC[j].x = fmaf(g[j].x, h, accC[j].x);
                hp[j].y = h;
                h = fmaf(av[j].y, h, in.y);
                accC[j].y = fmaf(g[j].y, h, accC[j].y);
            }
            // the reverse recurrence: the lane's part from zero, the scan over the lanes, then again from what enters
            float2 pp = __fmul2_rn(__fmul2_rn(av[0], av[1]), __fmul2_rn(av[2], av[3]));
            float p = pp.x * pp.y, e = 0.f;
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                const float2 t = __fmul2_rn(av[j], cg[j]);
                e = fmaf(av[j].y, e, t.y);
                e = fmaf(av[j].x, e, t.x);
            }
            if (ln == LPR - 1) e = fmaf(p, pr.w, e);
            scan_step_down<1, LPR>(p, e); scan_step_down<2, LPR>(p, e); scan_step_down<4, LPR>(p, e);
            if constexpr (LPR > 8) scan_step_down<8, LPR>(p, e);
            if constexpr (LPR > 16) scan_step_down<16, LPR>(p, e);
            float en = entering_state<true, LPR>(e, pr.w);
            if (ln == 0) par[i * kStep + wr].w = e;
            float2 dA = pk(0.f), dD = pk(0.f), db = pk(0.f), duo[4], ddo[4];
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                float2 ev;
                dhv[j].y = cg[j].y + en;
                en = av[j].y * dhv[j].y; ev.y = en;
                dhv[j].x = cg[j].x + en;
                en = av[j].x * dhv[j].x; ev.x = en;
                const float2 x = __fmul2_rn(ev, hp[j]);          // dh a h_prev
                const float2 dhd = __fmul2_rn(dhv[j], d[j]);
                accB[j] = __ffma2_rn(dhd, uv[j], accB[j]);
                duo[j] = __ffma2_rn(dhd, bv[j], __fmul2_rn(g[j], pk(pr.z)));
                ddo[j] = __fmul2_rn(__ffma2_rn(pk(An), x, __fmul2_rn(dhv[j], bu[j])), dsp[j]);
                dA = __ffma2_rn(d[j], x, dA);
                dD = __ffma2_rn(g[j], uv[j], dD);
                db = __fadd2_rn(db, ddo[j]);
            }
            float* q = racc + (i * kN1Warps + warp) * 96 + lane;
            q[0] += dA.x + dA.y; q[32] += dD.x + dD.y; q[64] += db.x + db.y;
            row8_store<Tin, AL, LPR>((Tin*)a.du + out, pos, real ? L : 0, duo, stage, lane);
            row8_store<Tin, AL, LPR>((Tin*)a.ddelta + out, pos, real ? L : 0, ddo, stage, lane);
        }
        if constexpr (G > 1) {                                   // the rows that share the warp
#pragma unroll
            for (int off = LPR; off < 32; off <<= 1)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    accB[j].x += __shfl_xor_sync(0xffffffffu, accB[j].x, off); accB[j].y += __shfl_xor_sync(0xffffffffu, accB[j].y, off);
                    accC[j].x += __shfl_xor_sync(0xffffffffu, accC[j].x, off); accC[j].y += __shfl_xor_sync(0xffffffffu, accC[j].y, off);
                }
        }
        if (lane < LPR) {
            float4* my = reinterpret_cast<float4*>(red + ((buf * kN1Warps + warp) * 2) * kChunk + ln * 8);
            my[0] = make_float4(accB[0].x, accB[0].y, accB[1].x, accB[1].y);
            my[1] = make_float4(accB[2].x, accB[2].y, accB[3].x, accB[3].y);
            my[kChunk / 4] = make_float4(accC[0].x, accC[0].y, accC[1].x, accC[1].y);
            my[kChunk / 4 + 1] = make_float4(accC[2].x, accC[2].y, accC[3].x, accC[3].y);
        }
        __syncthreads();
        float* bc_out = a.bcpart + (((int64_t)b * a.n_groups + k) * a.parts + part) * 2 * (int64_t)a.Lp + c * kChunk;
        for (int i = threadIdx.x; i < 2 * kChunk / 4; i += kN1Warps * 32) {
            const float4* s = reinterpret_cast<const float4*>(red + buf * kN1Warps * 2 * kChunk) + i;
            float4 t = s[0];
#pragma unroll
            for (int w = 1; w < kN1Warps; ++w) {
                const float4 v = s[w * 2 * kChunk / 4];
                t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
            }
            const int which = i / (kChunk / 4), el = (i - which * (kChunk / 4)) * 4;
            if (c * kChunk + el < a.Lp) *reinterpret_cast<float4*>(bc_out + (int64_t)which * a.Lp + el) = t;
        }
    }
    for (int i = 0; i < mine; ++i) {
        float v[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            v[j] = racc[((i * kN1Warps + warp) * 3 + j) * 32 + lane];
#pragma unroll
            for (int off = LPR / 2; off > 0; off >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], off);
        }
        if (ln == 0 && first + i * kStep < gs) {
            float* rr = a.rowred + (((int64_t)seg * a.batch + b) * a.dim + (int64_t)k * gs + first + i * kStep) * 3;
            rr[0] = v[0]; rr[1] = v[1]; rr[2] = v[2];
        }
    }
}

// What a segment does to e: a warp per (row, segment), chunks of 256 elements from the segment's end.
template <typename Tin, typename Tg, int AL, int BC>
__global__ void __launch_bounds__(kN1Warps * 32) n1_bwd_segments_kernel(const N1BwdArgs a) {
    follow_previous();
    const int lane = threadIdx.x & 31, L = a.L;
    const int64_t w = (int64_t)blockIdx.x * kN1Warps + (threadIdx.x >> 5);
    const int64_t row = w / (a.S - 1);
    const int seg = (int)(w - row * (a.S - 1)) + 1;              // nothing reads the first segment's
    if (row >= a.batch * a.dim) return;
    const int64_t b = row / a.dim, r = row - b * a.dim, k = r / a.group_size, rd = a.dratio == 1 ? r : r / a.dratio;
    const Tin* __restrict__ dt = (const Tin*)a.delta + b * a.d_bs + rd * a.d_ds;
    const Tg* __restrict__ gp = (const Tg*)a.dout + b * a.g_bs + r * a.g_ds;
    const Tin* __restrict__ Cm = (const Tin*)a.C + b * a.C_bs + k * a.C_gs;
    const float A2 = a.A[r] * kLog2e, bias = a.bias ? a.bias[rd] : 0.f;
    const int lo = seg * a.seg_len, hi = min(L, lo + a.seg_len);
    float e = 0.f, sum = 0.f;                                    // over the chunks taken so far
    for (int c = (hi - 1) / kN1Chunk; c * kN1Chunk >= lo; --c) {
        const int pos = c * kN1Chunk + lane * 8;
        float2 d[4], g[4], cv[4];
        {
            Row8<Tin, AL> xd;
            Row8<Tin, BC> xc;
            Row8<Tg, AL> xg;
            xd.load(dt, pos, 0, L); xg.load(gp, pos, 0, L); xc.load(Cm, pos, 0, L);
            row8_pairs(xd, dt, pos, L, d); row8_pairs(xg, gp, pos, L, g); row8_pairs(xc, Cm, pos, L, cv);
        }
        float le = 0.f, ls = 0.f;
#pragma unroll
        for (int j = 7; j >= 0; --j) {
            float x = (j & 1 ? d[j >> 1].y : d[j >> 1].x) + bias;
            if (a.softplus) x = softplus_fast(x);
            x = pos + j < L ? x : 0.f;
            ls += x;
            le = decay_fast(x, A2) * fmaf(j & 1 ? cv[j >> 1].y : cv[j >> 1].x, j & 1 ? g[j >> 1].y : g[j >> 1].x, le);
        }
        float p = decay_fast(ls, A2);
        if (lane == 31) le = fmaf(p, e, le);
        scan_step_down<1>(p, le); scan_step_down<2>(p, le); scan_step_down<4>(p, le); scan_step_down<8>(p, le); scan_step_down<16>(p, le);
        e = __shfl_sync(0xffffffffu, le, 0);
        sum += ls;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (lane == 0) { a.eagg[row * a.S + seg] = e; a.esum[row * a.S + seg] = sum; }
}

}  // namespace ss2d
