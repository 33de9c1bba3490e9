// Selective-scan forward for 2 .. 16 states (layout: scan_states.cuh).  One kernel in two forms:
//   kOut          the result, and the states in front of every `every`-th element where the backward pass wants them;
//   !kOut         no result: the end states of every segment (the first of the two passes over rows cut into segments), or
//                 the states in front of every `every`-th element alone (a backward call without the forward's).
// Bound: latency with 2.6 warps per scheduler (384 CTAs on 592 places), then the write-back of the shared-memory reads (scan_states.cuh, R).
// 16 x 768 rows of 3 136 elements, 16 states, bf16, 294 us; of a warp's six cycles per instruction 1.5 wait for shared memory and
// exponentials and 1.4 for the instruction in front.  B and C of a group of elements are therefore read while the group in front is
// worked on, which the compiler undoes unless it may use the registers that so few warps leave (312 -> 294 us, fp32 385 -> 339; packing
// 16-bit B and C, which halves their reads but unpacks them, 306).  The exponentials, one per (element, state), are 132 us, DRAM is at 11 %.
// Per (element, state) a lane issues about 7 instructions: half of a packed multiply each for dl * A and du * B, half of a packed fma
// each for the state and the result, the exponential, and its share of the shared-memory reads, of the sum over the lanes of a
// row and of the staging.
#pragma once
#include "scan_states.cuh"

namespace ss2d {

struct StFwdArgs {
    const void *u, *delta, *B, *C;
    const float *A, *D, *bias;
    void* out;
    int64_t dim, group_size;
    int64_t u_bs, u_ds, d_bs, d_ds, o_bs, o_ds;
    int64_t B_bs, B_gs, B_ss, C_bs, C_gs, C_ss;
    int L, N, n_groups, parts, softplus;
    int S, seg_len;          // segments per row
    float *ends, *sums;      // (row, S, NS), (row, S): written by the first pass, read by the second; null with S = 1
    int fold;                // the second pass
    float* ckpt;             // (row, nck, N) or null
    int64_t nck;
    int every;               // a multiple of 32
};

// Registers for sixteen warps an SM; twelve with two rows per lane (49 152 rows, 16 states, fp32 1 142 against 1 062 us), unless !kHeld (st_launch_fwd).
template <typename Tin, typename Tout, int NS, int R_, int VW, bool kOut, bool kHeld>
__global__ void __launch_bounds__(StLayout<NS, R_>::kWarps * 32, !kHeld ? 0 : (R_ == 2 ? 12 : 16) / StLayout<NS, R_>::kWarps) st_fwd_kernel(const StFwdArgs a) {
    follow_previous();
    using Y = StLayout<NS, R_>;
    constexpr int RPW = Y::RPW, SL = Y::SL, R = Y::R, RL = Y::RL, P = kStPitch;
    constexpr int kRow = RPW * P, kBC = kStChunk * Y::BCP;
    using Raw = StRaw<Tin, RPW, VW>;
    constexpr bool kAhead = R == 1;                  // B and C of a group, too, are read in front of it
    constexpr bool kPre = sizeof(Raw) <= (VW == 0 ? 128 : 64);         // the next chunk is fetched into registers while this one is worked on
    extern __shared__ __align__(16) float st_sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rl = lane / SL, sl = lane % SL, n0 = sl * 4;
    float* sd = st_sm + warp * 2 * kRow;             // step sizes of the warp's chunk
    float* su = sd + kRow;                           // u, then the results
    float* sbc = st_sm + Y::kWarps * 2 * kRow;       // two buffers of B and C, shared by the CTA
    int cta = blockIdx.x;
    const int seg = cta % a.S; cta /= a.S;
    const int part = cta % a.parts; cta /= a.parts;
    const int k = cta % a.n_groups;
    const int64_t b = cta / a.n_groups;
    const int in_group = part * kStRows + warp * RPW;
    const int count = max(0, min(RPW, (int)a.group_size - in_group));
    const int64_t r0 = (int64_t)k * a.group_size + in_group;            // row inside the image
    const int L = a.L, lo = seg * a.seg_len, hi = min(L, lo + a.seg_len);
    const Tin* __restrict__ u = (const Tin*)a.u + b * a.u_bs + r0 * a.u_ds;
    const Tin* __restrict__ dt = (const Tin*)a.delta + b * a.d_bs + r0 * a.d_ds;
    const Tin* __restrict__ Bm = (const Tin*)a.B + b * a.B_bs + k * a.B_gs;
    const Tin* __restrict__ Cm = kOut ? (const Tin*)a.C + b * a.C_bs + k * a.C_gs : nullptr;
    const bool sp = a.softplus != 0;

    float2 A2[R][2], h[R][2];
    float Dv[R], bias[R], sum_d[R];
    int64_t row[R];                                  // over all images
    bool mine[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
        mine[j] = rl + j * RL < count;
        const int64_t r = mine[j] ? r0 + rl + j * RL : (int64_t)k * a.group_size;     // padding rows read a real row's parameters
        row[j] = b * a.dim + r;
        float t[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = n0 + i < a.N ? a.A[r * a.N + n0 + i] * kLog2e : 0.f;
        A2[j][0] = make_float2(t[0], t[1]); A2[j][1] = make_float2(t[2], t[3]);
        bias[j] = a.bias ? a.bias[r] : 0.f;
        Dv[j] = kOut && a.D && sl == 0 ? a.D[r] : 0.f;          // one lane of a row adds D u
        sum_d[j] = 0.f;
        if (a.fold) st_fold_segments<false>(h[j], A2[j], a.ends, a.sums, row[j], a.S, seg, n0, NS);
        else h[j][0] = h[j][1] = f2(0.f);
    }

    // ---- a chunk on its way in: global memory -> registers -> (step size, u; B, C) in shared memory
    Raw xu, xd;
    StRawBC<Tin, NS, VW, Y::kWarps> xb, xc;
    auto fetch = [&](int t0) {
        xu.load(u, a.u_ds, count, t0, L, lane);
        xd.load(dt, a.d_ds, count, t0, L, lane);
        xb.load(Bm, a.B_ss, a.N, t0, L);
        if constexpr (kOut) xc.load(Cm, a.C_ss, a.N, t0, L);
    };
    auto put = [&](int t0, int buf) {
        Raw::for_each(lane, [&](int i, int rr, int el, auto n_el) {
            constexpr int E = decltype(n_el)::value;
            float uv[E], dv[E];
            xu.get(i, uv, u, a.u_ds, t0, L, lane); xd.get(i, dv, dt, a.d_ds, t0, L, lane);
            float bs = __shfl_sync(0xffffffffu, bias[0], (rr % RL) * SL);
            if constexpr (R == 2) {
                const float b1 = __shfl_sync(0xffffffffu, bias[1], (rr % RL) * SL);
                bs = rr < RL ? bs : b1;
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
                float d = dv[e] + bs;
                if (sp) d = softplus_fast(d);
                dv[e] = t0 + el + e < L ? d : 0.f;   // beyond the row: the state stays as it is
            }
            st_put(sd + rr * P + el, dv);
            st_put(su + rr * P + el, uv);
        });
        xb.put(sbc + buf * 2 * kBC, Bm, a.B_ss, t0, L);
        if constexpr (kOut) xc.put(sbc + buf * 2 * kBC + kBC, Cm, a.C_ss, t0, L);
    };
    if (lo < hi) { fetch(lo); put(lo, 0); }
    __syncthreads();
    int buf = 0;
    for (int t0 = lo; t0 < hi; t0 += kStChunk, buf ^= 1) {
        const bool more = t0 + kStChunk < hi;
        if (kPre && more) fetch(t0 + kStChunk);
        if (a.ckpt && t0 % a.every == 0) {
#pragma unroll
            for (int j = 0; j < R; ++j) {
                float* ck = a.ckpt + (row[j] * a.nck + t0 / a.every) * a.N + n0;
                const float v[4] = {h[j][0].x, h[j][0].y, h[j][1].x, h[j][1].y};
                if (!mine[j]) continue;
                if (a.N == NS) *reinterpret_cast<float4*>(ck) = make_float4(v[0], v[1], v[2], v[3]);
                else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (n0 + i < a.N) ck[i] = v[i];
                }
            }
        }
        // ---- the recurrence, four elements at a time
        const float* sB = sbc + buf * 2 * kBC + n0;
        const float* sC = sB + kBC;
        // A group's decays are formed while the group in front of it is worked on: the exponentials (one per eight
        // cycles and scheduler) then run beside the other arithmetic of the same warp.
        struct Group { float2 dec[R][4][2], x[R][2]; float y[R][4]; float4 b[kAhead ? 4 : 1], c[kAhead ? 4 : 1]; } grp[2];
        auto prepare = [&](int t, Group& g) {
            if constexpr (kAhead) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    g.b[e] = *reinterpret_cast<const float4*>(sB + (t + e) * Y::BCP);
                    if constexpr (kOut) g.c[e] = *reinterpret_cast<const float4*>(sC + (t + e) * Y::BCP);
                }
            }
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const float4 d4 = *reinterpret_cast<const float4*>(sd + (rl + j * RL) * P + t);
                const float4 u4 = *reinterpret_cast<const float4*>(su + (rl + j * RL) * P + t);
                const float2 dd[2] = {make_float2(d4.x, d4.y), make_float2(d4.z, d4.w)}, uu[2] = {make_float2(u4.x, u4.y), make_float2(u4.z, u4.w)};
                if constexpr (!kOut) sum_d[j] += (d4.x + d4.y) + (d4.z + d4.w);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    g.x[j][i] = __fmul2_rn(dd[i], uu[i]);
                    if constexpr (kOut) { g.y[j][2 * i] = Dv[j] * uu[i].x; g.y[j][2 * i + 1] = Dv[j] * uu[i].y; }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float2 g0 = __fmul2_rn(dd[i], f2(A2[j][q].x)), g1 = __fmul2_rn(dd[i], f2(A2[j][q].y));
                        g.dec[j][2 * i][q] = make_float2(ex2_approx(g0.x), ex2_approx(g1.x));
                        g.dec[j][2 * i + 1][q] = make_float2(ex2_approx(g0.y), ex2_approx(g1.y));
                    }
                }
            }
        };
        prepare(0, grp[0]);
#pragma unroll
        for (int t = 0; t < kStChunk; t += 4) {
            Group& g = grp[(t >> 2) & 1];
            float2 (&dec)[R][4][2] = g.dec;
            float2 (&x)[R][2] = g.x;
            float (&y)[R][4] = g.y;
            if (t + 4 < kStChunk) prepare(t + 4, grp[((t >> 2) & 1) ^ 1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 b4 = kAhead ? g.b[kAhead ? e : 0] : *reinterpret_cast<const float4*>(sB + (t + e) * Y::BCP);
                const float2 bb[2] = {make_float2(b4.x, b4.y), make_float2(b4.z, b4.w)};
                float2 cc[2];
                if constexpr (kOut) {
                    const float4 c4 = kAhead ? g.c[kAhead ? e : 0] : *reinterpret_cast<const float4*>(sC + (t + e) * Y::BCP);
                    cc[0] = make_float2(c4.x, c4.y); cc[1] = make_float2(c4.z, c4.w);
                }
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const float xe = e & 1 ? x[j][e >> 1].y : x[j][e >> 1].x;
#pragma unroll
                    for (int q = 0; q < 2; ++q) h[j][q] = __ffma2_rn(dec[j][e][q], h[j][q], __fmul2_rn(f2(xe), bb[q]));
                    if constexpr (kOut) {
                        const float2 s = __ffma2_rn(cc[1], h[j][1], __ffma2_rn(cc[0], h[j][0], make_float2(y[j][e], 0.f)));
                        y[j][e] = s.x + s.y;
                    }
                }
            }
            if constexpr (kOut) {
                // sum over the lanes of the row (which have all read this group's u); a lane keeps the elements that end up with it
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    float* o = su + (rl + j * RL) * P + t;
                    const float* v = y[j];
                    if constexpr (SL == 4) {
                        const bool up = sl & 2, odd = sl & 1;
                        const float k0 = (up ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 2);
                        const float k1 = (up ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 2);
                        o[sl] = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 1);
                    } else if constexpr (SL == 2) {
                        const bool up = sl & 1;
                        const float k0 = (up ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 1);
                        const float k1 = (up ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 1);
                        *reinterpret_cast<float2*>(o + sl * 2) = make_float2(k0, k1);
                    } else {
                        *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
                    }
                }
            }
        }
        __syncwarp();
        if constexpr (kOut) {
            st_unstage<Tout, RPW, VW == 0 ? 1 : VW>(su, (Tout*)a.out + b * a.o_bs + r0 * a.o_ds, a.o_ds, count, t0, L, lane);
            __syncwarp();
        }
        if (more) {
            if (!kPre) fetch(t0 + kStChunk);
            put(t0 + kStChunk, buf ^ 1);
        }
        __syncthreads();     // one barrier per chunk: the readers of the other B / C buffer are past it
    }
    if constexpr (!kOut) {
        if (a.ends && !a.fold && seg + 1 < a.S) {
#pragma unroll
            for (int j = 0; j < R; ++j) {
                if (!mine[j]) continue;
                const int64_t at = row[j] * a.S + seg;
                *reinterpret_cast<float4*>(a.ends + at * NS + n0) = make_float4(h[j][0].x, h[j][0].y, h[j][1].x, h[j][1].y);
                if (sl == 0) a.sums[at] = sum_d[j];
            }
        }
    }
}

template <typename Tin, typename Tout, int NS, int R, int VW, bool kOut>
static int st_launch_fwd(const StFwdArgs& a, int64_t batch, cudaStream_t st) {
    using Y = StLayout<NS, R>;
    constexpr size_t smem = sizeof(float) * (2 * kStRows * kStPitch + 4 * kStChunk * Y::BCP);
    static_assert(smem <= 48 * 1024, "default shared-memory limit");
    const int64_t ctas = batch * a.n_groups * a.parts * a.S;
    if (ctas > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
    // Registers as the compiler likes for pieces (4 608 rows of 8 594, 4 states, 438 us with sixteen warps an SM, 308), and for 16-bit rows of up to
    // four states by single elements where they are not cut: those spill at sixteen warps (64 to 120 bytes; 24 576 rows of 785 elements, f16 / bf16,
    // 168 / 293 us, 143 / 268), which cut rows fill all the same (4 608 rows of 8 594 306 / 453, and 373 / 708).
    constexpr bool spills = VW == 1 && NS == 4 && sizeof(Tin) == 2;
    if (VW == 0 || (spills && a.S == 1)) launch(st_fwd_kernel<Tin, Tout, NS, R, VW, kOut, (VW != 0 && !spills)>, (unsigned)ctas, Y::kWarps * 32, smem, st, a);
    else launch(st_fwd_kernel<Tin, Tout, NS, R, VW, kOut, VW != 0>, (unsigned)ctas, Y::kWarps * 32, smem, st, a);
    count_launch();
    return check_launch();
}

// Rows without vectors are read by pieces: 16-bit ones, and fp32 ones where a warp holds more than 16 of them (4 608 rows of 8 593, 16 states: 1.36 ms,
// 0.82 by single elements; 4 states: 445 against 508 us).
constexpr bool st_takes_pieces(size_t esize, int NS) { return esize == 2 || NS == 4; }
inline int st_pad_states(int64_t N) { return N <= 4 ? 4 : N <= 8 ? 8 : 16; }
inline int st_parts(int64_t group_size) { return (int)((group_size + kStRows - 1) / kStRows); }

template <typename Tin, typename Tout, int NS, int VW, bool kOut>
static int st_rows_per_lane(const StFwdArgs& a, int64_t batch, cudaStream_t st) {
    // two rows per lane from five CTAs (160 rows) per SM up: 16 states, 3 136 elements, bf16: 49 152 rows 1.00 against
    // 1.08 ms, 12 288 rows 0.39 against 0.31 ms
    if constexpr (kOut && NS > 4 && VW > 1) {
        if (batch * a.n_groups * a.parts >= 148 * 5) return st_launch_fwd<Tin, Tout, NS, 2, VW, kOut>(a, batch, st);
    }
    return st_launch_fwd<Tin, Tout, NS, 1, VW, kOut>(a, batch, st);
}

template <typename Tin, typename Tout, int NS, bool kOut> static int st_pieces(const StFwdArgs& a, int64_t batch, cudaStream_t st) {
    if constexpr (st_takes_pieces(sizeof(Tin), NS)) return st_rows_per_lane<Tin, Tout, NS, 0, kOut>(a, batch, st);
    return SS2D_ENOTSUP;                             // never chosen
}

// vw: vector width of the global accesses, 8, 4, 1, or 0 for pieces (st_takes_pieces), in tensors that start and end on 16-byte boundaries
// (no piece reaches beyond them then).
template <typename Tin, typename Tout, bool kOut>
static int st_dispatch_fwd(const StFwdArgs& a, int64_t batch, int vw, cudaStream_t st) {
    const int NS = st_pad_states(a.N);
#define SS2D_ST(NS_)                                                                            \
    if (NS == NS_)                                                                              \
        return vw == 8   ? st_rows_per_lane<Tin, Tout, NS_, 8, kOut>(a, batch, st)              \
               : vw == 4 ? st_rows_per_lane<Tin, Tout, NS_, 4, kOut>(a, batch, st)              \
               : vw == 0 ? st_pieces<Tin, Tout, NS_, kOut>(a, batch, st)                        \
                         : st_rows_per_lane<Tin, Tout, NS_, 1, kOut>(a, batch, st);
    SS2D_ST(4)
    SS2D_ST(8)
    SS2D_ST(16)
#undef SS2D_ST
    return SS2D_ENOTSUP;
}

}  // namespace ss2d
