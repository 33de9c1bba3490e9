// Selective-scan backward for 2 .. 16 states (layout: scan_states.cuh, one row per lane).
//
// A CTA owns RS sets of 32 rows of one (image, group) and walks them from the end in chunks of 32 elements, at whose starts
// the forward pass left the states.  Per chunk and row set the rows' step sizes, u and dout are staged in shared memory and a
// forward sweep leaves the states in front of the chunk's four tiles of eight elements.  The tiles are then taken from
// the last to the first; in a tile a lane forms its four states' decays and states forward and the reverse recurrence
// backward, all in registers, and adds its dB / dC terms to registers that collect over the row sets.  Over the lanes of a row
// only two sums per element are needed, S1 = sum dh B and S2 = sum A dh a h_prev (du = d' S1 + g D, dd' = S2 + u S1); over
// the rows the 64 collected dB / dC terms of a tile, once per tile whatever the number of row sets.  Both are halving
// exchanges between lanes: half of the values change hands in each round.
//
// Rows too few for the chip are cut into segments: st_bwd_segments_kernel leaves what a segment does to the reverse state.
//
// Bound: latency at eight warps per SM (254 registers).  4 x 1 536 rows of 1 001 elements, 16 states, fp32, 196 us: an SM issues in 47 %
// of its cycles with 1.8 warps per scheduler, 0.6 of them eligible, its shared memory at 52 %, DRAM at 8 %.  The
// instructions (about 11 per element and state) are 29 us at full rate, the exponentials (1.75) 37 us.
#pragma once
#include "scan_n1_bwd.cuh"
#include "scan_states_fwd.cuh"

namespace ss2d {

constexpr int kStTile = 8, kStTiles = kStChunk / kStTile, kStMaxSets = 2;

struct StBwdArgs {
    const void *u, *delta, *B, *C, *dout;
    const float *A, *D, *bias;
    void *du, *ddelta;
    float* rowred;           // (segment, image, row, N + 2): dA, dD, dbias
    float* bcpart;           // (image, group, part, 2, N, Lp)
    const float* ckpt;       // (rows, ceil(L / 32), N)
    float *ends, *sums;      // (row, S, NS), (row, S); null with S = 1
    int64_t dim, group_size, batch;
    int64_t u_bs, u_ds, d_bs, d_ds, g_bs, g_ds, B_bs, B_gs, B_ss, C_bs, C_gs, C_ss;
    int L, Lp, N, n_groups, parts, sets, softplus, S, seg_len;
};

// Derivative of the softplus from its value: 1 - exp(-d), as a series where the difference would cancel.
__device__ __forceinline__ float softplus_grad_of(float d) {
    const float s = d * fmaf(d, fmaf(d, fmaf(d, -0.041666668f, 0.16666667f), -0.5f), 1.f);
    return d < 0.03125f ? s : 1.f - ex2_approx(-d * kLog2e);
}

template <int NS> struct StBwdSmem {
    using Y = StLayout<NS>;
    static constexpr int kWarpRed = 2 * NS * kStTile;                   // `red`: [tile][warp][B / C][state][element]
    static constexpr int kTilePitch = Y::kWarps * kWarpRed + kStTile;
    static constexpr int kRowFloats = 3 * kStPitch;                     // per row and set
    static constexpr int kLaneFloats = 4 * kStTiles + 4 + 4 + 4 + 2;               // per lane and set: tile states, e, dA, (dD, dbias)
    static size_t bytes(int sets) {
        return sizeof(float) * ((size_t)sets * (kStRows * kRowFloats + Y::kWarps * 32 * kLaneFloats) + 2 * kStChunk * Y::BCP + kStTiles * kTilePitch);
    }
};

template <typename Tin, typename Tg, int NS, int VW>
__global__ void __launch_bounds__(StLayout<NS>::kWarps * 32, 8 / StLayout<NS>::kWarps) st_bwd_kernel(const StBwdArgs a) {
    follow_previous();
    using Y = StLayout<NS>;
    using M = StBwdSmem<NS>;
    constexpr int RPW = Y::RPW, SL = Y::SL, P = kStPitch, W = Y::kWarps, kRow = RPW * P;
    extern __shared__ __align__(16) float st_sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rl = lane / SL, sl = lane % SL, n0 = sl * 4;
    const int sets = a.sets, L = a.L, gs = (int)a.group_size;
    float* rows_s = st_sm + (size_t)warp * sets * 3 * kRow;                     // [set][d, u, g][row][36]
    float* q0 = st_sm + (size_t)W * sets * 3 * kRow;
    float4* hs = reinterpret_cast<float4*>(q0) + (size_t)warp * sets * kStTiles * 32;  // [set][tile][lane]: states in front of the tile
    q0 += (size_t)W * sets * kStTiles * 32 * 4;
    float4* ecar = reinterpret_cast<float4*>(q0) + (size_t)warp * sets * 32;    // [set][lane]
    q0 += (size_t)W * sets * 32 * 4;
    float4* dA_s = reinterpret_cast<float4*>(q0) + (size_t)warp * sets * 32;
    q0 += (size_t)W * sets * 32 * 4;
    float4* A_s = reinterpret_cast<float4*>(q0) + (size_t)warp * sets * 32;
    q0 += (size_t)W * sets * 32 * 4;
    float* sB = q0;
    float* sC = sB + kStChunk * Y::BCP;
    float* red = sC + kStChunk * Y::BCP;
    float2* dDb = reinterpret_cast<float2*>(red + kStTiles * M::kTilePitch) + (size_t)warp * sets * 32;
    int cta = blockIdx.x;
    const int seg = cta % a.S; cta /= a.S;
    const int part = cta % a.parts; cta /= a.parts;
    const int k = cta % a.n_groups;
    const int64_t b = cta / a.n_groups;
    const int first = part * sets * kStRows + warp * RPW;       // rows of set s inside the group: first + s * 32 ..
    const int lo = seg * a.seg_len, hi = min(L, lo + a.seg_len);
    const int64_t g0 = (int64_t)k * gs;                         // first row of the group
    const Tin* __restrict__ u = (const Tin*)a.u + b * a.u_bs + g0 * a.u_ds;
    const Tin* __restrict__ dt = (const Tin*)a.delta + b * a.d_bs + g0 * a.d_ds;
    const Tg* __restrict__ gp = (const Tg*)a.dout + b * a.g_bs + g0 * a.g_ds;
    const Tin* __restrict__ Bm = (const Tin*)a.B + b * a.B_bs + k * a.B_gs;
    const Tin* __restrict__ Cm = (const Tin*)a.C + b * a.C_bs + k * a.C_gs;
    Tin* __restrict__ du = (Tin*)a.du + (b * a.dim + g0) * L;
    Tin* __restrict__ dd = (Tin*)a.ddelta + (b * a.dim + g0) * L;
    const int nck = (L + kStChunk - 1) / kStChunk;
    const bool sp = a.softplus != 0;

    auto row_in_group = [&](int s) { const int ig = first + s * kStRows + rl; return ig < gs ? ig : gs - 1; };
    auto count_of = [&](int s) { return max(0, min(RPW, gs - first - s * kStRows)); };
    auto load_A = [&](int s, float2 (&A)[2]) {
        const float4 v = A_s[s * 32 + lane];
        A[0] = make_float2(v.x, v.y); A[1] = make_float2(v.z, v.w);
    };
    for (int s = 0; s < sets; ++s) {
        float2 e[2] = {f2(0.f), f2(0.f)}, A[2];
        {
            const float* p = a.A + (g0 + row_in_group(s)) * a.N + n0;
            float t[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] = n0 + i < a.N ? p[i] : 0.f;
            A_s[s * 32 + lane] = make_float4(t[0], t[1], t[2], t[3]);
            load_A(s, A);
        }
        A[0] = __fmul2_rn(A[0], f2(kLog2e)); A[1] = __fmul2_rn(A[1], f2(kLog2e));
        if (a.S > 1) st_fold_segments<true>(e, A, a.ends, a.sums, b * a.dim + g0 + row_in_group(s), a.S, seg, n0, NS);
        ecar[s * 32 + lane] = make_float4(e[0].x, e[0].y, e[1].x, e[1].y);
        dA_s[s * 32 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
        dDb[s * 32 + lane] = make_float2(0.f, 0.f);
    }

    for (int t0 = (hi - 1) / kStChunk * kStChunk; t0 >= lo; t0 -= kStChunk) {
        // ---- stage B and C of the chunk
        {
            StRawBC<Tin, NS, VW, W> xb, xc;
            xb.load(Bm, a.B_ss, a.N, t0, L); xc.load(Cm, a.C_ss, a.N, t0, L);
            xb.put(sB, Bm, a.B_ss, t0, L); xc.put(sC, Cm, a.C_ss, t0, L);
        }
        // ---- stage the rows
        for (int s = 0; s < sets; ++s) {
            const int count = count_of(s);
            const int64_t o = first + s * kStRows;
            float* sd = rows_s + (size_t)s * 3 * kRow;
            StRaw<Tin, RPW, VW> xu, xd;
            StRaw<Tg, RPW, VW> xg;
            xd.load(dt + o * a.d_ds, a.d_ds, count, t0, L, lane);
            xu.load(u + o * a.u_ds, a.u_ds, count, t0, L, lane);
            xg.load(gp + o * a.g_ds, a.g_ds, count, t0, L, lane);
            const float bias_rl = a.bias ? a.bias[g0 + row_in_group(s)] : 0.f;
            {                                        // the state in front of the chunk
                const float* ck = a.ckpt + ((b * a.dim + g0 + row_in_group(s)) * nck + t0 / kStChunk) * a.N + n0;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (a.N == NS) v = *reinterpret_cast<const float4*>(ck);
                else {
                    if (n0 < a.N) v.x = *ck;
                    if (n0 + 1 < a.N) v.y = ck[1];
                    if (n0 + 2 < a.N) v.z = ck[2];
                    if (n0 + 3 < a.N) v.w = ck[3];
                }
                hs[s * kStTiles * 32 + lane] = v;
            }
            StRaw<Tin, RPW, VW>::for_each(lane, [&](int i, int rr, int el, auto n_el) {
                constexpr int E = decltype(n_el)::value;
                float uv[E], dv[E], gv[E];
                xd.get(i, dv, dt + o * a.d_ds, a.d_ds, t0, L, lane); xu.get(i, uv, u + o * a.u_ds, a.u_ds, t0, L, lane);
                xg.get(i, gv, gp + o * a.g_ds, a.g_ds, t0, L, lane);
                const float bs = __shfl_sync(0xffffffffu, bias_rl, rr * SL);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    float d = dv[e] + bs;
                    if (sp) d = softplus_fast(d);
                    dv[e] = t0 + el + e < L && rr < count ? d : 0.f;    // beyond the row: a step of zero
                }
                st_put(sd + rr * P + el, dv);
                st_put(sd + kRow + rr * P + el, uv);
                st_put(sd + 2 * kRow + rr * P + el, gv);
            });
        }
        if (t0 > lo) {                               // the next chunk of every row, on its way into L2
            for (int s = 0; s < sets; ++s) {
                const int64_t ig = row_in_group(s);
                const void* at = sl == 0 ? (const void*)(u + ig * a.u_ds + t0 - kStChunk) : (const void*)(dt + ig * a.d_ds + t0 - kStChunk);
                if (SL > 2 && sl == 2) at = gp + ig * a.g_ds + t0 - kStChunk;
                if (SL > 2 && sl == 3) at = a.ckpt + ((b * a.dim + g0 + ig) * nck + t0 / kStChunk - 1) * a.N;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
                if (SL < 4) asm volatile("prefetch.global.L2 [%0];" ::"l"(gp + ig * a.g_ds + t0 - kStChunk));
            }
        }
        __syncthreads();
        // ---- forward sweep: the states in front of the tiles
        for (int s = 0; s < sets; ++s) {
            const float* sd = rows_s + (size_t)s * 3 * kRow + rl * P;
            const float* su = sd + kRow;
            float2 A[2], h[2];
            load_A(s, A);
            A[0] = __fmul2_rn(A[0], f2(kLog2e)); A[1] = __fmul2_rn(A[1], f2(kLog2e));
            {
                const float4 v = hs[s * kStTiles * 32 + lane];
                h[0] = make_float2(v.x, v.y); h[1] = make_float2(v.z, v.w);
            }
#pragma unroll 1
            for (int tile = 1; tile < kStTiles; ++tile) {
#pragma unroll
                for (int t = 0; t < kStTile; t += 4) {
                    const int at = (tile - 1) * kStTile + t;
                    const float4 d4 = *reinterpret_cast<const float4*>(sd + at), u4 = *reinterpret_cast<const float4*>(su + at);
                    const float d[4] = {d4.x, d4.y, d4.z, d4.w}, uv[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float4 b4 = *reinterpret_cast<const float4*>(sB + (at + e) * Y::BCP + n0);
                        const float2 bb[2] = {make_float2(b4.x, b4.y), make_float2(b4.z, b4.w)};
                        const float x = d[e] * uv[e];
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const float2 g = __fmul2_rn(f2(d[e]), A[q]);
                            h[q] = __ffma2_rn(make_float2(ex2_approx(g.x), ex2_approx(g.y)), h[q], __fmul2_rn(f2(x), bb[q]));
                        }
                    }
                }
                hs[(s * kStTiles + tile) * 32 + lane] = make_float4(h[0].x, h[0].y, h[1].x, h[1].y);
            }
        }
        // ---- the tiles, last first
#pragma unroll 1
        for (int tile = kStTiles - 1; tile >= 0; --tile) {
            const int at = tile * kStTile;
            float2 acc[kStTile][2][2];              // [element][dB, dC][state pair], over the row sets
#pragma unroll
            for (int t = 0; t < kStTile; ++t)
#pragma unroll
                for (int q = 0; q < 2; ++q) acc[t][0][q] = acc[t][1][q] = f2(0.f);
#pragma unroll 1
            for (int s = 0; s < sets; ++s) {
                float* sd = rows_s + (size_t)s * 3 * kRow + rl * P + at;
                float* su = sd + kRow;
                const float* sg = sd + 2 * kRow;
                float2 A[2], av[kStTile][2], hp[kStTile][2], h[2], e[2];
                float d[kStTile], x[kStTile];
                load_A(s, A);
                {
                    const float4 v = hs[(s * kStTiles + tile) * 32 + lane], w = ecar[s * 32 + lane];
                    h[0] = make_float2(v.x, v.y); h[1] = make_float2(v.z, v.w);
                    e[0] = make_float2(w.x, w.y); e[1] = make_float2(w.z, w.w);
                }
                float gv[kStTile];
#pragma unroll
                for (int t = 0; t < kStTile; t += 4) {
                    const float4 d4 = *reinterpret_cast<const float4*>(sd + t), u4 = *reinterpret_cast<const float4*>(su + t),
                                 g4 = *reinterpret_cast<const float4*>(sg + t);
                    d[t] = d4.x; d[t + 1] = d4.y; d[t + 2] = d4.z; d[t + 3] = d4.w;
                    x[t] = d4.x * u4.x; x[t + 1] = d4.y * u4.y; x[t + 2] = d4.z * u4.z; x[t + 3] = d4.w * u4.w;
                    gv[t] = g4.x; gv[t + 1] = g4.y; gv[t + 2] = g4.z; gv[t + 3] = g4.w;
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float2 A2 = __fmul2_rn(A[q], f2(kLog2e));
#pragma unroll
                    for (int t = 0; t < kStTile; ++t) {
                        const float2 w = __fmul2_rn(f2(d[t]), A2);
                        av[t][q] = make_float2(ex2_approx(w.x), ex2_approx(w.y));
                    }
                }
#pragma unroll
                for (int t = 0; t < kStTile; ++t) {
                    const float4 b4 = *reinterpret_cast<const float4*>(sB + (at + t) * Y::BCP + n0);
                    const float2 bb[2] = {make_float2(b4.x, b4.y), make_float2(b4.z, b4.w)};
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        hp[t][q] = h[q];
                        h[q] = __ffma2_rn(av[t][q], h[q], __fmul2_rn(f2(x[t]), bb[q]));
                        acc[t][1][q] = __ffma2_rn(f2(gv[t]), h[q], acc[t][1][q]);
                    }
                }
                float2 dA[2] = {f2(0.f), f2(0.f)};
                float S[2][kStTile];                 // S1, S2 of the tile's elements
#pragma unroll
                for (int t = kStTile - 1; t >= 0; --t) {
                    const float4 b4 = *reinterpret_cast<const float4*>(sB + (at + t) * Y::BCP + n0), c4 = *reinterpret_cast<const float4*>(sC + (at + t) * Y::BCP + n0);
                    const float2 bb[2] = {make_float2(b4.x, b4.y), make_float2(b4.z, b4.w)}, cc[2] = {make_float2(c4.x, c4.y), make_float2(c4.z, c4.w)};
                    float2 s1, s2;
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const float2 dh = __ffma2_rn(cc[q], f2(gv[t]), e[q]);
                        e[q] = __fmul2_rn(av[t][q], dh);
                        const float2 y = __fmul2_rn(e[q], hp[t][q]);                 // dh a h_prev
                        acc[t][0][q] = __ffma2_rn(dh, f2(x[t]), acc[t][0][q]);
                        dA[q] = __ffma2_rn(f2(d[t]), y, dA[q]);
                        s1 = q ? __ffma2_rn(dh, bb[q], s1) : __fmul2_rn(dh, bb[q]);
                        s2 = q ? __ffma2_rn(A[q], y, s2) : __fmul2_rn(A[q], y);
                    }
                    S[0][t] = s1.x + s1.y; S[1][t] = s2.x + s2.y;
                }
                ecar[s * 32 + lane] = make_float4(e[0].x, e[0].y, e[1].x, e[1].y);
                {
                    const float4 v = dA_s[s * 32 + lane];
                    dA_s[s * 32 + lane] = make_float4(v.x + dA[0].x, v.y + dA[0].y, v.z + dA[1].x, v.w + dA[1].y);
                }
                // sums over the lanes of the row: lane sl keeps elements [sl * E, (sl + 1) * E)
                constexpr int E = kStTile / SL;
#pragma unroll
                for (int n = kStTile / 2, off = SL / 2; off > 0; n >>= 1, off >>= 1) {
                    const bool up = sl & off;
#pragma unroll
                    for (int w = 0; w < 2; ++w)
#pragma unroll
                        for (int t = 0; t < n; ++t)
                            S[w][t] = (up ? S[w][t + n] : S[w][t]) + __shfl_xor_sync(0xffffffffu, up ? S[w][t] : S[w][t + n], off);
                }
                __syncwarp();                        // every lane of the row has read d, u, g of the tile
                const float Dv = a.D ? a.D[g0 + row_in_group(s)] : 0.f;
                float2 db = dDb[s * 32 + lane];
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    const int t = sl * E + i;
                    const float dv = sd[t], uv = su[t], g = sg[t];
                    const float o = fmaf(uv, S[0][i], S[1][i]) * (sp ? softplus_grad_of(dv) : (t0 + at + t < L ? 1.f : 0.f));
                    db.x = fmaf(g, uv, db.x);
                    db.y += o;
                    su[t] = fmaf(dv, S[0][i], g * Dv);
                    sd[t] = o;
                }
                dDb[s * 32 + lane] = db;
            }
            // dB / dC of the tile over the warp's rows.  Values v = (element, which, state): every round of the exchange
            // halves the highest bit left
            {
                float v[8 * kStTile];
#pragma unroll
                for (int t = 0; t < kStTile; ++t)
#pragma unroll
                    for (int w = 0; w < 2; ++w) {
                        v[t * 8 + w * 4] = acc[t][w][0].x; v[t * 8 + w * 4 + 1] = acc[t][w][0].y;
                        v[t * 8 + w * 4 + 2] = acc[t][w][1].x; v[t * 8 + w * 4 + 3] = acc[t][w][1].y;
                    }
                int at_v = 0;                        // index of this lane's first value
#pragma unroll
                for (int n = 4 * kStTile, off = 16; off >= SL; n >>= 1, off >>= 1) {
                    const bool up = lane & off;
#pragma unroll
                    for (int i = 0; i < n; ++i) v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + n], off);
                    if (up) at_v += n;
                }
                constexpr int KEEP = 8 * kStTile / RPW;          // consecutive values, of one element
                float* o = red + tile * M::kTilePitch + warp * M::kWarpRed + (at_v >> 3);
#pragma unroll
                for (int i = 0; i < KEEP; ++i) o[(((at_v + i) >> 2) & 1) * NS * kStTile + (n0 + ((at_v + i) & 3)) * kStTile] = v[i];
            }
        }
        __syncthreads();
        // ---- out: du, ddelta from the rows' slots; dB, dC summed over the warps
        for (int s = 0; s < sets; ++s) {
            const float* sd = rows_s + (size_t)s * 3 * kRow;
            const int64_t o = first + s * kStRows;
            st_unstage<Tin, RPW, VW>(sd, dd + o * L, L, count_of(s), t0, L, lane);
            st_unstage<Tin, RPW, VW>(sd + kRow, du + o * L, L, count_of(s), t0, L, lane);
        }
        float* bc_out = a.bcpart + ((b * a.n_groups + k) * a.parts + part) * 2 * (int64_t)a.N * a.Lp + t0;
        for (int i = threadIdx.x; i < 2 * NS * kStChunk; i += W * 32) {
            const int el = i & 31, m = i >> 5, w2 = m / NS, n = m % NS;
            if (n < a.N) {
                const float* p = red + (el / kStTile) * M::kTilePitch + (w2 * NS + n) * kStTile + (el & (kStTile - 1));
                float t = p[0];
#pragma unroll
                for (int w = 1; w < W; ++w) t += p[w * M::kWarpRed];
                bc_out[((int64_t)w2 * a.N + n) * a.Lp + el] = t;
            }
        }
        __syncwarp();
    }
    for (int s = 0; s < sets; ++s) {
        const int ig = first + s * kStRows + rl;
        float2 v = dDb[s * 32 + lane];
#pragma unroll
        for (int off = 1; off < SL; off <<= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
        }
        if (ig < gs) {
            float* rr = a.rowred + (((int64_t)seg * a.batch + b) * a.dim + g0 + ig) * (a.N + 2);
            const float4 w = dA_s[s * 32 + lane];
            const float x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (n0 + i < a.N) rr[n0 + i] = x[i];
            if (sl == 0) { rr[a.N] = v.x; rr[a.N + 1] = v.y; }
        }
    }
}

// What a segment does to the reverse state: its value from zero and the sum of its step sizes.  Segment 0 is read by nobody.
template <typename Tin, typename Tg, int NS, int VW>
__global__ void __launch_bounds__(StLayout<NS>::kWarps * 32) st_bwd_segments_kernel(const StBwdArgs a) {
    follow_previous();
    using Y = StLayout<NS>;
    constexpr int RPW = Y::RPW, SL = Y::SL, P = kStPitch, W = Y::kWarps, kRow = RPW * P;
    extern __shared__ __align__(16) float st_sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rl = lane / SL, sl = lane % SL, n0 = sl * 4;
    float* sd = st_sm + warp * 2 * kRow;
    float* sg = sd + kRow;
    float* sC = st_sm + W * 2 * kRow;
    const int segs = a.S - 1, parts = (int)((a.group_size + kStRows - 1) / kStRows), L = a.L, gs = (int)a.group_size;
    int cta = blockIdx.x;
    const int seg = cta % segs + 1; cta /= segs;
    const int part = cta % parts; cta /= parts;
    const int k = cta % a.n_groups;
    const int64_t b = cta / a.n_groups;
    const int first = part * kStRows + warp * RPW, count = max(0, min(RPW, gs - first)), ig = min(first + rl, gs - 1);
    const int64_t g0 = (int64_t)k * gs, row = b * a.dim + g0 + ig;
    const Tin* __restrict__ dt = (const Tin*)a.delta + b * a.d_bs + (g0 + first) * a.d_ds;
    const Tg* __restrict__ gp = (const Tg*)a.dout + b * a.g_bs + (g0 + first) * a.g_ds;
    const Tin* __restrict__ Cm = (const Tin*)a.C + b * a.C_bs + k * a.C_gs;
    float2 A2[2], e[2] = {f2(0.f), f2(0.f)};
    {
        float t[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = n0 + i < a.N ? a.A[(g0 + ig) * a.N + n0 + i] * kLog2e : 0.f;
        A2[0] = make_float2(t[0], t[1]); A2[1] = make_float2(t[2], t[3]);
    }
    const float bias_rl = a.bias ? a.bias[g0 + ig] : 0.f;
    const bool sp = a.softplus != 0;
    const int lo = seg * a.seg_len, hi = min(L, lo + a.seg_len);
    float sum = 0.f;
    for (int t0 = (hi - 1) / kStChunk * kStChunk; t0 >= lo; t0 -= kStChunk) {
        {
            StRawBC<Tin, NS, VW, W> xc;
            StRaw<Tin, RPW, VW> xd;
            StRaw<Tg, RPW, VW> xg;
            xc.load(Cm, a.C_ss, a.N, t0, L);
            xd.load(dt, a.d_ds, count, t0, L, lane);
            xg.load(gp, a.g_ds, count, t0, L, lane);
            __syncthreads();                         // the chunk in front is read
            xc.put(sC, Cm, a.C_ss, t0, L);
            StRaw<Tin, RPW, VW>::for_each(lane, [&](int i, int rr, int el, auto n_el) {
                constexpr int E = decltype(n_el)::value;
                float dv[E], gv[E];
                xd.get(i, dv, dt, a.d_ds, t0, L, lane); xg.get(i, gv, gp, a.g_ds, t0, L, lane);
                const float bs = __shfl_sync(0xffffffffu, bias_rl, rr * SL);
#pragma unroll
                for (int j = 0; j < E; ++j) {
                    float d = dv[j] + bs;
                    if (sp) d = softplus_fast(d);
                    dv[j] = t0 + el + j < L && rr < count ? d : 0.f;
                }
                st_put(sd + rr * P + el, dv);
                st_put(sg + rr * P + el, gv);
            });
        }
        __syncthreads();
#pragma unroll 2
        for (int t = kStChunk - 4; t >= 0; t -= 4) {
            const float4 d4 = *reinterpret_cast<const float4*>(sd + rl * P + t), g4 = *reinterpret_cast<const float4*>(sg + rl * P + t);
            const float d[4] = {d4.x, d4.y, d4.z, d4.w}, g[4] = {g4.x, g4.y, g4.z, g4.w};
            sum += (d[0] + d[1]) + (d[2] + d[3]);
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                const float4 c4 = *reinterpret_cast<const float4*>(sC + (t + j) * Y::BCP + n0);
                const float2 cc[2] = {make_float2(c4.x, c4.y), make_float2(c4.z, c4.w)};
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float2 w = __fmul2_rn(f2(d[j]), A2[q]);
                    e[q] = __fmul2_rn(make_float2(ex2_approx(w.x), ex2_approx(w.y)), __ffma2_rn(cc[q], f2(g[j]), e[q]));
                }
            }
        }
    }
    if (first + rl < gs) {
        *reinterpret_cast<float4*>(a.ends + (row * a.S + seg) * NS + n0) = make_float4(e[0].x, e[0].y, e[1].x, e[1].y);
        if (sl == 0) a.sums[row * a.S + seg] = sum;
    }
}

}  // namespace ss2d
