// Backward of the channel LayerNorm (layer_norm_cf.cu) on dense (B, D, L) maps.
//
//   xhat = (y - mean) rstd,  dy = rstd (g w - mean_D(g w) - xhat mean_D(g w xhat)),  dw = sum g xhat,  db = sum g
//
// A CTA of eight warps takes tiles of 32 pixels (or pixel pairs) of one image: a lane is a pixel, a warp every eighth group of four channels.
// Three passes over the tile (mean; squares and the two sums of g w; results).  Up to 96 channels they work on registers; wider
// maps read the tile again from the caches.  dw / db: the eight values of a warp's four channels are summed over its pixels by halving exchanges
// (nine shuffles) and kept per CTA in shared memory over all its tiles; a second kernel folds the CTAs in a fixed order.
// Bound of the register form: HBM, 6 + 4 bytes per value in 16 bits (32 x 96 x 3 136: 21 us, 0.7 of the copy bandwidth; a pixel per lane, the tile
// read three times and 64-bit addresses for each value took 91 us).
#include "common.cuh"

namespace ss2d {

constexpr int kLnbWarps = 8;
struct NormBwdArgs {
    const float* y;
    const void* g;
    const float* w;
    float *dy, *part;            // part: (CTA, 2, D)
    int D, L, tiles_per_image;
    long long tiles;
    float eps;
};

// PV: pixels per lane (neighbours, one access).  IT > 0: a warp's IT groups of channels stay in registers (D <= 32 * IT).
template <typename Tg, int PV, int IT>
__global__ void __launch_bounds__(kLnbWarps * 32, 3) layer_norm_cf_bwd_kernel(const NormBwdArgs a) {
    follow_previous();
    extern __shared__ __align__(16) float lnb_sm[];                // [2][D] sums of dw, db
    __shared__ float red[3][kLnbWarps][32 * PV];
    using VY = Vec<float, PV>;
    using VG = Vec<Tg, PV>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, D = a.D, L = a.L;
    for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) lnb_sm[i] = 0.f;
    const float inv_d = 1.f / (float)D;
    auto put = [&](int which, const float (&v)[PV]) {
#pragma unroll
        for (int p = 0; p < PV; ++p) red[which][warp][p * 32 + lane] = v[p];
    };
    auto total = [&](int which, float (&t)[PV]) {
#pragma unroll
        for (int p = 0; p < PV; ++p) {
            t[p] = 0.f;
#pragma unroll
            for (int w = 0; w < kLnbWarps; ++w) t[p] += red[which][w][p * 32 + lane];
        }
    };
    constexpr int C = IT > 0 ? IT : 1;
    for (long long tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
        const long long b = tile / a.tiles_per_image;
        const int l = ((int)(tile - b * a.tiles_per_image) * 32 + lane) * PV;
        const bool in = l < L;                       // L is a multiple of PV
        const long long at = b * D * (long long)L + (in ? l : L - PV);
        const float* __restrict__ y = a.y + at;
        const Tg* __restrict__ g = (const Tg*)a.g + at;
        typename VY::Raw ry[C][4];
        typename VG::Raw rg[C][4];
        auto channel = [&](int j, int i) { return (j * kLnbWarps + warp) * 4 + i; };
        // body(j, d of the group's first channel, y values, g values) for every group of four channels of the warp
        auto groups = [&](bool with_g, auto body) {
            if constexpr (IT > 0) {
#pragma unroll
                for (int j = 0; j < IT; ++j) body(ry[j], rg[j], channel(j, 0));
            } else {
#pragma unroll 2
                for (int d0 = warp * 4; d0 < D; d0 += kLnbWarps * 4) {
                    typename VY::Raw qy[4];
                    typename VG::Raw qg[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const long long o = (long long)min(d0 + i, D - 1) * L;
                        qy[i] = VY::load_raw(y + o);
                        if (with_g) qg[i] = VG::load_raw(g + o);
                    }
                    body(qy, qg, d0);
                }
            }
        };
        if constexpr (IT > 0) {
#pragma unroll
            for (int j = 0; j < IT; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const long long o = (long long)min(channel(j, i), D - 1) * L;
                    ry[j][i] = VY::load_raw(y + o); rg[j][i] = VG::load_raw(g + o);
                }
        }
        float s[PV], mean[PV];
#pragma unroll
        for (int p = 0; p < PV; ++p) s[p] = 0.f;
        groups(false, [&](const typename VY::Raw (&qy)[4], const typename VG::Raw (&)[4], int d0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float v[PV];
                VY::unpack(qy[i], v);
#pragma unroll
                for (int p = 0; p < PV; ++p) s[p] += d0 + i < D ? v[p] : 0.f;
            }
        });
        put(0, s);
        __syncthreads();
        total(0, mean);
        float q[PV], s1[PV], s2[PV];
#pragma unroll
        for (int p = 0; p < PV; ++p) { mean[p] *= inv_d; q[p] = s1[p] = s2[p] = 0.f; }
        groups(true, [&](const typename VY::Raw (&qy)[4], const typename VG::Raw (&qg)[4], int d0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float v[PV], gv[PV];
                VY::unpack(qy[i], v); VG::unpack(qg[i], gv);
                const float w = d0 + i < D ? (a.w ? a.w[d0 + i] : 1.f) : 0.f;
#pragma unroll
                for (int p = 0; p < PV; ++p) {
                    const float c = d0 + i < D ? v[p] - mean[p] : 0.f, gw = gv[p] * w;
                    q[p] = fmaf(c, c, q[p]); s1[p] += gw; s2[p] = fmaf(gw, c, s2[p]);
                }
            }
        });
        __syncthreads();
        put(0, q); put(1, s1); put(2, s2);
        __syncthreads();
        float rstd[PV], c1[PV], c2[PV];
        total(0, rstd); total(1, c1); total(2, c2);
#pragma unroll
        for (int p = 0; p < PV; ++p) {
            rstd[p] = rsqrtf(fmaf(rstd[p], inv_d, a.eps));
            c1[p] *= inv_d; c2[p] *= inv_d * rstd[p] * rstd[p];
        }
        __syncthreads();
        float* __restrict__ dy = a.dy + at;
        groups(true, [&](const typename VY::Raw (&qy)[4], const typename VG::Raw (&qg)[4], int d0) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float c[PV], gv[PV], o[PV];
                VY::unpack(qy[i], c); VG::unpack(qg[i], gv);
                const bool real = d0 + i < D && in;
                const float w = d0 + i < D ? (a.w ? a.w[d0 + i] : 1.f) : 0.f;
                v[2 * i] = v[2 * i + 1] = 0.f;
#pragma unroll
                for (int p = 0; p < PV; ++p) {
                    c[p] -= mean[p];
                    o[p] = rstd[p] * (gv[p] * w - c1[p] - c[p] * c2[p]);
                    v[2 * i] = fmaf(gv[p], c[p] * rstd[p], v[2 * i]); v[2 * i + 1] += gv[p];
                }
                if (real) VY::store(dy + (long long)(d0 + i) * L, o);
                else v[2 * i] = v[2 * i + 1] = 0.f;
            }
            int at_v = 0;
#pragma unroll
            for (int n = 4, off = 16; n > 0; n >>= 1, off >>= 1) {
                const bool up = lane & off;
#pragma unroll
                for (int i = 0; i < n; ++i) v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + n], off);
                if (up) at_v += n;
            }
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
            const int d = d0 + (at_v >> 1);
            if ((lane & 3) == 0 && d < D) lnb_sm[(at_v & 1) * D + d] += v[0];
        });
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) a.part[(long long)blockIdx.x * 2 * D + i] = lnb_sm[i];
}

// The tile in registers up to 96 channels, three groups of four per warp: 32 x 96 x 3 136, both launches on cold caches, 38 us against 54
// with three reads.  Six groups spill (80 registers, 1 KB of stack): 32 x 128 x 3 136 124 us against 69 (1.9 TB/s) with three
// reads, 32 x 192 x 3 136 140 against 93 (2.1 TB/s); 16 x 384 x 3 136 runs at 1.9, 32 x 768 x 196 at 0.8 TB/s.
template <typename Tg>
static void launch_lnb(const NormBwdArgs& a, int pv, unsigned ctas, cudaStream_t st) {
    const size_t smem = (size_t)2 * a.D * sizeof(float);
    const int threads = kLnbWarps * 32;
    if (pv == 2) {
        if (a.D <= 96) launch(layer_norm_cf_bwd_kernel<Tg, 2, 3>, ctas, threads, smem, st, a);
        else launch(layer_norm_cf_bwd_kernel<Tg, 2, 0>, ctas, threads, smem, st, a);
    } else {
        if (a.D <= 96) launch(layer_norm_cf_bwd_kernel<Tg, 1, 3>, ctas, threads, smem, st, a);
        else launch(layer_norm_cf_bwd_kernel<Tg, 1, 0>, ctas, threads, smem, st, a);
    }
}

__global__ void __launch_bounds__(256) layer_norm_cf_bwd_fold_kernel(const float* part, int ctas, int D, float* dw, float* db) {
    follow_previous();
    __shared__ float red[8][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), row = threadIdx.x >> 5;
    float s = 0.f;
    if (i < 2 * D)
#pragma unroll 4
        for (int c = row; c < ctas; c += 8) s += part[(long long)c * 2 * D + i];
    red[row][threadIdx.x & 31] = s;
    __syncthreads();
    if (row == 0 && i < 2 * D) {
#pragma unroll
        for (int r = 1; r < 8; ++r) s += red[r][threadIdx.x & 31];
        if (i < D) dw[i] = s;
        else db[i - D] = s;
    }
}

// Pixel pairs where they are aligned and leave a tile for every CTA.
static int lnb_pv(const ss2d_norm_bwd_params* p) {
    const bool even = p->L % 2 == 0 && aligned_to(p->y, 8) && aligned_to(p->dy, 8) && aligned_to(p->g, 2 * dtype_size(p->g_dtype));
    return even && p->B * ((p->L + 63) / 64) >= 148 * 3 ? 2 : 1;
}
static long long lnb_ctas(const ss2d_norm_bwd_params* p) {
    const long long px = 32 * lnb_pv(p), tiles = p->B * ((p->L + px - 1) / px);
    return tiles < 148 * 3 ? tiles : 148 * 3;        // resident at once
}

static int validate_lnb(const ss2d_norm_bwd_params* p) {
    if (!p || !p->y || !p->g || !p->dy || !p->dweight || !p->dbias) return SS2D_EINVAL_NULL;
    if (!dtype_ok(p->g_dtype)) return SS2D_EINVAL_DTYPE;
    if (p->B <= 0 || p->D <= 0 || p->L <= 0 || p->L > 0x3fffffffLL) return SS2D_EINVAL_SHAPE;
    if (p->D > 5500) return SS2D_ENOTSUP;            // two sums per channel in 48 KB of shared memory
    if (!aligned_to(p->y, 4) || !aligned_to(p->dy, 4) || !aligned_to(p->g, dtype_size(p->g_dtype)) || !aligned_to(p->weight, 4) ||
        !aligned_to(p->dweight, 4) || !aligned_to(p->dbias, 4))
        return SS2D_EINVAL_ALIGN;
    return SS2D_OK;
}

long long layer_norm_cf_bwd_workspace_bytes(const ss2d_norm_bwd_params* p) {
    return validate_lnb(p) == SS2D_OK ? lnb_ctas(p) * 2 * p->D * 4 : -1;
}

int layer_norm_cf_bwd(const ss2d_norm_bwd_params* p, cudaStream_t st) {
    const int rc = validate_lnb(p);
    if (rc != SS2D_OK) return rc;
    if (!p->workspace || p->workspace_bytes < layer_norm_cf_bwd_workspace_bytes(p)) return SS2D_EWORKSPACE;
    NormBwdArgs a;
    a.y = (const float*)p->y; a.g = p->g; a.w = (const float*)p->weight; a.dy = (float*)p->dy; a.part = (float*)p->workspace;
    const int pv = lnb_pv(p);
    a.D = (int)p->D; a.L = (int)p->L; a.tiles_per_image = (int)((p->L + 32 * pv - 1) / (32 * pv)); a.tiles = p->B * a.tiles_per_image; a.eps = p->eps;
    const unsigned ctas = (unsigned)lnb_ctas(p);
    if (p->g_dtype == SS2D_F32) launch_lnb<float>(a, pv, ctas, st);
    else if (p->g_dtype == SS2D_BF16) launch_lnb<__nv_bfloat16>(a, pv, ctas, st);
    else launch_lnb<__half>(a, pv, ctas, st);
    launch(layer_norm_cf_bwd_fold_kernel, (unsigned)((2 * p->D + 31) / 32), 256, 0, st, a.part, (int)ctas, a.D, (float*)p->dweight, (float*)p->dbias);
    count_launch(2);
    return check_launch();
}

}  // namespace ss2d
