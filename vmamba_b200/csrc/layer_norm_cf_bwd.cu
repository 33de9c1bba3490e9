// Backward of the channel LayerNorm (layer_norm_cf.cu) on dense (B, D, L) maps.
//
//   xhat = (y - mean) rstd,  dy = rstd (g w - mean_D(g w) - xhat mean_D(g w xhat)),  dw = sum g xhat,  db = sum g
//
// A CTA of eight warps takes tiles of 32 pixels of one image: a lane is a pixel, a warp every eighth group of four channels.
// Three passes over the tile (mean; squares and the two sums of g w; results), of which the first reads memory and the
// others the caches.  dw / db: the eight values of a warp's four channels are summed over its pixels by halving exchanges
// (nine shuffles) and kept per CTA in shared memory over all its tiles; a second kernel folds the CTAs in a fixed order.
// Bound: HBM, 6 + 4 bytes per value in 16 bits.
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

template <typename Tg>
__global__ void __launch_bounds__(kLnbWarps * 32) layer_norm_cf_bwd_kernel(const NormBwdArgs a) {
    extern __shared__ float lnb_sm[];                // [2][D] sums of dw, db
    __shared__ float red[3][kLnbWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, D = a.D, L = a.L;
    for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) lnb_sm[i] = 0.f;
    __syncthreads();
    const float inv_d = 1.f / (float)D;
    auto total = [&](int which) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < kLnbWarps; ++w) t += red[which][w][lane];
        return t;
    };
    for (long long tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
        const long long b = tile / a.tiles_per_image;
        const int l = (int)(tile - b * a.tiles_per_image) * 32 + lane;
        const bool in = l < L;
        const long long at = b * D * (long long)L + (in ? l : L - 1);
        const float* __restrict__ y = a.y + at;
        const Tg* __restrict__ g = (const Tg*)a.g + at;
        float s = 0.f;
#pragma unroll 2
        for (int d0 = warp * 4; d0 < D; d0 += kLnbWarps * 4)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (d0 + i < D) s += __ldg(y + (long long)(d0 + i) * L);
        red[0][warp][lane] = s;
        __syncthreads();
        const float mean = total(0) * inv_d;
        __syncthreads();
        float q = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll 2
        for (int d0 = warp * 4; d0 < D; d0 += kLnbWarps * 4)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (d0 + i < D) {
                    const float v = __ldg(y + (long long)(d0 + i) * L) - mean;
                    const float gw = to_f<Tg>(__ldg(g + (long long)(d0 + i) * L)) * (a.w ? __ldg(a.w + d0 + i) : 1.f);
                    q = fmaf(v, v, q); s1 += gw; s2 = fmaf(gw, v, s2);
                }
        red[0][warp][lane] = q; red[1][warp][lane] = s1; red[2][warp][lane] = s2;
        __syncthreads();
        const float rstd = rsqrtf(fmaf(total(0), inv_d, a.eps));
        const float c1 = total(1) * inv_d, c2 = total(2) * inv_d * rstd * rstd;
        __syncthreads();
        float* __restrict__ dy = a.dy + at;
        for (int d0 = warp * 4; d0 < D; d0 += kLnbWarps * 4) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[2 * i] = v[2 * i + 1] = 0.f;
                if (d0 + i < D && in) {
                    const float c = __ldg(y + (long long)(d0 + i) * L) - mean, gv = to_f<Tg>(__ldg(g + (long long)(d0 + i) * L));
                    const float gw = gv * (a.w ? __ldg(a.w + d0 + i) : 1.f);
                    dy[(long long)(d0 + i) * L] = rstd * (gw - c1 - c * c2);
                    v[2 * i] = gv * c * rstd; v[2 * i + 1] = gv;
                }
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
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) a.part[(long long)blockIdx.x * 2 * D + i] = lnb_sm[i];
}

__global__ void __launch_bounds__(256) layer_norm_cf_bwd_fold_kernel(const float* part, int ctas, int D, float* dw, float* db) {
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

static long long lnb_ctas(const ss2d_norm_bwd_params* p) {
    const long long tiles = p->B * ((p->L + 31) / 32);
    return tiles < 148 * 6 ? tiles : 148 * 6;
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
    a.D = (int)p->D; a.L = (int)p->L; a.tiles_per_image = (int)((p->L + 31) / 32); a.tiles = p->B * a.tiles_per_image; a.eps = p->eps;
    const unsigned ctas = (unsigned)lnb_ctas(p);
    const size_t smem = (size_t)2 * p->D * sizeof(float);
    if (p->g_dtype == SS2D_F32) layer_norm_cf_bwd_kernel<float><<<ctas, kLnbWarps * 32, smem, st>>>(a);
    else if (p->g_dtype == SS2D_BF16) layer_norm_cf_bwd_kernel<__nv_bfloat16><<<ctas, kLnbWarps * 32, smem, st>>>(a);
    else layer_norm_cf_bwd_kernel<__half><<<ctas, kLnbWarps * 32, smem, st>>>(a);
    layer_norm_cf_bwd_fold_kernel<<<(unsigned)((2 * p->D + 31) / 32), 256, 0, st>>>(a.part, (int)ctas, a.D, (float*)p->dweight, (float*)p->dbias);
    count_launch(2);
    return check_launch();
}

}  // namespace ss2d
