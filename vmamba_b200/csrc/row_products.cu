// Sums of products of rows: out (G, M, N) = sum over o and l of a (O, G, M, L) . b (O, G, N, L), 16-bit rows, fp32 sums.  The
// weight gradients of the core's projections, whose result is a few thousand numbers and whose rows are a whole map.
//
// A warp owns 16 rows of a and all N rows of b over one part of the (o, l) range.  Both operands have the summed index innermost, and its order is
// free: a lane's 16-byte vector of a row is four words of two elements, and words 0, 1 and words 2, 3 of the lanes of a row are the two halves
// of a k16 operand, the same for a and b, so that the tensor-core fragments are the vectors as they come from memory.  The
// parts' sums meet in the workspace and are added in a fixed order by a second kernel.
// Bound: HBM (a is read once).  The core's training step on 32 x 96 planes of 56 x 56, bf16, 525 -> 507 us (the library's product of 96 x 6 over the
// 3 136 pixels of 128 rows, 37 us, and the sum over the images, 9 us, and 11 and 9 us for x_proj).
#include <algorithm>

#include "common.cuh"

namespace ss2d {

struct RowProductsArgs {
    const void *a, *b;
    float* part;                         // (part, G, M, N)
    int G, M, N, L, len, per_row, blocks;        // elements of a part, parts of a row, blocks of 16 rows of a
    int64_t a_os, a_gs, a_rs, b_os, b_gs, b_rs;
};
constexpr int kRpMost = 64, kRpWarps = 8;        // most rows of b; warps of a CTA

template <typename T, int NT>
__global__ void __launch_bounds__(kRpWarps * 32) row_products_kernel(const RowProductsArgs p) {
    follow_previous();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, warps = blockDim.x >> 5;
    const int block = blockIdx.y * warps + (threadIdx.x >> 5);
    if (block >= p.blocks) return;
    const int part = blockIdx.x, o = part / p.per_row, l_lo = (part - o * p.per_row) * p.len, l_hi = min(p.L, l_lo + p.len), group = blockIdx.z;
    const int m = block * 16 + g;
    const T* __restrict__ a = (const T*)p.a + o * p.a_os + group * p.a_gs;
    const T* __restrict__ b = (const T*)p.b + o * p.b_os + group * p.b_gs;
    const T* a0 = a + min(m, p.M - 1) * p.a_rs;
    const T* a1 = a + min(m + 8, p.M - 1) * p.a_rs;
    const bool in0 = m < p.M, in1 = m + 8 < p.M;
    float acc[NT][4] = {};
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 2
    for (int l = l_lo + t * 8; l - t * 8 < l_hi; l += 32) {
        const bool in = l < l_hi;
        const uint4 x = in && in0 ? *reinterpret_cast<const uint4*>(a0 + l) : zero, y = in && in1 ? *reinterpret_cast<const uint4*>(a1 + l) : zero;
        uint4 v[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) v[n] = in && n * 8 + g < p.N ? *reinterpret_cast<const uint4*>(b + (n * 8 + g) * p.b_rs + l) : zero;
        const uint32_t f0[4] = {x.x, y.x, x.y, y.y}, f1[4] = {x.z, y.z, x.w, y.w};
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const uint32_t b0[2] = {v[n].x, v[n].y}, b1[2] = {v[n].z, v[n].w};
            MmaK16<T>::run(acc[n], f0, b0);
            MmaK16<T>::run(acc[n], f1, b1);
        }
    }
    float* out = p.part + ((int64_t)part * p.G + group) * p.M * p.N;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = m + (e >> 1) * 8, col = n * 8 + 2 * t + (e & 1);
            if (row < p.M && col < p.N) out[row * p.N + col] = acc[n][e];
        }
}

// out[g][m][n], or [g][n][m] with `turned`: the parts in eight runs, then the runs.
__global__ void __launch_bounds__(256) row_products_fold_kernel(const float* part, float* out, int parts, int total, int M, int N, int turned) {
    follow_previous();
    __shared__ float sums[8][32];
    const int lane = threadIdx.x & 31, run = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < total)
        for (int q = run; q < parts; q += 8) s += part[(int64_t)q * total + i];
    sums[run][lane] = s;
    __syncthreads();
    if (run == 0 && i < total) {
#pragma unroll
        for (int q = 1; q < 8; ++q) s += sums[q][lane];
        const int g = i / (M * N), m = (i - g * M * N) / N, n = i - (g * M + m) * N;
        out[turned ? (g * N + n) * M + m : i] = s;
    }
}

static int validate_rp(const ss2d_row_products_params* p) {
    if (!p) return SS2D_EINVAL_NULL;
    if (p->outer <= 0 || p->groups <= 0 || p->M <= 0 || p->N <= 0 || p->L <= 0) return SS2D_EINVAL_SHAPE;
    if (p->dtype != SS2D_BF16 && p->dtype != SS2D_F16) return SS2D_ENOTSUP;
    if (p->N > kRpMost || p->L > 0x3fffffffLL || p->groups > 65535 || p->M > 65535 * 16LL || p->groups * p->M * p->N > 0x7fffffffLL) return SS2D_ENOTSUP;
    for (int64_t x : {p->L, p->a_outer_stride, p->a_group_stride, p->a_row_stride, p->b_outer_stride, p->b_group_stride, p->b_row_stride})
        if (x % 8 != 0) return SS2D_ENOTSUP;
    return SS2D_OK;
}

// Parts: about thirty-two warps for every SM, of at least 64 elements each.
static int64_t rp_plan(const ss2d_row_products_params* p, RowProductsArgs& a) {
    a.blocks = (int)((p->M + 15) / 16);
    const int64_t want = std::max<int64_t>(1, 148 * 32 / (p->groups * a.blocks)), per_row = std::max<int64_t>(1, std::min((want + p->outer - 1) / p->outer, (p->L + 63) / 64));
    a.len = (int)(((p->L + per_row - 1) / per_row + 31) / 32 * 32);
    a.per_row = (int)((p->L + a.len - 1) / a.len);
    return p->outer * a.per_row;
}

long long row_products_workspace_bytes(const ss2d_row_products_params* p) {
    if (validate_rp(p) != SS2D_OK) return -1;
    RowProductsArgs a;
    return (long long)rp_plan(p, a) * p->groups * p->M * p->N * 4;
}

template <typename T, int NT> static void launch_rp(const RowProductsArgs& a, dim3 grid, int threads, cudaStream_t st) {
    launch(row_products_kernel<T, NT>, grid, threads, 0, st, a);
}
template <typename T> static void launch_rp_t(const RowProductsArgs& a, dim3 grid, int threads, cudaStream_t st) {
    switch ((a.N + 7) / 8) {
        case 1: return launch_rp<T, 1>(a, grid, threads, st);
        case 2: return launch_rp<T, 2>(a, grid, threads, st);
        case 3: return launch_rp<T, 3>(a, grid, threads, st);
        case 4: return launch_rp<T, 4>(a, grid, threads, st);
        case 5: return launch_rp<T, 5>(a, grid, threads, st);
        case 6: return launch_rp<T, 6>(a, grid, threads, st);
        case 7: return launch_rp<T, 7>(a, grid, threads, st);
        default: return launch_rp<T, 8>(a, grid, threads, st);
    }
}

int row_products(const ss2d_row_products_params* p, cudaStream_t st) {
    const int rc = validate_rp(p);
    if (rc != SS2D_OK) return rc;
    if (!p->a || !p->b || !p->out) return SS2D_EINVAL_NULL;
    if (!aligned_to(p->a, 16) || !aligned_to(p->b, 16) || !aligned_to(p->out, 4)) return SS2D_EINVAL_ALIGN;
    RowProductsArgs a = {};
    const int64_t parts = rp_plan(p, a), total = p->groups * p->M * p->N;
    if (!p->workspace || p->workspace_bytes < parts * total * 4) return SS2D_EWORKSPACE;
    if (parts > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
    a.a = p->a; a.b = p->b; a.part = (float*)p->workspace;
    a.G = (int)p->groups; a.M = (int)p->M; a.N = (int)p->N; a.L = (int)p->L;
    a.a_os = p->a_outer_stride; a.a_gs = p->a_group_stride; a.a_rs = p->a_row_stride;
    a.b_os = p->b_outer_stride; a.b_gs = p->b_group_stride; a.b_rs = p->b_row_stride;
    const int warps = std::min(a.blocks, kRpWarps);
    const dim3 grid((unsigned)parts, (unsigned)((a.blocks + warps - 1) / warps), (unsigned)p->groups);
    if (p->dtype == SS2D_BF16) launch_rp_t<__nv_bfloat16>(a, grid, warps * 32, st);
    else launch_rp_t<__half>(a, grid, warps * 32, st);
    count_launch();
    launch(row_products_fold_kernel, (unsigned)((total + 31) / 32), 256, 0, st, (const float*)a.part, (float*)p->out, (int)parts, (int)total, a.M, a.N, (int)p->turned);
    count_launch();
    return check_launch();
}

}  // namespace ss2d
