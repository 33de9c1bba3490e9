// CrossMerge of planes with rows of whole vectors and columns of whole pairs.
//
// A CTA takes a tile of one plane, or a few small planes, and fetches all four routes of it into shared memory in one burst of
// asynchronous copies: the row-like routes in vectors, the column-like ones as they are stored, column by column, in pairs.  A
// warp then takes 8 rows x 4 groups of V pixels.  The pitches (2 modulo 8 elements for columns, an odd number of vectors for
// rows) let its 32 lanes read without bank conflicts; nothing is transposed.
// Bound: HBM.  The burst keeps up to 200 KB of an SM under way; with the row-like routes read as they are needed the same kernel
// waits (62 us), as the kernels that transpose in shared memory do.  fp32, against those: 32 x 96 planes of 56 x 56 68 -> 42 us
// (4.6 TB/s), 512 planes of 256 x 256 188 -> 127 us (5.3 TB/s); bf16, 8 x 96 planes of 128 x 128 89 -> 43 us.
#pragma once
#include "cross_flat.cuh"

namespace ss2d {

struct MergeRowsArgs {
    const void* in;
    void* out;
    int planes, C, H, W, L, PP;          // planes: B * C;  PP of a CTA
    int TH, TW, tiles_w, hb;             // tile, tiles of a row, groups of 8 rows of a tile
    int cpitch, rpitch, slot;            // of columns, of rows, of a route of a plane, in elements
    int clanes, rlanes;                  // lanes (powers of two) of the copies of a column and of a row
    int base[4], sh[4], sw[4], col[4];   // of the routes
    unsigned magic_hb;
};

constexpr int kMergeRowsThreads = 256;

template <int BYTES> __device__ __forceinline__ void cross_copy_async(void* to, const void* from) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(to);
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(from) : "memory");
    else if constexpr (BYTES == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(from) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(from) : "memory");
}

template <typename T, int V>
__global__ void __launch_bounds__(kMergeRowsThreads) cross_merge_rows_kernel(const MergeRowsArgs a, const int scans) {
    extern __shared__ __align__(16) unsigned char cmr_raw[];
    T* sm = reinterpret_cast<T*>(cmr_raw);           // [plane][route][slot]
    const int plane0 = blockIdx.x * a.PP, np = min(a.PP, a.planes - plane0), L = a.L, W = a.W;
    const int ty = blockIdx.y / a.tiles_w, h0 = ty * a.TH, w0 = (blockIdx.y - ty * a.tiles_w) * a.TW;
    const int th = min(a.TH, a.H - h0), tw = min(a.TW, W - w0), tid = threadIdx.x;
    for (int p = 0; p < np; ++p) {
        const int plane = plane0 + p, b = plane / a.C;
        const T* src = (const T*)a.in + ((long long)b * 3 * a.C + plane) * L;        // route 0 of the plane
        T* dst = sm + p * 4 * a.slot;
#pragma unroll
        for (int k = 0; k < 4; ++k, src += (long long)a.C * L, dst += a.slot) {
            if (a.col[k]) {
                const int r0 = 2 * (tid & (a.clanes - 1)), c0 = tid / a.clanes, step = kMergeRowsThreads / a.clanes;
                for (int r = r0; r < th; r += 2 * a.clanes) {
                    const T* q = src + a.base[k] + (w0 + c0) * a.sw[k] + (a.sh[k] < 0 ? -(h0 + r) - 1 : h0 + r);
                    T* d = dst + c0 * a.cpitch + r;
                    for (int c = c0; c < tw; c += step, q += step * a.sw[k], d += step * a.cpitch) cross_copy_async<2 * sizeof(T)>(d, q);
                }
            } else {
                const int c0 = V * (tid & (a.rlanes - 1)), r0 = tid / a.rlanes, step = kMergeRowsThreads / a.rlanes;
                const int dir = a.sw[k] < 0 ? -1 : 1;
                for (int c = c0; c < tw; c += V * a.rlanes) {
                    const int at = (h0 + r0) * W + w0 + c;
                    const T* q = src + (dir < 0 ? L - V - at : at);
                    T* d = dst + r0 * a.rpitch + c;
                    for (int r = r0; r < th; r += step, q += dir * step * W, d += step * a.rpitch) cross_copy_async<V * sizeof(T)>(d, q);
                }
            }
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int lane = tid & 31;
    for (int u = tid >> 5; u < np * a.hb; u += kMergeRowsThreads / 32) {
        const int p = flat_div(u, a.magic_hb), hr = (u - p * a.hb) * 8 + (lane & 7);
        if (hr >= th) continue;
        const T* src[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)      // a column that runs upwards has its pairs in the map's order, each turned round
            src[k] = sm + (p * 4 + k) * a.slot + (a.col[k] ? (a.sh[k] < 0 ? hr ^ 1 : hr) : hr * a.rpitch);
        T* __restrict__ out = (T*)a.out + (long long)(plane0 + p) * L + (h0 + hr) * W + w0;
        for (int w = (lane >> 3) * V; w < tw; w += 4 * V) {
            T v[4][V];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (a.col[k]) {
#pragma unroll
                    for (int i = 0; i < V; ++i) v[k][i] = src[k][(w + i) * a.cpitch];
                } else {                 // a row that runs leftwards likewise, its vectors turned round
                    const typename Vec<T, V>::Raw q = Vec<T, V>::template load_raw<false>(src[k] + w);
                    const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
                    for (int i = 0; i < V; ++i) v[k][i] = a.sw[k] < 0 ? e[V - 1 - i] : e[i];
                }
            }
            typename Vec<T, V>::Raw o;
            T* e = reinterpret_cast<T*>(&o);
#pragma unroll
            for (int i = 0; i < V; ++i) e[i] = flat_sum<T>(scans, v[0][i], v[1][i], v[2][i], v[3][i]);
            Vec<T, V>::store_raw(out + w, o);
        }
    }
}

}  // namespace ss2d
