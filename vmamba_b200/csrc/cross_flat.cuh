// CrossScan / CrossMerge of whole planes whose pixel count no vector width divides.
//
// The planes of an image are neighbours in x and in every route, so the PP planes of a CTA are ONE run of PP * L elements in
// each of them.  A run is moved as aligned 8-byte words whatever L is; the permutation happens on the shared-memory side,
// where a thread finds the place of its word's first element (two multiply-high divisions) and walks on from there: a
// step along the line, and at its end a jump to the next line, at the plane's end to the next plane.
// Bound by that index arithmetic (flat runs with the two divisions for every element, and lines of a group of lanes, were
// slower).  37 x 53 maps, 8 x 192 planes, bf16: scan 32 -> 21 us, merge 48 -> 22 us; fp32 32 -> 22, 49 -> 26 us against the
// single-element form of the plane kernels.
// The rows of the routes may be padded to a multiple of eight elements (`stride` > L), which gives the kernels behind them
// aligned rows whatever L is: the run is then taken over the padded rows, whose words never cross planes, and the
// padding is written as zero.
#pragma once
#include "common.cuh"

namespace ss2d {

constexpr int kWordBytes = 8;
struct Walk {            // constants of a walk over the lines of shared planes
    int len, lines, plane;         // elements per line, lines per plane, elements of the run per plane (with padding)
    unsigned magic_len, magic_plane;
    int o0, line, step, next;      // place of element j of line i of plane p: o0 + i * line + j * step + p * next
};
struct Place { int at, j, i; };
__device__ __forceinline__ int flat_div(int n, unsigned magic) { return magic ? (int)__umulhi((unsigned)n, magic) : n; }
__device__ __forceinline__ Place place_of(const Walk& w, int f) {
    const int p = flat_div(f, w.magic_plane), l = f - p * w.plane, i = flat_div(l, w.magic_len), j = l - i * w.len;
    return {w.o0 + i * w.line + j * w.step + p * w.next, j, i};
}
__device__ __forceinline__ void advance(const Walk& w, Place& q) {
    q.at += w.step;
    if (++q.j == w.len) {
        q.j = 0;
        q.at += w.line - w.len * w.step;
        if (++q.i == w.lines && w.len * w.lines == w.plane) { q.i = 0; q.at += w.next - w.lines * w.line; }
    }
}
template <typename T> union Word { T e[kWordBytes / sizeof(T)]; uint2 w; };
template <typename T> __device__ __forceinline__ int phase_of(const T* p) { return (int)((reinterpret_cast<uintptr_t>(p) & (kWordBytes - 1)) / sizeof(T)); }
template <typename T> __device__ __forceinline__ void load_word(Word<T>& v, const T* __restrict__ run, int f, int n) {
    constexpr int E = kWordBytes / (int)sizeof(T);
    if (f >= 0 && f + E <= n) v.w = __ldg(reinterpret_cast<const uint2*>(run + f));
    else {
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (f + e >= 0 && f + e < n) v.e[e] = run[f + e];
    }
}
template <typename T> __device__ __forceinline__ void store_word(const Word<T>& v, T* __restrict__ run, int f, int n) {
    constexpr int E = kWordBytes / (int)sizeof(T);
    if (f >= 0 && f + E <= n) *reinterpret_cast<uint2*>(run + f) = v.w;
    else {
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (f + e >= 0 && f + e < n) run[f + e] = v.e[e];
    }
}
// A run of n elements of global memory into shared planes, and back.
template <typename T> __device__ __forceinline__ void run_in(const Walk& w, const T* __restrict__ run, int n, T* sm) {
    constexpr int E = kWordBytes / (int)sizeof(T), kFlight = 4;
    const int step = E * blockDim.x;
    for (int f0 = E * (int)threadIdx.x - phase_of(run); f0 < n; f0 += kFlight * step) {
        Word<T> v[kFlight];
#pragma unroll
        for (int i = 0; i < kFlight; ++i) load_word(v[i], run, f0 + i * step, n);
#pragma unroll
        for (int i = 0; i < kFlight; ++i) {
            const int f = f0 + i * step;
            if (f >= n) break;
            Place q = place_of(w, max(f, 0));
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (f + e >= 0) {
                    if (f + e < n && q.i < w.lines) sm[q.at] = v[i].e[e];
                    advance(w, q);
                }
        }
    }
}
template <typename T> __device__ __forceinline__ void run_out(const Walk& w, const T* sm, T* __restrict__ run, int n) {
    constexpr int E = kWordBytes / (int)sizeof(T);
    for (int f = E * (int)threadIdx.x - phase_of(run); f < n; f += E * blockDim.x) {
        Place q = place_of(w, max(f, 0));
        Word<T> v;
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (f + e >= 0) {
                if (f + e < n) v.e[e] = q.i < w.lines ? sm[q.at] : static_cast<T>(0.f);
                advance(w, q);
            }
        store_word(v, run, f, n);
    }
}

struct FlatRoute { int col_like, h_up, w_up; };      // walked by column; h (w) rises along the route
struct FlatArgs {
    const void* in;
    void* out;
    int C, H, W, L, PP, blocks;                      // blocks: CTAs per image
    int stride;                                      // elements between the rows of a route
    FlatRoute route[4];
    unsigned magic_H, magic_W, magic_L, magic_S;         // S: stride
};

// Route k over row-major shared planes of pitch W | 1.
__device__ __forceinline__ Walk route_walk(const FlatArgs& a, int k) {
    const FlatRoute m = a.route[k];
    const int H = a.H, W = a.W, Wp = W | 1, Lp = H * Wp;
    if (m.col_like)
        return {H, W, a.stride, a.magic_H, a.magic_S, (m.w_up ? 0 : W - 1) + (m.h_up ? 0 : (H - 1) * Wp), m.w_up ? 1 : -1, m.h_up ? Wp : -Wp, Lp};
    if (!m.w_up) return {W, H, a.stride, a.magic_W, a.magic_S, (H - 1) * Wp + W - 1, -Wp, -1, Lp};
    return {W, H, a.stride, a.magic_W, a.magic_S, 0, Wp, 1, Lp};
}

template <typename T>
__global__ void __launch_bounds__(512) cross_scan_flat_kernel(const FlatArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    T* sm = reinterpret_cast<T*>(smraw);             // [PP][H][W | 1]
    const int b = blockIdx.x / a.blocks, c0 = (blockIdx.x - b * a.blocks) * a.PP, np = min(a.PP, a.C - c0);
    const int L = a.L, H = a.H, W = a.W, Wp = W | 1, Lp = H * Wp, n = np * L;
    run_in<T>({W, H, L, a.magic_W, a.magic_L, 0, Wp, 1, Lp}, (const T*)a.in + ((long long)b * a.C + c0) * L, n, sm);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k)
        run_out<T>(route_walk(a, k), sm, (T*)a.out + ((long long)(b * 4 + k) * a.C + c0) * a.stride, np * a.stride);
}

// Rows (B, 4, C, H x W), `stride` elements apart: row (k, c) is brought from pixel order into the order of route k (or back,
// with `back`).  The CrossScan of rows that each belong to one route.
template <typename T>
__global__ void __launch_bounds__(512) cross_rows_kernel(const FlatArgs a, const int back) {
    extern __shared__ __align__(16) unsigned char smraw[];
    T* sm = reinterpret_cast<T*>(smraw);             // [PP][H][W | 1]
    const int bk = blockIdx.x / a.blocks, k = bk & 3, c0 = (blockIdx.x - bk * a.blocks) * a.PP, np = min(a.PP, a.C - c0);
    const int H = a.H, W = a.W, Wp = W | 1, n = np * a.stride;
    const long long at = ((long long)bk * a.C + c0) * a.stride;
    const Walk by_row = {W, H, a.stride, a.magic_W, a.magic_S, 0, Wp, 1, H * Wp}, by_route = route_walk(a, k);
    run_in<T>(back ? by_route : by_row, (const T*)a.in + at, n, sm);
    __syncthreads();
    run_out<T>(back ? by_row : by_route, sm, (T*)a.out + at, n);
}

// Sum of four routes in the association order of the reference's additions, rounded to the storage type after each.
template <typename T> __device__ __forceinline__ T flat_add(T x, T y) { return from_f<T>(to_f<T>(x) + to_f<T>(y)); }
template <typename T> __device__ __forceinline__ T flat_sum(int scans, T x0, T x1, T x2, T x3) {
    if (scans == 0 || scans == 2) return flat_add(flat_add(x0, x2), flat_add(x1, x3));
    if (scans == 3) return flat_add(flat_add(flat_add(x0, x1), x2), x3);
    return from_f<T>(((to_f<T>(x0) + to_f<T>(x1)) + to_f<T>(x2)) + to_f<T>(x3));
}

// The row-like routes are read in place, the column-like ones (at most two) through shared memory.
template <typename T>
__global__ void __launch_bounds__(512) cross_merge_flat_kernel(const FlatArgs a, const int scans) {
    extern __shared__ __align__(16) unsigned char smraw[];
    T* sm = reinterpret_cast<T*>(smraw);             // [column-like route][PP][W][H | 1]
    constexpr int E = kWordBytes / (int)sizeof(T);
    const int b = blockIdx.x / a.blocks, c0 = (blockIdx.x - b * a.blocks) * a.PP, np = min(a.PP, a.C - c0);
    const int L = a.L, S = a.stride, H = a.H, W = a.W, Hp = H | 1, Lp = W * Hp, n = np * L;
    const T* in[4];
    bool col[4], fwd[4], same[4];
    Walk w[4];                                       // of the column-like routes, in the order of the result
    int slots = 0;
    T* __restrict__ out = (T*)a.out + ((long long)b * a.C + c0) * L;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const FlatRoute m = a.route[k];
        in[k] = (const T*)a.in + ((long long)(b * 4 + k) * a.C + c0) * S;
        col[k] = m.col_like != 0;
        fwd[k] = m.w_up != 0;
        same[k] = S == L && phase_of(in[k]) == phase_of(out);
        w[k] = {W, H, L, a.magic_W, a.magic_L, 0, 0, 0, 0};
        if (!col[k]) continue;
        run_in<T>({H, W, S, a.magic_H, a.magic_S, 0, Hp, 1, Lp}, in[k], np * S, sm + slots * a.PP * Lp);
        w[k] = {W, H, L, a.magic_W, a.magic_L, slots * a.PP * Lp + (m.w_up ? 0 : (W - 1) * Hp) + (m.h_up ? 0 : H - 1), m.h_up ? 1 : -1,
                m.w_up ? Hp : -Hp, Lp};
        ++slots;
    }
    __syncthreads();
    for (int f = E * (int)threadIdx.x - phase_of(out); f < n; f += E * blockDim.x) {
        Word<T> v[4], r;
        const int f1 = max(f, 0), p = flat_div(f1, a.magic_L), l = f1 - p * L;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (col[k]) {
                Place q = place_of(w[k], f1);
#pragma unroll
                for (int e = 0; e < E; ++e)
                    if (f + e >= 0) {
                        if (f + e < n) v[k].e[e] = sm[q.at];
                        advance(w[k], q);
                    }
            } else if (fwd[k]) {
                if (same[k]) load_word(v[k], in[k], f, n);
                else {
                    int at = p * S + l, gone = l;
#pragma unroll
                    for (int e = 0; e < E; ++e)
                        if (f + e >= 0) {
                            if (f + e < n) v[k].e[e] = __ldg(in[k] + at);
                            ++at;
                            if (++gone == L) { gone = 0; at += S - L; }
                        }
                }
            } else {
                int at = p * S + L - 1 - l, gone = l;
#pragma unroll
                for (int e = 0; e < E; ++e)
                    if (f + e >= 0) {
                        if (f + e < n) v[k].e[e] = __ldg(in[k] + at);
                        --at;
                        if (++gone == L) { gone = 0; at += S + L; }
                    }
            }
        }
#pragma unroll
        for (int e = 0; e < E; ++e) r.e[e] = flat_sum<T>(scans, v[0].e[e], v[1].e[e], v[2].e[e], v[3].e[e]);
        store_word(r, out, f, n);
    }
}

}  // namespace ss2d
