// CrossScan / CrossMerge of whole planes, of any size that shared memory holds and any alignment.
//
// The planes of an image are neighbours in the map and in every route, so the PP planes of a CTA are ONE run in each of them.
// Runs are brought into shared memory as they lie, in 16-byte pieces by asynchronous copies (all of a CTA's input is under way
// at once, which is what a merge of four routes needs), and the permutation is the address of a shared-memory read.  A
// thread takes every blockDim-th pixel: its next place in the transposed order follows by an addition, and one more
// at the end of a line.
// Bound, where the planes are many: HBM (fp32, 32 x 96 planes of 56 x 56: scan 31.4 us, 4.9 TB/s, merge 32.5).  fp32 / bf16 against the forms that
// gathered whole vectors of the routes, with a place and a division for each: 64 x 192 planes of 28 x 28 merge 55 -> 34 / 49 -> 31 us;
// 8 x 192 of 37 x 53 scan 24.9 -> 12.8 / 24.6 -> 11.4, merge 26.1 -> 17.1 / 23.9 -> 13.4 (a second, half-empty round of CTAs); 128 x 768 of
// 7 x 7 scan 37.8 -> 19.4 / 36.5 -> 17.0, merge 42 -> 25 / 37 -> 19.
#pragma once
#include "cross_pieces.cuh"

namespace ss2d {

struct RunArgs {
    const void* in;
    void* out;
    int C, H, W, L, S;                               // S: elements between the rows of a route
    int PP, blocks, slot;                            // planes of a CTA, CTAs per image, elements of a run's place in shared memory
    int pad;                                         // elements between the lines of the transposed order's source in shared memory
};

// A run of n elements into shared memory (16-byte aligned, with room for 32 bytes more): whole pieces asynchronously, the elements in
// front of the first and behind the last one by one.  Returns where element 0 lies.
// pad: the run is of lines of `line` elements, whole pieces that start on one, which are set `pad` elements apart.
template <typename T> __device__ __forceinline__ T* run_fetch(const T* __restrict__ run, int n, T* sm, int line, int pad) {
    constexpr int E = 16 / (int)sizeof(T);
    const int t = threadIdx.x;
    if (pad) {
        const int per = line / E;                    // pieces of a line
        int l = t / per, j = t - l * per;
        const int sl = (int)blockDim.x / per, sj = (int)blockDim.x - sl * per;
        for (int i = t; i < n / E; i += blockDim.x) {
            piece_copy_async(sm + l * (line + pad) + j * E, run + i * E);
            l += sl; j += sj;
            if (j >= per) { j -= per; ++l; }
        }
        return sm;
    }
    const int ph = (int)((reinterpret_cast<uintptr_t>(run) & 15) / sizeof(T));
    const int head = min(n, (E - ph) & (E - 1)), pieces = (n - head) / E, tail = head + pieces * E;
    T* to = sm + ph;
    for (int i = t; i < pieces; i += blockDim.x) piece_copy_async(to + head + i * E, run + head + i * E);
    if (t < head) to[t] = run[t];
    else if (t >= 32 && t - 32 < n - tail) to[tail + t - 32] = run[tail + t - 32];
    return to;
}

// A thread's walk over the pixels of the planes with lines of `fast` pixels, `unit` pixels of a line at a time: l, the place in that order,
// and q, the place in the transposed order, whose lines (`slow` pixels) lie `slow + pad` elements apart; both inside the plane p.
struct RunWalk {
    int fast, slow, L, f, l, step, step_l, q, q_step, q_wrap, p, p_step;
    __device__ __forceinline__ RunWalk(int fast_, int slow_, int pad, int unit) : fast(fast_), slow(slow_), L(fast_ * slow_) {
        const int nt = (int)blockDim.x * unit, t = (int)threadIdx.x * unit;
        p_step = nt / L; step_l = nt - p_step * L;
        q = step_l / fast;
        step = step_l - q * fast; q_step = step * (slow + pad) + q; q_wrap = 1 - fast * (slow + pad);
        p = t / L; l = t - p * L;
        q = l / fast; f = l - q * fast;
        q += f * (slow + pad);
    }
    __device__ __forceinline__ void next() {
        f += step; l += step_l; q += q_step; p += p_step;
        if (f >= fast) { f -= fast; q += q_wrap; }
        if (l >= L) { l -= L; ++p; q -= slow; }
    }
};

template <typename T> __device__ __forceinline__ void run_pad(const RunArgs& a, int np, T* rows) {      // the padding of a route's rows
    const int pad = a.S - a.L;
    if (pad)
        for (int i = threadIdx.x; i < np * pad; i += blockDim.x) rows[i / pad * a.S + a.L + i % pad] = static_cast<T>(0.f);
}

// V: pixels of a thread at a time, 1, or 2 of 16-bit maps with even sides whose planes start on words.
template <typename T, int SCANS, int V, bool kPad>
__global__ void __launch_bounds__(512) cross_scan_runs_kernel(const RunArgs a) {
    follow_previous();
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr bool kCols = SCANS == 0 || SCANS == 3;
    const int b = blockIdx.x / a.blocks, c0 = (blockIdx.x - b * a.blocks) * a.PP, np = min(a.PP, a.C - c0);
    const int L = a.L, S = a.S, H = a.H, W = a.W, pad = kPad ? a.pad : 0, n = np * L, Wp = W + pad;
    const T* sm = run_fetch((const T*)a.in + ((long long)b * a.C + c0) * L, n, reinterpret_cast<T*>(smraw), W, pad);
    T* out[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        out[k] = (T*)a.out + (((long long)b * 4 + k) * a.C + c0) * S;
        run_pad(a, np, out[k]);
    }
    piece_wait();
    {                               // the row-like routes run with the map or against it
        RunWalk w(W, H, 0, V);
#pragma unroll 4
        for (int at = threadIdx.x * V; at < n; at += blockDim.x * V, w.next()) {
            const int o = w.p * S, r = o + L - V - w.l;
            const T* from = sm + at + (kPad ? (w.p * H + w.q - w.f * H) * pad : 0);
            Pixels<T, V> v;
            v.load(from);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (kCols && k % 2) continue;
                if (SCANS == 1 || k < (SCANS == 2 ? 2 : 1)) v.store(out[k] + (o + w.l));
                else v.turned().store(out[k] + r);
            }
        }
    }
    if constexpr (kCols) {          // and the column-like ones with or against the transposed map (of scans 3: its columns from the last)
        RunWalk w(H, W, pad, V);
#pragma unroll 4
        for (int at = threadIdx.x * V; at < n; at += blockDim.x * V, w.next()) {
            const int o = w.p * S;
            const T* from = sm + w.p * H * Wp + (SCANS == 0 ? w.q : 2 * w.f * Wp + W - 1 - w.q);
            Pixels<T, V> v;
#pragma unroll
            for (int e = 0; e < V; ++e) v.set(e, from[e * Wp]);
            v.store(out[1] + (o + w.l));
            v.turned().store(out[3] + (o + L - V - w.l));
        }
    }
}

// Rows (B, 4, C, H x W), S elements apart: row (k, c) is brought from pixel order into the order of route k (or back, with
// `back`).  The CrossScan of rows that each belong to one route.
template <typename T>
__global__ void __launch_bounds__(512) cross_rows_kernel(const RunArgs a, const int scans, const int back) {
    follow_previous();
    extern __shared__ __align__(16) unsigned char smraw[];
    const int bk = blockIdx.x / a.blocks, k = bk & 3, c0 = (blockIdx.x - bk * a.blocks) * a.PP, np = min(a.PP, a.C - c0);
    const int L = a.L, S = a.S, H = a.H, W = a.W, n = np * L;
    const long long row0 = ((long long)bk * a.C + c0) * S;
    const T* sm = run_fetch((const T*)a.in + row0, (np - 1) * S + L, reinterpret_cast<T*>(smraw), 0, 0);
    T* __restrict__ out = (T*)a.out + row0;
    run_pad(a, np, out);
    piece_wait();
    // in the order of the result; routes 2 and 3 are 0 and 1 turned round, and scans 3 take the columns from the last
    const bool col = k % 2 && (scans == 0 || scans == 3), turned = k >= 2 && scans != 1, by_col = col && !back, mirror = col && scans == 3;
    RunWalk w(by_col ? H : W, by_col ? W : H, 0, 1);
#pragma unroll 4
    for (int at = threadIdx.x; at < n; at += blockDim.x, w.next()) {
        int from = col ? w.q : w.l, to = w.l;
        if (mirror) from = back ? (W - 1) * H + 2 * (w.q - w.f * H) - w.q : 2 * w.f * W + W - 1 - w.q;
        if (turned) { if (by_col) to = L - 1 - to; else from = L - 1 - from; }
        out[w.p * S + to] = sm[w.p * S + from];
    }
}

// V: as above, of routes that start on words.
template <typename T, int SCANS, int V>
__global__ void __launch_bounds__(512) cross_merge_runs_kernel(const RunArgs a) {
    follow_previous();
    extern __shared__ __align__(16) unsigned char smraw[];
    T* sm = reinterpret_cast<T*>(smraw);
    constexpr bool kCols = SCANS == 0 || SCANS == 3;
    const int b = blockIdx.x / a.blocks, c0 = (blockIdx.x - b * a.blocks) * a.PP, np = min(a.PP, a.C - c0);
    const int L = a.L, S = a.S, H = a.H, W = a.W, pad = a.pad, Hp = H + pad;
    const T* in[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        in[k] = run_fetch((const T*)a.in + (((long long)b * 4 + k) * a.C + c0) * S, (np - 1) * S + L, sm + k * a.slot, H, kCols && k % 2 ? pad : 0);
    T* __restrict__ out = (T*)a.out + ((long long)b * a.C + c0) * L;
    piece_wait();
    const int n = np * L, last = W * Hp - pad - 1;
    RunWalk w(W, H, pad, V);
#pragma unroll 4
    for (int at = threadIdx.x * V; at < n; at += blockDim.x * V, w.next()) {
        const int o = w.p * S, f = o + w.l, r = o + L - V - w.l, oc = o + w.p * W * pad;      // padded lines: S = L
        const auto row = [&](int k) {                // V pixels of a row-like route, in the order of the map
            const bool with = SCANS == 1 || k < (SCANS == 2 ? 2 : 1);
            Pixels<T, V> x;
            x.load(in[k] + (with ? f : r));
            return with ? x : x.turned();
        };
        const Pixels<T, V> v0 = row(0), v2 = row(2);
        Pixels<T, V> v1, v3, y;
        if constexpr (!kCols) { v1 = row(1); v3 = row(3); }
        // q = w * Hp + h; route 3 is route 1 turned round; of scans 3 route 1 takes the columns from the last
        const int q = SCANS == 0 ? w.q : (W - 1) * Hp + 2 * (w.q - w.f * Hp) - w.q;
#pragma unroll
        for (int e = 0; e < V; ++e) {
            T x1, x3;
            if constexpr (kCols) {
                const int qe = q + (SCANS == 0 ? e * Hp : -e * Hp);
                x1 = in[1][oc + qe]; x3 = in[3][oc + last - qe];
            } else { x1 = v1.at(e); x3 = v3.at(e); }
            y.set(e, flat_sum<T>(SCANS, v0.at(e), x1, v2.at(e), x3));
        }
        y.store(out + at);
    }
}

}  // namespace ss2d
