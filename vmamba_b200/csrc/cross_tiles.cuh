// CrossScan / CrossMerge of planes that are taken in tiles, of any size and alignment, single elements.
//
// The pixels of a tile are walked twice: in the order of the map (w fastest), where the lanes of a warp are neighbours in the map
// and in the row-like routes, and with h fastest, where they are neighbours in the column-like ones; what the two orders
// exchange lies in shared memory.  A thread takes every 256th pixel: its next places follow from the last ones by an
// addition each, and one more at the end of a line.  Every access is coalesced whatever the sides are.
// Bound: the loads in flight, and partial sectors where rows start anywhere.  fp32 / bf16, against a place by two products and a test per
// element in tiles of 32 x 32 (and, of the merge, against 16-byte copies into tiles of 64 x 64 where rows are whole vectors): 256 planes of
// 256 x 256 merge 65 -> 59 / 53 -> 43 us (5.7 TB/s), 256 of 247 x 231 merge 88 -> 53 / 107 -> 54, scan 92 -> 88 / 62 -> 49.
#pragma once
#include "cross_pieces.cuh"

namespace ss2d {

struct TileRoute { int base, sh, sw, col; };         // place of pixel (h, w): base + sh * h + sw * w; col: |sh| = 1, else |sw| = 1
struct TileArgs {
    const void* in;
    void* out;
    const void* end;                                 // of `in`
    int C, H, W, L, S;                               // S: elements between the rows of a route
    int TH, TW, tiles_h, tiles_w, pitch;             // pitch: of the tile's rows in shared memory
    TileRoute route[4];
};
constexpr int kTileThreads = 256, kTileFlight = 4;   // pixels of a thread whose loads are under way together

struct TilePlace {                                   // of a CTA
    int b, c, h0, w0, th, tw;
    __device__ __forceinline__ explicit TilePlace(const TileArgs& a) {
        const int ty = blockIdx.x / a.tiles_w, plane = ty / a.tiles_h;
        b = plane / a.C; c = plane - b * a.C;
        h0 = (ty - plane * a.tiles_h) * a.TH; w0 = ((int)blockIdx.x - ty * a.tiles_w) * a.TW;
        th = min(a.TH, a.H - h0); tw = min(a.TW, a.W - w0);
    }
    __device__ __forceinline__ int origin(const TileRoute& m) const { return m.base + m.sh * h0 + m.sw * w0; }
};

// The pixels of a tile with `kByRow ? w : h` fastest, V of a line at a time.  Per pixel: its place in shared memory (rows of `pitch`) and in global memory,
// where a step along h is `gh` elements and one along w `gw`.
template <bool kByRow, int V> struct TileWalk {
    int fast, f, step, sm, sm_step, sm_wrap, g, g_step, g_wrap;
    __device__ __forceinline__ TileWalk(const TilePlace& t, int pitch, int gh, int gw) {
        fast = kByRow ? t.tw : t.th;
        const int sf = kByRow ? 1 : pitch, ss = kByRow ? pitch : 1, gf = kByRow ? gw : gh, gs = kByRow ? gh : gw;
        int q = kTileThreads * V / fast;
        step = kTileThreads * V - q * fast;
        sm_step = step * sf + q * ss; g_step = step * gf + q * gs;
        sm_wrap = ss - fast * sf; g_wrap = gs - fast * gf;
        q = (int)threadIdx.x * V / fast;
        f = (int)threadIdx.x * V - q * fast;
        sm = f * sf + q * ss; g = f * gf + q * gs;
    }
    __device__ __forceinline__ void next() {
        f += step; sm += sm_step; g += g_step;
        if (f >= fast) { f -= fast; sm += sm_wrap; g += g_wrap; }
    }
};

// load(i, sm, g), then use(i, sm, g), for kTileFlight places of the walk at a time (i: their number)
template <bool kByRow, int V, typename F, typename U> __device__ __forceinline__ void tile_for_each(TileWalk<kByRow, V> w, int n, F load, U use) {
    constexpr int kStep = kTileThreads * V;
    int at = threadIdx.x * V, sm[kTileFlight], g[kTileFlight];
    for (; at + (kTileFlight - 1) * kStep < n; at += kTileFlight * kStep) {
#pragma unroll
        for (int i = 0; i < kTileFlight; ++i, w.next()) { sm[i] = w.sm; g[i] = w.g; load(i, sm[i], g[i]); }
#pragma unroll
        for (int i = 0; i < kTileFlight; ++i) use(i, sm[i], g[i]);
    }
#pragma unroll
    for (int i = 0; i < kTileFlight - 1; ++i, w.next())
        if (at + i * kStep < n) { sm[i] = w.sm; g[i] = w.g; load(i, sm[i], g[i]); }
#pragma unroll
    for (int i = 0; i < kTileFlight - 1; ++i)
        if (at + i * kStep < n) use(i, sm[i], g[i]);
}

// The map's rows of the tile come as the aligned 16-byte pieces around them, asynchronously, into shared rows of whole pieces, so that
// a row keeps the phase it has in global memory; pieces that reach beyond the map are taken by single elements.
template <typename T>
__global__ void __launch_bounds__(kTileThreads) cross_scan_tiles_kernel(const TileArgs a) {
    follow_previous();
    extern __shared__ __align__(16) unsigned char smraw[];
    T* sm = reinterpret_cast<T*>(smraw);
    constexpr int E = 16 / (int)sizeof(T);
    const TilePlace t(a);
    const int n = t.th * t.tw, W = a.W, P = a.pitch;
    const T* __restrict__ x = (const T*)a.in + ((long long)t.b * a.C + t.c) * a.L + t.h0 * W + t.w0;
    const int phase0 = (int)((reinterpret_cast<uintptr_t>(x) & 15) / sizeof(T));
    const auto phase = [&](int h) { return (phase0 + h * W) & (E - 1); };
    {
        const int per = (t.tw + 2 * E - 2) / E;      // pieces of a row at most
        int h = (int)threadIdx.x / per, j = (int)threadIdx.x - h * per;
        const int sh = kTileThreads / per, sj = kTileThreads - sh * per;
        while (h < t.th) {
            const int e = j * E - phase(h);          // column at the start of the piece
            const T* from = x + h * W + e;
            T* to = sm + h * P + j * E;
            if (e < t.tw) {
                if (from >= (const T*)a.in && from + E <= (const T*)a.end) piece_copy_async(to, from);
                else
                    for (int i = 0; i < E; ++i)
                        if (e + i >= 0 && e + i < t.tw) to[i] = from[i];
            }
            h += sh; j += sj;
            if (j >= per) { j -= per; ++h; }
        }
    }
    T* out[4];
    bool any_col = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        out[k] = (T*)a.out + ((long long)(t.b * 4 + k) * a.C + t.c) * a.L + t.origin(a.route[k]);
        any_col = any_col || a.route[k].col;
    }
    piece_wait();
    const auto walk = [&](int fast, bool cols) {     // lines of `fast` pixels
        int s = (int)threadIdx.x / fast, f = (int)threadIdx.x - s * fast;
        const int ss = kTileThreads / fast, sf = kTileThreads - ss * fast;
#pragma unroll 4
        for (int at = threadIdx.x; at < n; at += kTileThreads) {
            const int h = cols ? f : s, w = cols ? s : f;
            const T v = sm[h * P + phase(h) + w];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if ((a.route[k].col != 0) == cols) out[k][a.route[k].sh * h + a.route[k].sw * w] = v;
            f += sf; s += ss;
            if (f >= fast) { f -= fast; ++s; }
        }
    };
    walk(t.tw, false);
    if (any_col) walk(t.th, true);
}

// The row-like routes are read where they are summed, the column-like ones (at most two: 1 and 3) through shared memory, as
// their sum where the order of the additions has one (scans 0).  V: pixels of a thread at a time, 1, or 2 of 16-bit maps with
// even sides whose planes start on words.
template <typename T, int SCANS, int V>
__global__ void __launch_bounds__(kTileThreads, 6) cross_merge_tiles_kernel(const TileArgs a) {
    follow_previous();
    extern __shared__ __align__(16) unsigned char smraw[];
    T* sm = reinterpret_cast<T*>(smraw);             // [slot][th][pitch]
    constexpr bool kCols = SCANS == 0 || SCANS == 3;
    const TilePlace t(a);
    const int n = t.th * t.tw, slot = t.th * a.pitch, P = a.pitch;
    const T* in[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) in[k] = (const T*)a.in + ((long long)(t.b * 4 + k) * a.C + t.c) * a.S + t.origin(a.route[k]);
    using Unit = Pixels<T, V>;
    Unit v[4][kTileFlight];
    if constexpr (kCols) {                           // route 3 is route 1 turned round
        tile_for_each(TileWalk<false, V>(t, P, a.route[1].sh, a.route[1].sw), n,
                      [&](int i, int, int g) { v[1][i].load(in[1] + g); v[3][i].load(in[3] - g - (V - 1)); },
                      [&](int i, int s, int) {
#pragma unroll
                          for (int e = 0; e < V; ++e) {
                              const T x = v[1][i].at(e), y = v[3][i].at(V - 1 - e);
                              if constexpr (SCANS == 0) sm[s + e * P] = flat_add(x, y);
                              else { sm[s + e * P] = x; sm[slot + s + e * P] = y; }
                          }
                      });
        __syncthreads();
    }
    T* __restrict__ out = (T*)a.out + ((long long)t.b * a.C + t.c) * a.L + t.h0 * a.W + t.w0;
    constexpr int kTurned = SCANS == 1 ? 4 : SCANS == 2 ? 2 : 1;      // routes from here on run against the map
    tile_for_each(TileWalk<true, V>(t, P, a.W, 1), n,
                  [&](int i, int, int g) {
#pragma unroll
                      for (int k = 0; k < 4; ++k)
                          if (!kCols || k % 2 == 0) v[k][i].load(in[k] + (k < kTurned ? g : -g - (V - 1)));
                  },
                  [&](int i, int s, int g) {
                      const auto route = [&](int k, int e) { return v[k][i].at(k < kTurned ? e : V - 1 - e); };
                      Unit y;
#pragma unroll
                      for (int e = 0; e < V; ++e) {
                          if constexpr (SCANS == 0) y.set(e, flat_add(flat_add(route(0, e), route(2, e)), sm[s + e]));
                          else if constexpr (SCANS == 3) y.set(e, flat_sum<T>(3, route(0, e), sm[s + e], route(2, e), sm[slot + s + e]));
                          else y.set(e, flat_sum<T>(SCANS, route(0, e), route(1, e), route(2, e), route(3, e)));
                      }
                      y.store(out + g);
                  });
}

}  // namespace ss2d
