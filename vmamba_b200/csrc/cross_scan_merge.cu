// CrossScan / CrossMerge as stand-alone tensor-to-tensor operators (channel-first).
//
// Every route is an index map  (h, w) -> l  that is contiguous either along w ("row-like") or along h ("column-like").
// Planes that fit are taken whole (cross_runs.cuh), larger ones in tiles (cross_tiles.cuh, and the pair kernel below).
// Data movement only: results are bit-identical to indexing.
#include <algorithm>

#include "common.cuh"
#include "cross_runs.cuh"
#include "cross_tiles.cuh"

namespace ss2d {

struct RouteMap {
    // l = base + sh * h + sw * w ; col_like: |sh| == 1 (contiguous along h)
    long long base, sh, sw;
    int col_like;
};

__host__ __device__ inline RouteMap route_map(int scans, int k, long long H, long long W) {
    const long long L = H * W;
    RouteMap m;
    auto row_f = [&]() { m.base = 0; m.sh = W; m.sw = 1; m.col_like = 0; };
    auto row_r = [&]() { m.base = L - 1; m.sh = -W; m.sw = -1; m.col_like = 0; };
    auto col_f = [&]() { m.base = 0; m.sh = 1; m.sw = H; m.col_like = 1; };
    auto col_r = [&]() { m.base = L - 1; m.sh = -1; m.sw = -H; m.col_like = 1; };
    if (scans == 0) { if (k == 0) row_f(); else if (k == 1) col_f(); else if (k == 2) row_r(); else col_r(); }
    else if (scans == 1) row_f();
    else if (scans == 2) { if (k < 2) row_f(); else row_r(); }
    else {
        // rotations: k=1 -> l = (W-1-w)*H + h ; k=3 -> l = w*H + (H-1-h)
        if (k == 0) row_f();
        else if (k == 1) { m.base = (W - 1) * H; m.sh = 1; m.sw = -H; m.col_like = 1; }
        else if (k == 2) row_r();
        else { m.base = H - 1; m.sh = -1; m.sw = H; m.col_like = 1; }
    }
    return m;
}

struct CrossArgs {
    const void* in;
    void* out;
    long long C, H, W, tiles_h, tiles_w;
    RouteMap route[4];
};

// 16-bit maps with even H and W: a thread moves PAIRS of elements as one 32-bit word.  (512 planes of 128 x 128: 19 us; as single
// elements 29.)  Tile: 64 x 64 elements = 32 words along the fast index of either orientation; a reversed route writes the
// pair at the mirrored address with its halves swapped.
constexpr int kPairTile = 64;
__global__ void __launch_bounds__(256) cross_scan_pair_kernel(const CrossArgs a) {
    follow_previous();
    __shared__ __align__(4) uint16_t tile[kPairTile][kPairTile + 2];       // pitch 33 words
    const unsigned t = blockIdx.x, tiles_w = (unsigned)a.tiles_w, tiles_h = (unsigned)a.tiles_h, C = (unsigned)a.C;
    const unsigned tw = t % tiles_w, rest = t / tiles_w, th = rest % tiles_h, plane = rest / tiles_h;
    const unsigned b = plane / C, c = plane - b * C;
    const int H = (int)a.H, W = (int)a.W, L = H * W;
    const uint16_t* __restrict__ x = (const uint16_t*)a.in + (long long)plane * L;
    const int h0 = (int)th * kPairTile, w0 = (int)tw * kPairTile;
    const int tx = threadIdx.x, ty = threadIdx.y;          // 32 x 8
#pragma unroll
    for (int j = 0; j < kPairTile; j += 8) {
        const int h = h0 + ty + j, w = w0 + 2 * tx;
        if (h < H && w < W) *reinterpret_cast<uint32_t*>(&tile[ty + j][2 * tx]) = *reinterpret_cast<const uint32_t*>(x + h * W + w);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int base = (int)a.route[k].base, sh = (int)a.route[k].sh, sw = (int)a.route[k].sw;
        const bool col_like = a.route[k].col_like != 0;
        uint16_t* __restrict__ y = (uint16_t*)a.out + ((long long)(b * 4 + k) * C + c) * L;
#pragma unroll
        for (int j = 0; j < kPairTile; j += 8) {
            // the pair runs along w (row-like) or along h (column-like); `step` is the route's stride along the pair
            const int lh = col_like ? 2 * tx : ty + j, lw = col_like ? ty + j : 2 * tx;
            const int h = h0 + lh, w = w0 + lw;
            if (h < H && w < W) {
                const uint32_t e0 = col_like ? tile[lh][lw] : tile[lh][lw];
                const uint32_t e1 = col_like ? tile[lh + 1][lw] : tile[lh][lw + 1];
                const int step = col_like ? sh : sw;               // +1 or -1
                const int l0 = base + sh * h + sw * w;
                if (step > 0) *reinterpret_cast<uint32_t*>(y + l0) = e0 | (e1 << 16);
                else *reinterpret_cast<uint32_t*>(y + l0 - 1) = e1 | (e0 << 16);
            }
        }
    }
}

// How the tile kernels cut a plane.  Scan: sides of at most 64 pixels, shared rows of an odd number of pieces.  Merge: whole rows, or equal
// parts of at most 128 pixels, of 32 lines or 4 096 pixels; `slots` tiles in shared memory.
static bool plan_tiles(const ss2d_cross_params* p, int slots, TileArgs& a, size_t& smem) {
    const int es = (int)dtype_size(p->dtype), E = 16 / es;
    const auto part = [](long long n, long long most, long long unit) {      // equal parts
        const long long parts = (n + most - 1) / most, each = (n + parts - 1) / parts;
        return (int)((each + unit - 1) / unit * unit);
    };
    a.in = p->in; a.out = p->out; a.end = (const char*)p->in + p->B * p->C * p->H * p->W * es;      // of a map
    a.C = (int)p->C; a.H = (int)p->H; a.W = (int)p->W; a.L = (int)(p->H * p->W);
    a.S = p->route_stride ? (int)p->route_stride : a.L;
    if (slots == 0) {
        a.TH = part(p->H, 64, 8); a.TW = part(p->W, 64, 8);
        a.pitch = ((a.TW + 2 * E - 2) / E | 1) * E;
    } else {
        a.TW = p->W > 160 ? part(p->W, 128, 2) : a.W;          // even, for pairs
        a.TH = part(p->H, std::max(32, 4096 / a.TW), 2);
        a.pitch = es == 4 ? a.TW | 1 : a.TW + (6 - a.TW % 4) % 4;            // columns without bank conflicts
        while (a.TH * a.pitch * es * slots > 48 * 1024) a.TH = (a.TH + 3) / 4 * 2;
    }
    a.tiles_h = (a.H + a.TH - 1) / a.TH; a.tiles_w = (a.W + a.TW - 1) / a.TW;
    for (int k = 0; k < 4; ++k) {
        const RouteMap m = route_map(p->scans, k, p->H, p->W);
        a.route[k] = {(int)m.base, (int)m.sh, (int)m.sw, m.col_like};
    }
    smem = (size_t)std::max(slots, 1) * a.TH * a.pitch * es;
    return p->B * p->C * a.tiles_h * a.tiles_w <= 0x7fffffffLL;
}
static unsigned tile_grid(const TileArgs& a, int64_t images) { return (unsigned)(images * a.C * a.tiles_h * a.tiles_w); }
template <typename T>
static int launch_scan_tiles(const TileArgs& a, int64_t B, size_t smem, cudaStream_t st) {
    launch(cross_scan_tiles_kernel<T>, tile_grid(a, B), kTileThreads, smem, st, a);
    count_launch();
    return check_launch();
}
template <typename T, int V>
static int merge_tiles_v(const TileArgs& a, int64_t B, int scans, size_t smem, cudaStream_t st) {
    const unsigned g = tile_grid(a, B);
    if (scans == 0) launch(cross_merge_tiles_kernel<T, 0, V>, g, kTileThreads, smem, st, a);
    else if (scans == 1) launch(cross_merge_tiles_kernel<T, 1, V>, g, kTileThreads, smem, st, a);
    else if (scans == 2) launch(cross_merge_tiles_kernel<T, 2, V>, g, kTileThreads, smem, st, a);
    else launch(cross_merge_tiles_kernel<T, 3, V>, g, kTileThreads, smem, st, a);
    count_launch();
    return check_launch();
}
template <typename T>
static int launch_merge_tiles(const TileArgs& a, int64_t B, int scans, bool pairs, size_t smem, cudaStream_t st) {
    if constexpr (sizeof(T) == 2) {
        if (pairs) return merge_tiles_v<T, 2>(a, B, scans, smem, st);
    }
    return merge_tiles_v<T, 1>(a, B, scans, smem, st);
}

constexpr long long kRunBytes = 72 * 1024, kRunMost = 202 * 1024;       // of shared memory: three CTAs of an SM, one
// How the run kernels take the planes: as many as are 2 048 pixels, one at least, of an image.  `copies`: runs in shared memory, 1 (scan) or 4
// (merge).
static bool plan_runs(const ss2d_cross_params* p, long long images, int copies, long long most, RunArgs& a, int& threads, size_t& smem) {
    const long long L = p->H * p->W, S = p->route_stride ? p->route_stride : L, es = (long long)dtype_size(p->dtype), E = 16 / es;
    // lines of the transposed order's source whose starts share a bank, or two, are set a piece apart
    const long long line = copies == 1 ? p->W : p->H, lines = copies == 1 ? p->H : p->W;
    const bool pad = most != kRunMost && p->scans != 1 && p->scans != 2 && line * es % 64 == 0 && S == L && aligned_to(p->in, 16);
    const auto bytes = [&](long long planes) { return (((planes - 1) * S + L + (pad ? planes * lines * E : 0)) * es + 47) / 16 * 16 * copies; };
    if (bytes(1) > most) return false;
    long long PP = std::max<long long>(1, std::min<long long>(2048 / L, p->C));
    while (PP > 1 && (bytes(PP) > 48 * 1024 || (PP * L > 256 && images * ((p->C + PP - 1) / PP) < 148 * 4))) --PP;
    const long long blocks = (p->C + PP - 1) / PP;
    if (images * blocks > 0x7fffffffLL) return false;
    a.in = p->in; a.out = p->out; a.C = (int)p->C; a.H = (int)p->H; a.W = (int)p->W; a.L = (int)L; a.S = (int)S;
    a.PP = (int)PP; a.blocks = (int)blocks; a.slot = (int)(bytes(PP) / copies / es); a.pad = pad ? (int)E : 0;
    smem = (size_t)bytes(PP);
    threads = PP * L > 4096 ? 512 : PP * L > 1024 ? 256 : 128;
    return true;
}
template <typename T, int SCANS, int V, bool kPad> static int launch_scan_runs(const RunArgs& a, int64_t B, int threads, size_t smem, cudaStream_t st) {
    auto k = cross_scan_runs_kernel<T, SCANS, V, kPad>;
    if (const int rc = allow_dynamic_smem(k, smem)) return rc;
    launch(k, (unsigned)(B * a.blocks), threads, smem, st, a);
    count_launch();
    return check_launch();
}
template <typename T, int SCANS, int V> static int launch_merge_runs(const RunArgs& a, int64_t B, int threads, size_t smem, cudaStream_t st) {
    auto k = cross_merge_runs_kernel<T, SCANS, V>;
    if (const int rc = allow_dynamic_smem(k, smem)) return rc;
    launch(k, (unsigned)(B * a.blocks), threads, smem, st, a);
    count_launch();
    return check_launch();
}
template <typename T, int SCANS> static int scan_runs_v(const RunArgs& a, bool pairs, int64_t B, int threads, size_t smem, cudaStream_t st) {
    if constexpr (sizeof(T) == 2) {
        if (pairs) return a.pad ? launch_scan_runs<T, SCANS, 2, true>(a, B, threads, smem, st) : launch_scan_runs<T, SCANS, 2, false>(a, B, threads, smem, st);
    }
    return a.pad ? launch_scan_runs<T, SCANS, 1, true>(a, B, threads, smem, st) : launch_scan_runs<T, SCANS, 1, false>(a, B, threads, smem, st);
}
template <typename T> static int scan_runs_s(const RunArgs& a, int scans, bool pairs, int64_t B, int threads, size_t smem, cudaStream_t st) {
    return scans == 0   ? scan_runs_v<T, 0>(a, pairs, B, threads, smem, st)
           : scans == 1 ? scan_runs_v<T, 1>(a, pairs, B, threads, smem, st)
           : scans == 2 ? scan_runs_v<T, 2>(a, pairs, B, threads, smem, st)
                        : scan_runs_v<T, 3>(a, pairs, B, threads, smem, st);
}
template <typename T, int SCANS> static int merge_runs_v(const RunArgs& a, bool pairs, int64_t B, int threads, size_t smem, cudaStream_t st) {
    if constexpr (sizeof(T) == 2) {
        if (pairs) return launch_merge_runs<T, SCANS, 2>(a, B, threads, smem, st);
    }
    return launch_merge_runs<T, SCANS, 1>(a, B, threads, smem, st);
}
template <typename T> static int merge_runs_s(const RunArgs& a, int scans, bool pairs, int64_t B, int threads, size_t smem, cudaStream_t st) {
    return scans == 0   ? merge_runs_v<T, 0>(a, pairs, B, threads, smem, st)
           : scans == 1 ? merge_runs_v<T, 1>(a, pairs, B, threads, smem, st)
           : scans == 2 ? merge_runs_v<T, 2>(a, pairs, B, threads, smem, st)
                        : merge_runs_v<T, 3>(a, pairs, B, threads, smem, st);
}
// A pair of 16-bit pixels stays on one line of either orientation, in one word of the map and of every route.
static bool run_pairs(const ss2d_cross_params* p) {
    return p->H % 2 == 0 && p->W % 2 == 0 && p->route_stride % 2 == 0 && aligned_to(p->in, 4) && aligned_to(p->out, 4);
}
static bool scan_runs(const ss2d_cross_params* p, long long most, cudaStream_t st, int& rc) {
    RunArgs a; int threads; size_t smem;
    if (!plan_runs(p, p->B, 1, most, a, threads, smem)) return false;
    rc = p->dtype == SS2D_F32 ? scan_runs_s<float>(a, p->scans, false, p->B, threads, smem, st) : scan_runs_s<uint16_t>(a, p->scans, run_pairs(p), p->B, threads, smem, st);
    return true;
}
static bool merge_runs(const ss2d_cross_params* p, cudaStream_t st, int& rc) {
    RunArgs a; int threads; size_t smem;
    if (!plan_runs(p, p->B, 4, kRunBytes, a, threads, smem)) return false;
    rc = p->dtype == SS2D_F32    ? merge_runs_s<float>(a, p->scans, false, p->B, threads, smem, st)
         : p->dtype == SS2D_BF16 ? merge_runs_s<__nv_bfloat16>(a, p->scans, run_pairs(p), p->B, threads, smem, st)
                                 : merge_runs_s<__half>(a, p->scans, run_pairs(p), p->B, threads, smem, st);
    return true;
}

// What cross_rows and calls with padded rows take: rows of at most 65 536 elements, planes of at most 200 KB (`slots` of them).
static bool padding_fits(const ss2d_cross_params* p, size_t esize, int slots) {
    const long long plane = slots == 1 ? p->H * (p->W | 1) : p->W * (p->H | 1), S = p->route_stride ? p->route_stride : p->H * p->W;
    return plane * (long long)esize * slots <= 200 * 1024 && S <= 65536;
}

static int launch_rows(const ss2d_cross_params* p, bool back, cudaStream_t st) {
    RunArgs a; int threads; size_t smem;
    if (!padding_fits(p, dtype_size(p->dtype), 1) || !plan_runs(p, p->B * 4, 1, kRunMost, a, threads, smem)) return SS2D_ENOTSUP;
    if (!aligned_to(p->in, 8) || !aligned_to(p->out, 8) || (a.S != a.L && a.S % 8 != 0)) return SS2D_EINVAL_ALIGN;
    const unsigned grid = (unsigned)(p->B * 4 * a.blocks);
    const int rc = p->dtype == SS2D_F32 ? allow_dynamic_smem(cross_rows_kernel<float>, smem) : allow_dynamic_smem(cross_rows_kernel<uint16_t>, smem);
    if (rc) return rc;
    if (p->dtype == SS2D_F32) launch(cross_rows_kernel<float>, grid, threads, smem, st, a, p->scans, back);
    else launch(cross_rows_kernel<uint16_t>, grid, threads, smem, st, a, p->scans, back);
    count_launch();
    return check_launch();
}

static int fill_args(const ss2d_cross_params* p, CrossArgs& a) {
    if (!p) return SS2D_EINVAL_NULL;
    if (!p->in || !p->out) return SS2D_EINVAL_NULL;
    if (!dtype_ok(p->dtype)) return SS2D_EINVAL_DTYPE;
    if (p->scans < 0 || p->scans > 3) return SS2D_ENOTSUP;
    if (p->B <= 0 || p->C <= 0 || p->H <= 0 || p->W <= 0) return SS2D_EINVAL_SHAPE;
    if (p->H * p->W > 0x3fffffffLL || p->C > 0x7fffffffLL || p->B * p->C > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;   // 32-bit indices inside a plane
    const size_t s = dtype_size(p->dtype);
    if (!aligned_to(p->in, s) || !aligned_to(p->out, s)) return SS2D_EINVAL_ALIGN;
    if (p->route_stride && p->route_stride < p->H * p->W) return SS2D_EINVAL_STRIDE;
    a.in = p->in; a.out = p->out;
    a.C = p->C; a.H = p->H; a.W = p->W;
    if ((p->H + 31) / 32 * ((p->W + 31) / 32) * p->B * p->C > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;      // tiles are numbered by 32 bits
    for (int k = 0; k < 4; ++k) a.route[k] = route_map(p->scans, k, p->H, p->W);
    return SS2D_OK;
}

// Routes with padded rows: the run kernels, and the tile kernel of a merge, take them.
static bool padded(const ss2d_cross_params* p) { return p->route_stride && p->route_stride != p->H * p->W; }

static int scan_tiles(const ss2d_cross_params* p, cudaStream_t st) {
    TileArgs a; size_t smem;
    if (!plan_tiles(p, 0, a, smem)) return SS2D_EINVAL_SHAPE;
    return p->dtype == SS2D_F32 ? launch_scan_tiles<float>(a, p->B, smem, st) : launch_scan_tiles<uint16_t>(a, p->B, smem, st);   // 16-bit types: bits are moved as-is
}

int cross_scan(const ss2d_cross_params* p, cudaStream_t st) {
    CrossArgs a;
    const int rc = fill_args(p, a);
    if (rc != SS2D_OK) return rc;
    if (padded(p)) {
        if (p->route_stride % 8 != 0 || !aligned_to(p->out, 8)) return SS2D_EINVAL_ALIGN;
        int done;
        return padding_fits(p, dtype_size(p->dtype), 1) && scan_runs(p, kRunMost, st, done) ? done : SS2D_ENOTSUP;
    }
    // 16-bit maps with even sides: the pair kernel where a plane of 64 x 64 and more does not fit, or has lines that start in one bank
    // (pieces set apart: 64 x 64 7.1 against 6.3 us, 128 x 128 20.4 against 18.8; dense lines: 56 x 56 21.2 against 23.7, 150 x 200 17.1
    // against 22.5).  Single elements: whole planes up to 72 KB, or 48 KB with such lines (fp32, 113 x 97 45 us, in tiles 68; 90 x 155, 56 KB,
    // 8.5 and 10.5; 107 x 160, 68 KB, 19.6 and 15.7).
    const bool pairs = p->dtype != SS2D_F32 && p->H % 2 == 0 && p->W % 2 == 0 && aligned_to(p->in, 4) && aligned_to(p->out, 4);
    const bool wide = pairs && p->H >= 48 && p->W >= 48;
    int done;
    if (!(wide && p->W % 32 == 0) && scan_runs(p, pairs || p->W * dtype_size(p->dtype) % 64 != 0 ? kRunBytes : kRunBytes / 3 * 2, st, done)) return done;
    if (wide) {
        CrossArgs q = a;
        q.tiles_h = (p->H + kPairTile - 1) / kPairTile;
        q.tiles_w = (p->W + kPairTile - 1) / kPairTile;
        launch(cross_scan_pair_kernel, (unsigned)(q.tiles_h * q.tiles_w * p->B * p->C), dim3(32, 8), 0, st, q);
        count_launch();
        return check_launch();
    }
    return scan_tiles(p, st);
}

int cross_rows(const ss2d_cross_params* p, int back, cudaStream_t st) {
    CrossArgs a;
    const int rc = fill_args(p, a);
    return rc != SS2D_OK ? rc : launch_rows(p, back != 0, st);
}

int cross_padding_supported(const ss2d_cross_params* p) {
    return p && dtype_ok(p->dtype) && p->H > 0 && p->W > 0 && p->C > 0 && padding_fits(p, 4, 2) ? 1 : 0;
}

static int merge_tiles(const ss2d_cross_params* p, cudaStream_t st) {
    TileArgs a; size_t smem;
    if (!plan_tiles(p, p->scans == 3 ? 2 : 1, a, smem)) return SS2D_EINVAL_SHAPE;
    return p->dtype == SS2D_F32    ? launch_merge_tiles<float>(a, p->B, p->scans, false, smem, st)
           : p->dtype == SS2D_BF16 ? launch_merge_tiles<__nv_bfloat16>(a, p->B, p->scans, run_pairs(p), smem, st)
                                   : launch_merge_tiles<__half>(a, p->B, p->scans, run_pairs(p), smem, st);
}

int cross_merge(const ss2d_cross_params* p, cudaStream_t st) {
    CrossArgs a;
    const int rc = fill_args(p, a);
    if (rc != SS2D_OK) return rc;
    if (padded(p)) {
        if (p->route_stride % 8 != 0 || !aligned_to(p->in, 8)) return SS2D_EINVAL_ALIGN;
        if (!padding_fits(p, dtype_size(p->dtype), 2)) return SS2D_ENOTSUP;
    }
    // Whole planes up to 72 KB of routes, three CTAs an SM, against tiles: fp32, 57 x 58 18.9 and 21.9 us, 28 x 28 34 and 44.
    int done;
    return merge_runs(p, st, done) ? done : merge_tiles(p, st);
}

// ------------------------------------------------------------------------------------------------
// Layout and one-by-one variants (channel-last x and / or routes; every route reading its own map):
// index-only variants of the two operators, off the benchmarked path.  One thread per (image, pixel,
// channel) handles the four routes; the fastest thread index follows the contiguous axis of the
// routes tensor (pixels for channel-first routes, channels for channel-last ones).
struct CrossExArgs {
    const void* in;
    void* out;
    RouteMap route[4];
    long long B, C, H, W, L, total;
    int x_cf, r_cf, one_by_one, scans;       // x / routes channel-first; every route has its own map
    int flat_1b1_copy;                       // one_by_one, scans 1: the four maps pass through unchanged
};

__device__ __forceinline__ long long x_index(const CrossExArgs& a, long long b, int k, long long c, long long p) {
    const long long K = a.one_by_one ? 4 : 1, kk = a.one_by_one ? k : 0;
    return a.x_cf ? ((b * K + kk) * a.C + c) * a.L + p : ((b * a.L + p) * K + kk) * a.C + c;
}
__device__ __forceinline__ long long r_index(const CrossExArgs& a, long long b, int k, long long c, long long l) {
    return a.r_cf ? ((b * 4 + k) * a.C + c) * a.L + l : ((b * a.L + l) * 4 + k) * a.C + c;
}
__device__ __forceinline__ void ex_decompose(const CrossExArgs& a, long long i, long long& b, long long& c, long long& p) {
    if (a.r_cf) { p = i % a.L; const long long t = i / a.L; c = t % a.C; b = t / a.C; }
    else { c = i % a.C; const long long t = i / a.C; p = t % a.L; b = t / a.L; }
}

template <typename T>
__global__ void __launch_bounds__(256) cross_scan_ex_kernel(const CrossExArgs a) {
    follow_previous();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.total; i += (long long)gridDim.x * blockDim.x) {
        long long b, c, p;
        ex_decompose(a, i, b, c, p);
        const long long h = p / a.W, w = p - h * a.W;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const RouteMap& m = a.route[k];
            const long long l = a.flat_1b1_copy ? p : m.base + m.sh * h + m.sw * w;
            ((T*)a.out)[r_index(a, b, k, c, l)] = ((const T*)a.in)[x_index(a, b, k, c, p)];
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) cross_merge_ex_kernel(const CrossExArgs a) {
    follow_previous();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.total; i += (long long)gridDim.x * blockDim.x) {
        long long b, c, p;
        ex_decompose(a, i, b, c, p);
        const long long h = p / a.W, w = p - h * a.W;
        T v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const RouteMap& m = a.route[k];
            const long long l = a.flat_1b1_copy ? p : m.base + m.sh * h + m.sw * w;
            v[k] = ((const T*)a.in)[r_index(a, b, k, c, l)];
        }
        if (a.one_by_one) {
#pragma unroll
            for (int k = 0; k < 4; ++k) ((T*)a.out)[x_index(a, b, k, c, p)] = v[k];
        } else {
            ((T*)a.out)[x_index(a, b, 0, c, p)] = flat_sum<T>(a.scans, v[0], v[1], v[2], v[3]);
        }
    }
}

static int fill_ex(const ss2d_cross_ex_params* p, CrossExArgs& a) {
    if (!p) return SS2D_EINVAL_NULL;
    if (!p->in || !p->out) return SS2D_EINVAL_NULL;
    if (!dtype_ok(p->dtype)) return SS2D_EINVAL_DTYPE;
    if (p->scans < 0 || p->scans > 3) return SS2D_ENOTSUP;
    if (p->B <= 0 || p->C <= 0 || p->H <= 0 || p->W <= 0) return SS2D_EINVAL_SHAPE;
    if (p->scans == 3 && p->H != p->W) return SS2D_EINVAL_SHAPE;
    if (p->H * p->W > 0x3fffffffLL) return SS2D_EINVAL_SHAPE;
    // one map per route with a channel-last side: the route sets the reference's GPU kernel defines (csm_triton.py:313-336:
    // 0, 1 and 2; its torch branch for 2 indexes the wrong axes, csm_triton.py:117-123, and neither path has 3)
    if (p->one_by_one && !(p->in_channel_first && p->out_channel_first) && p->scans > 2) return SS2D_ENOTSUP;
    const size_t s = dtype_size(p->dtype);
    if (!aligned_to(p->in, s) || !aligned_to(p->out, s)) return SS2D_EINVAL_ALIGN;
    a.in = p->in; a.out = p->out;
    a.B = p->B; a.C = p->C; a.H = p->H; a.W = p->W; a.L = p->H * p->W; a.total = p->B * p->C * a.L;
    a.x_cf = p->in_channel_first ? 1 : 0; a.r_cf = p->out_channel_first ? 1 : 0;
    a.one_by_one = p->one_by_one ? 1 : 0; a.scans = p->scans;
    a.flat_1b1_copy = (p->one_by_one && p->scans == 1) ? 1 : 0;
    for (int k = 0; k < 4; ++k) a.route[k] = route_map(p->scans, k, p->H, p->W);
    return SS2D_OK;
}

template <typename T, bool kScan>
static int launch_ex(const CrossExArgs& a, cudaStream_t st) {
    long long ctas = (a.total + 255) / 256;
    if (ctas > 148LL * 32) ctas = 148LL * 32;
    if constexpr (kScan) launch(cross_scan_ex_kernel<T>, (unsigned)ctas, 256, 0, st, a);
    else launch(cross_merge_ex_kernel<T>, (unsigned)ctas, 256, 0, st, a);
    count_launch();
    return check_launch();
}

int cross_scan_ex(const ss2d_cross_ex_params* p, cudaStream_t st) {
    CrossExArgs a;
    const int rc = fill_ex(p, a);
    if (rc != SS2D_OK) return rc;
    if (p->dtype == SS2D_F32) return launch_ex<float, true>(a, st);
    return launch_ex<unsigned short, true>(a, st);           // 16-bit types: a copy does not look inside
}

int cross_merge_ex(const ss2d_cross_ex_params* p, cudaStream_t st) {
    CrossExArgs a;
    const int rc = fill_ex(p, a);
    if (rc != SS2D_OK) return rc;
    if (p->dtype == SS2D_F32) return launch_ex<float, false>(a, st);
    if (p->dtype == SS2D_BF16) return launch_ex<__nv_bfloat16, false>(a, st);
    return launch_ex<__half, false>(a, st);
}

}  // namespace ss2d
