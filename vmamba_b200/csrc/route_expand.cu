// Per-route expansion of the low-rank projections into the streams the fused scan consumes.
//
// Input: x_dbl = x_proj(x) computed ONCE on the map in its native (row-major) pixel order,
// (B, 4, R+2N, L).  For every route k this kernel writes, in the ORIENTATION order of the route
// (row-major pixels for k = 0, 2; column-major for k = 1, 3):
//   delta_k[b, d, q] = sum_r Wdt[k, d, r] * x_dbl[b, k, r, pix(q)]     (R -> D, rounded to the activation type)
//   bc_k[b, n, q]    = x_dbl[b, k, R + n, pix(q)]   n < 2N            (B then C rows, activation type)
// i.e. dt_projs (a grouped 1x1 convolution with a contraction length of only R = 6..64), the
// split/contiguous copies, and the CrossScan permutation of the projected rows, in one pass whose
// cost is the write of delta.  Two kernels: the FMA form below (fp32 maps, unaligned runs) and the
// mma.sync form further down (16-bit maps, every rank), which has no FMA loop and no weight
// broadcasts through shared memory and is 10 to 30 % faster.
//
// Mapping of the FMA form: an "item" is VEC consecutive pixels q of one (image, route) plane.  A CTA stages the
// R+2N projected rows of NI items in shared memory as fp32 (the column-major gather happens
// here), then thread (item, channel group) accumulates 4 channels x VEC pixels at a time with
// the weights broadcast from shared memory; lanes of a warp hold consecutive items, so every
// delta store is a full 512-byte line per channel.
#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace ss2d {

struct ExpandArgs {
    const void* xd;      // (B, 4, C, L)
    const void* wdt;     // (4, D, R) activation dtype
    void* delta[4];      // (B, D, L) each
    void* bc[4];         // (B, 2N, L) each, activation dtype
    long long xd_bs, xd_ks, xd_rs;     // element strides of x_dbl: batch, route, row
    long long d_bs[4], d_cs[4], bc_bs[4], bc_rs[4];   // delta: batch / channel strides; B-C rows: batch / row strides
    int B, D, R, N2, C, H, W, L;       // N2 = 2N, C = R + 2N; L = run length (H*W, or B*H*W when images are adjacent)
    int Limg, Lmap;                    // H * W; images of a run times that
    const void* xt;                    // transposed rows of routes 1, 3: (2, C, Btot, Limg), or NULL (gather)
    long long xt_rs;                   // Btot * Limg
    int items_per_plane, items_total;  // L / VEC, B * L / VEC
    int mma_tiles;                     // pixel tiles per CTA of the tensor-core kernel
};

constexpr int kExpThreads = 256;
constexpr int kDChunk = 128;   // channels per CTA (grid.z walks the slices)

template <typename T, int VEC, int NI>
__global__ void __launch_bounds__(kExpThreads) route_expand_kernel(const ExpandArgs a) {
    follow_previous();
    constexpr int NDG = kExpThreads / NI;   // channel groups working side by side
    constexpr int NP = (VEC + 1) / 2;
    extern __shared__ __align__(16) float sm[];
    float* s_rows = sm;                                  // [C][NI * VEC]
    float* s_w = sm + (size_t)a.C * NI * VEC;            // [R][kDChunk] (transposed: 4 channels = one float4)
    const int k = blockIdx.y;
    const bool col = (k & 1) != 0 && a.H > 1 && a.W > 1;      // a single row or column: both orders are one
    const int tid = threadIdx.x;
    const int item0 = blockIdx.x * NI;
    const T* __restrict__ xd = (const T*)a.xd + (long long)k * a.xd_ks;

    // ---- stage the projected rows of this CTA's items (gathering column-major pixels for odd k) ----
    const int it = tid % NI, dg = tid / NI;
    const int item = item0 + it;
    const bool live = item < a.items_total;
    const int b = live ? item / a.items_per_plane : 0;
    const int q0 = live ? (item - b * a.items_per_plane) * VEC : 0;
    {
        const int img0 = (q0 / a.Limg) * a.Limg, qi = q0 - img0;     // image of the first pixel, position inside it
        const int w0 = qi / a.H, h0 = qi - w0 * a.H;
        const T* src = xd + (long long)b * a.xd_bs;
        for (int row = dg; row < a.C; row += NDG) {
            float v[VEC];
#pragma unroll
            for (int i = 0; i < VEC; ++i) v[i] = 0.f;
            if (live) {
                const T* rp = src + (long long)row * a.xd_rs;
                if (!col) {
                    Vec<T, VEC>::load(rp + q0, v);
                } else if (a.xt) {
                    Vec<T, VEC>::load((const T*)a.xt + ((long long)(k >> 1) * a.C + row) * a.xt_rs + (long long)b * a.Limg + q0, v);
                } else {
                    int w = w0, h = h0, base = img0;      // a run may continue into the next image
#pragma unroll
                    for (int i = 0; i < VEC; ++i) {
                        v[i] = to_f<T>(rp[base + h * a.W + w]);
                        if (++h == a.H) { h = 0; if (++w == a.W) { w = 0; base += a.Limg; } }
                    }
                }
            }
            Vec<float, VEC>::store(s_rows + (size_t)row * (NI * VEC) + it * VEC, v);
        }
    }
    // this CTA's slice of the channels (grid.z splits D so that small maps still fill the GPU)
    const int dc = blockIdx.z * kDChunk;
    const int dn = min(kDChunk, a.D - dc);
    const T* __restrict__ wk = (const T*)a.wdt + (long long)k * a.D * a.R;
    for (int idx = tid; idx < kDChunk * a.R; idx += kExpThreads) {
        const int r = idx / kDChunk, dl = idx - r * kDChunk;
        s_w[idx] = (dl < dn) ? to_f<T>(wk[(long long)(dc + dl) * a.R + r]) : 0.f;
    }
    __syncthreads();

    // ---- B / C rows: pass through (first channel slice only) --------------------------------
    if (live && blockIdx.z == 0) {
        for (int n = dg; n < a.N2; n += NDG) {
            float v[VEC];
            Vec<float, VEC>::load(s_rows + (size_t)(a.R + n) * (NI * VEC) + it * VEC, v);
            Vec<T, VEC>::store((T*)a.bc[k] + b * a.bc_bs[k] + (long long)n * a.bc_rs[k] + q0, v);
        }
    }

    // ---- delta: R -> D expansion for the channels of this slice -------------------------------------
    T* __restrict__ dout = (T*)a.delta[k] + b * a.d_bs[k] + q0;
    for (int dl0 = dg * 4; dl0 < dn; dl0 += NDG * 4) {
        float2 acc[4][NP];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int j = 0; j < NP; ++j) acc[c][j] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int r = 0; r < a.R; ++r) {
            float sv[VEC];
            Vec<float, VEC>::load(s_rows + (size_t)r * (NI * VEC) + it * VEC, sv);
            const float4 w4 = *reinterpret_cast<const float4*>(s_w + r * kDChunk + dl0);
            const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
#pragma unroll
                for (int j = 0; j < NP; ++j) {
                    const float2 s2 = make_float2(sv[2 * j], (VEC > 1) ? sv[(2 * j + 1) % VEC] : 0.f);
                    acc[c][j] = __ffma2_rn(make_float2(wv[c], wv[c]), s2, acc[c][j]);
                }
            }
        }
        if (live) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (dl0 + c < dn) {
                    float o[VEC];
#pragma unroll
                    for (int i = 0; i < VEC; ++i) o[i] = (i & 1) ? acc[c][i >> 1].y : acc[c][i >> 1].x;
                    Vec<T, VEC>::store(dout + (long long)(dc + dl0 + c) * a.d_cs[k], o);
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Tensor-core variant for 16-bit maps: delta tile (channels x pixels) = W (channels x R) . X (R x pixels)
// with mma.sync m16n8k16 (fp32 accumulation, R zero-padded to a multiple of 16).  The contraction is
// far too short for the tensor pipe to matter as arithmetic; what it buys is that the shared-memory
// traffic and the issue slots of the FMA loop disappear, leaving the kernel with the write of delta.
//
// A warp owns 16 channels and walks the pixels in blocks of 32.  The pixels of a block are dealt to the columns of the four
// n8 operands so that a thread's accumulators are eight neighbouring pixels of two channels: column 2 t + e of operand n is pixel
// 8 t + 2 n + e.  The results leave from registers as 16-byte vectors, 64 bytes of a row at a time, and a vector of x enters
// shared memory as four words, 16 bytes apart; there is one barrier per tile of kMmaPix pixels.
// Bound: HBM writes, and the warps that keep them coming: four CTAs of 256 threads to an SM (2 x 512 planes of 64 x 64: 12.9, 10.6,
// 12.1 and 15.2 us with three to six).  Against two barriers a tile with the results through a shared tile: 64 x 192 planes
// of 28 x 28 28 -> 22 us (3.4 TB/s written), 2 x 512 of 64 x 64 16.2 -> 10.6 us, 16 x 1024 of 16 x 16 21.7 -> 15.3 us.
constexpr int kMmaPix = 64;
constexpr int kMmaTilesPerCta = 8;      // most pixel tiles per CTA: the staged weights then serve 512 pixels

template <typename T> __device__ __forceinline__ uint32_t pack2(float x, float y) {
    const T v[2] = {from_f<T>(x), from_f<T>(y)};
    uint32_t w;
    memcpy(&w, v, 4);
    return w;
}

template <typename T, int KP>
__global__ void __launch_bounds__(256, 4) route_expand_mma_kernel(const ExpandArgs a) {
    follow_previous();
    constexpr int PIX = kMmaPix;
    constexpr int KPAD = KP + 8, XPAD = PIX + 8;       // pitches (elements): conflict-free fragment loads and vector stores
    __shared__ __align__(16) T Ws[kDChunk * KPAD];     // [channel][k]
    __shared__ __align__(16) T Xs[2][KP * XPAD];       // [k][dealt pixel]
    const int k = blockIdx.y;
    const bool col = (k & 1) != 0 && a.H > 1 && a.W > 1;      // a single row or column: both orders are one
    const int tid = threadIdx.x, threads = blockDim.x, lane = tid & 31, warp = tid >> 5, slice = threads / 2;
    const int tiles_per_run = (a.L + PIX - 1) / PIX;
    const int groups_per_run = (tiles_per_run + a.mma_tiles - 1) / a.mma_tiles;
    const int b = blockIdx.x / groups_per_run;
    const int tile0 = (blockIdx.x - b * groups_per_run) * a.mma_tiles;
    const T* __restrict__ xd = (const T*)a.xd + (long long)k * a.xd_ks + (long long)b * a.xd_bs;
    const int dc = blockIdx.z * slice;
    const int dn = min(slice, a.D - dc);
    const T zero = from_f<T>(0.f);

    // one projected row of eight pixels, gathered column-major for the odd routes
    auto fetch8 = [&](int row, int q) {
        const T* rp = xd + (long long)row * a.xd_rs;
        if (!col) return *reinterpret_cast<const uint4*>(rp + q);
        if (a.xt)
            return *reinterpret_cast<const uint4*>((const T*)a.xt + ((long long)(k >> 1) * a.C + row) * a.xt_rs + (long long)b * a.Limg + q);
        __align__(16) T v[8];
        const int img0 = (q / a.Limg) * a.Limg, qi = q - img0;
        int w = qi / a.H, h = qi - w * a.H, base = img0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = base < a.Lmap ? rp[base + h * a.W + w] : zero;          // zero: the padding of a run
            if (++h == a.H) { h = 0; if (++w == a.W) { w = 0; base += a.Limg; } }
        }
        return *reinterpret_cast<const uint4*>(v);
    };
    // The X tile is read into registers one step ahead: the loads of tile t + 1 are in flight while tile t is contracted,
    // those of the first while the weights are staged.
    constexpr int VR = PIX / 8;                        // vectors of a row
    constexpr int NI = VR / 4;                         // of a thread: at least 4 KP threads
    uint4 pre[NI];
    auto load_tile = [&](int q0) {
#pragma unroll
        for (int n = 0; n < NI; ++n) {
            const int i = tid + n * threads, r = i / VR, q = q0 + (i % VR) * 8;
            if (r < a.R) pre[n] = q < a.L ? fetch8(r, q) : make_uint4(0u, 0u, 0u, 0u);      // L is a multiple of 8
        }
    };
    auto store_tile = [&](T* xs) {
#pragma unroll
        for (int n = 0; n < NI; ++n) {
            const int i = tid + n * threads, r = i / VR, c = i % VR;
            if (r < a.R) {
                uint32_t* x = reinterpret_cast<uint32_t*>(xs + r * XPAD + (c / 4) * 32) + c % 4;
                x[0] = pre[n].x; x[4] = pre[n].y; x[8] = pre[n].z; x[12] = pre[n].w;
            }
        }
    };
    if (tile0 * PIX < a.L) load_tile(tile0 * PIX);

    // ---- weights of this channel slice, [channel][k], zero beyond R and beyond the slice ----------------
    const T* __restrict__ wk = (const T*)a.wdt + (long long)k * a.D * a.R;
    if ((a.R & 7) == 0 && (reinterpret_cast<uintptr_t>(wk) & 15) == 0) {       // rows of whole 16-byte pieces
        for (int i = tid; i < slice * (KP / 8); i += threads) {
            const int dl = i / (KP / 8), r = (i - dl * (KP / 8)) * 8;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (dl < dn && r < a.R) v = *reinterpret_cast<const uint4*>(wk + (long long)(dc + dl) * a.R + r);
            *reinterpret_cast<uint4*>(&Ws[dl * KPAD + r]) = v;
        }
    } else {
        for (int i = tid; i < slice * KP; i += threads) {
            const int dl = i / KP, r = i - dl * KP;
            Ws[dl * KPAD + r] = (dl < dn && r < a.R) ? wk[(long long)(dc + dl) * a.R + r] : zero;
        }
    }
    for (int i = tid; i < 2 * (KP - a.R) * XPAD; i += threads) {              // rows R .. KP - 1 are zero
        const int s = i / ((KP - a.R) * XPAD);
        Xs[s][a.R * XPAD + i - s * (KP - a.R) * XPAD] = zero;
    }
    if (tile0 * PIX < a.L) store_tile(Xs[0]);
    __syncthreads();
    const int g = lane >> 2, t4 = lane & 3, m0 = warp * 16;
    uint32_t af[KP / 16][4];
#pragma unroll
    for (int k0 = 0; k0 < KP; k0 += 16) {
        const T* w = Ws + (m0 + g) * KPAD + k0 + 2 * t4;
        af[k0 / 16][0] = *reinterpret_cast<const uint32_t*>(w);
        af[k0 / 16][1] = *reinterpret_cast<const uint32_t*>(w + 8 * KPAD);
        af[k0 / 16][2] = *reinterpret_cast<const uint32_t*>(w + 8);
        af[k0 / 16][3] = *reinterpret_cast<const uint32_t*>(w + 8 * KPAD + 8);
    }
    T* __restrict__ out = (T*)a.delta[k] + b * a.d_bs[k] + (long long)(dc + m0 + g) * a.d_cs[k] + t4 * 8;
    const bool low = m0 + g < dn, high = m0 + g + 8 < dn;
    const long long eight = 8 * a.d_cs[k];
    for (int tt = 0; tt < a.mma_tiles; ++tt) {
        const int q0 = (tile0 + tt) * PIX;
        if (q0 >= a.L) break;                        // uniform over the CTA
        const bool has_next = tt + 1 < a.mma_tiles && q0 + PIX < a.L;
        if (has_next) load_tile(q0 + PIX);
        // ---- B / C rows pass through (first channel slice only) ---------------------------------------------
        if (blockIdx.z == 0) {
            for (int i = tid; i < a.N2 * VR; i += threads) {
                const int n = i / VR, q = q0 + (i - n * VR) * 8;
                if (q < a.L) *reinterpret_cast<uint4*>((T*)a.bc[k] + b * a.bc_bs[k] + (long long)n * a.bc_rs[k] + q) = fetch8(a.R + n, q);
            }
        }
        const T* xs = Xs[tt & 1];
#pragma unroll
        for (int p0 = 0; p0 < PIX; p0 += 32) {
            float acc[4][4] = {};
#pragma unroll
            for (int k0 = 0; k0 < KP; k0 += 16) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t f[4];
                    const unsigned p = (unsigned)__cvta_generic_to_shared(xs + (k0 + (lane & 15)) * XPAD + p0 + h * 16 + (lane >> 4) * 8);
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(p) : "memory");
                    const uint32_t f0[2] = {f[0], f[1]}, f1[2] = {f[2], f[3]};
                    MmaK16<T>::run(acc[2 * h], af[k0 / 16], f0);
                    MmaK16<T>::run(acc[2 * h + 1], af[k0 / 16], f1);
                }
            }
            T* o = out + q0 + p0;
            if (q0 + p0 + t4 * 8 < a.L) {
                if (low)
                    *reinterpret_cast<uint4*>(o) = make_uint4(pack2<T>(acc[0][0], acc[0][1]), pack2<T>(acc[1][0], acc[1][1]),
                                                              pack2<T>(acc[2][0], acc[2][1]), pack2<T>(acc[3][0], acc[3][1]));
                if (high)
                    *reinterpret_cast<uint4*>(o + eight) = make_uint4(pack2<T>(acc[0][2], acc[0][3]), pack2<T>(acc[1][2], acc[1][3]),
                                                                      pack2<T>(acc[2][2], acc[2][3]), pack2<T>(acc[3][2], acc[3][3]));
            }
        }
        if (has_next) store_tile(Xs[(tt + 1) & 1]);  // its last readers passed the barrier of the step before
        __syncthreads();
    }
}

static int expand_cuts(const ExpandArgs& a) { return (a.D + kDChunk - 1) / kDChunk; }
static bool expand_idle(const ExpandArgs& a, long long pixel_ctas) { return pixel_ctas * 4 * expand_cuts(a) < 148 * 2; }

template <typename T>
static int launch_expand_mma(ExpandArgs a, cudaStream_t st) {
    const int kp = (a.R + 15) / 16 * 16;
    const long long tiles_per_run = (a.L + kMmaPix - 1) / kMmaPix;
    // equal slices of at most 128 channels, a warp for every 16 and threads enough for two vectors of the X tile each
    const int cuts = expand_cuts(a);
    const int threads = std::max(4 * kp, ((a.D + cuts - 1) / cuts + 15) / 16 * 32);
    // Eight pixel tiles per CTA: measured over the ten launches of the 14 x 14 and 7 x 7 stages of a batch-128
    // forward, 4 and 8 tiles are equal (253 / 255 us), 16 and more leave too few CTAs, 1 or 2 re-stage the weights
    // too often.
    // Fewer where that leaves SMs idle; a run is cut into equal parts.
    int per = kMmaTilesPerCta;
    while (per > 1 && expand_idle(a, a.B * ((tiles_per_run + per - 1) / per))) per /= 2;
    const long long parts = (tiles_per_run + per - 1) / per;
    a.mma_tiles = (int)((tiles_per_run + parts - 1) / parts);
    const long long tiles = (long long)a.B * ((tiles_per_run + a.mma_tiles - 1) / a.mma_tiles);
    if (tiles > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
    const dim3 grid((unsigned)tiles, 4, (unsigned)cuts);
    if (kp == 16) launch(route_expand_mma_kernel<T, 16>, grid, threads, 0, st, a);
    else if (kp == 32) launch(route_expand_mma_kernel<T, 32>, grid, threads, 0, st, a);
    else if (kp == 48) launch(route_expand_mma_kernel<T, 48>, grid, threads, 0, st, a);
    else if (kp == 64) launch(route_expand_mma_kernel<T, 64>, grid, threads, 0, st, a);
    else return SS2D_ENOTSUP;
    count_launch();
    return check_launch();
}

template <typename T, int VEC, int NI>
static int launch_expand(const ExpandArgs& a, cudaStream_t st) {
    const size_t smem = ((size_t)a.C * NI * VEC + (size_t)a.R * kDChunk) * sizeof(float);
    if (smem > 200 * 1024) return SS2D_ENOTSUP;
    auto kern = route_expand_kernel<T, VEC, NI>;
    if (const int rc = allow_dynamic_smem(kern, smem)) return rc;
    const dim3 grid((unsigned)((a.items_total + NI - 1) / NI), 4, (unsigned)((a.D + kDChunk - 1) / kDChunk));
    launch(kern, grid, kExpThreads, smem, st, a);
    count_launch();
    return check_launch();
}

template <typename T, int VEC>
static int launch_expand_ni(const ExpandArgs& a, cudaStream_t st) {
    // fewer items per CTA when many rows have to be staged
    if ((size_t)a.C * 64 * VEC * 4 <= 56 * 1024) return launch_expand<T, VEC, 64>(a, st);
    return launch_expand<T, VEC, 32>(a, st);
}

template <typename T>
static int launch_expand_v(const ExpandArgs& a, int vec, cudaStream_t st) {
    switch (vec) {
        case 8: return launch_expand_ni<T, 8>(a, st);
        case 4: return launch_expand_ni<T, 4>(a, st);
        case 2: return launch_expand_ni<T, 2>(a, st);
        default: return launch_expand_ni<T, 1>(a, st);
    }
}

// Plane transposes of the projected rows of the two column-major routes: (route 1|3, row c, image b) plane
// H x W (row-major) -> W x H, written as (2, C, Btot, L).  A CTA takes a few planes through shared memory
// (pitch W + 1), reads and writes coalesced.
struct TransArgs {
    const void* xd;
    void* xt;
    long long xd_bs, xd_ks, xd_rs;
    long long xt_rs;
    int C, B, H, W, L, planes, vec_ok;  // planes = 2 * C * B; vec_ok: every plane start is 16-byte aligned
};

template <typename T>
__global__ void __launch_bounds__(256) plane_transpose_kernel(const TransArgs a) {
    follow_previous();
    extern __shared__ __align__(16) unsigned char traw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int P = a.W + 1, psz = a.H * P;
    T* tile = reinterpret_cast<T*>(traw) + (size_t)warp * psz;     // one plane per warp: no CTA barrier
    constexpr int PV = 16 / (int)sizeof(T);
    const bool vec = (a.L % PV) == 0 && a.vec_ok;
    for (int pid = blockIdx.x * nwarps + warp; pid < a.planes; pid += gridDim.x * nwarps) {
        const int b = pid % a.B, c = (pid / a.B) % a.C, kk = pid / (a.B * a.C);
        const T* src = (const T*)a.xd + (long long)(2 * kk + 1) * a.xd_ks + (long long)b * a.xd_bs + (long long)c * a.xd_rs;
        T* dst = (T*)a.xt + (long long)(pid / a.B) * a.xt_rs + (long long)b * a.L;
        if (vec) {
            for (int e = lane * PV; e < a.L; e += 32 * PV) {
                T v[PV];
                *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(src + e);
                int h = e / a.W, w = e - h * a.W;
#pragma unroll
                for (int i = 0; i < PV; ++i) {
                    tile[h * P + w] = v[i];
                    if (++w == a.W) { w = 0; ++h; }
                }
            }
            __syncwarp();
            for (int q = lane * PV; q < a.L; q += 32 * PV) {
                T v[PV];
                int w = q / a.H, h = q - w * a.H;
#pragma unroll
                for (int i = 0; i < PV; ++i) {
                    v[i] = tile[h * P + w];
                    if (++h == a.H) { h = 0; ++w; }
                }
                *reinterpret_cast<uint4*>(dst + q) = *reinterpret_cast<const uint4*>(v);
            }
        } else {
            for (int e = lane; e < a.L; e += 32) { const int h = e / a.W, w = e - h * a.W; tile[h * P + w] = src[e]; }
            __syncwarp();
            for (int q = lane; q < a.L; q += 32) { const int w = q / a.H, h = q - w * a.H; dst[q] = tile[h * P + w]; }
        }
        __syncwarp();
    }
}

static bool transpose_fits(const ss2d_expand_params* p) {
    return (size_t)p->H * (p->W + 1) * dtype_size(p->act_dtype) <= 16 * 1024;
}

// Elements of a row over all images (rows of a workspace, adjacent images).
static long long expand_run(const ss2d_expand_params* p) {
    const long long n = p->B * p->H * p->W;
    return p->padded_rows ? (n + 7) / 8 * 8 : n;
}

long long route_expand_workspace_bytes(const ss2d_expand_params* p) {
    if (!p || !dtype_ok(p->act_dtype) || p->B <= 0 || p->R <= 0 || p->N <= 0 || p->H <= 0 || p->W <= 0) return -1;
    if (p->image_row) return 4 * (p->R + 2 * p->N) * p->B * p->image_row * (long long)dtype_size(p->act_dtype);
    if (!transpose_fits(p) || p->H == 1 || p->W == 1) return 0;
    return 2 * (p->R + 2 * p->N) * expand_run(p) * (long long)dtype_size(p->act_dtype);
}

// All projected rows in the orientation order of their route (pixel order for routes 0, 2, column-major for 1, 3), a row of an
// image padded to `pad` elements with zeros: (4, C, B, pad).  Small next to what the expansion writes.  A warp per plane, or, where
// that leaves SMs idle, a CTA (104 planes of 62 x 64: 28 us with warps).
template <typename T, bool kCta>
__global__ void __launch_bounds__(256) orient_rows_kernel(const TransArgs a, const int pad) {
    follow_previous();
    extern __shared__ __align__(16) unsigned char traw[];
    const int step = kCta ? blockDim.x : 32, lane = kCta ? threadIdx.x : threadIdx.x & 31;
    const int warp = kCta ? 0 : threadIdx.x >> 5, nwarps = kCta ? 1 : blockDim.x >> 5;
    const auto sync = [] { if constexpr (kCta) __syncthreads(); else __syncwarp(); };
    const int P = a.W | 1;
    T* tile = reinterpret_cast<T*>(traw) + (size_t)warp * a.H * P;
    const T zero = from_f<T>(0.f);
    for (int pid = blockIdx.x * nwarps + warp; pid < a.planes; pid += gridDim.x * nwarps) {
        const int b = pid % a.B, kc = pid / a.B, k = kc / a.C, c = kc - k * a.C;
        const T* __restrict__ src = (const T*)a.xd + k * a.xd_ks + b * a.xd_bs + c * a.xd_rs;
        T* __restrict__ dst = (T*)a.xt + (long long)pid * pad;
        if (k & 1) {
#pragma unroll 4
            for (int e = lane; e < a.L; e += step) { const int h = e / a.W; tile[h * P + (e - h * a.W)] = src[e]; }
            sync();
#pragma unroll 4
            for (int q = lane; q < pad; q += step) { const int w = q / a.H; dst[q] = q < a.L ? tile[(q - w * a.H) * P + w] : zero; }
            sync();
        } else {
#pragma unroll 4
            for (int e = lane; e < pad; e += step) dst[e] = e < a.L ? src[e] : zero;
        }
    }
}

template <typename T>
static int launch_orient(const ss2d_expand_params* p, cudaStream_t st) {
    TransArgs t;
    t.xd = p->x_dbl; t.xt = p->workspace;
    t.xd_bs = p->x_dbl_batch_stride; t.xd_ks = p->x_dbl_route_stride; t.xd_rs = p->x_dbl_row_stride ? p->x_dbl_row_stride : p->H * p->W;
    t.C = (int)(p->R + 2 * p->N); t.B = (int)p->B; t.H = (int)p->H; t.W = (int)p->W; t.L = (int)(p->H * p->W); t.xt_rs = 0; t.vec_ok = 0;
    if (4LL * t.C * t.B > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
    t.planes = 4 * t.C * t.B;
    const size_t plane_bytes = (size_t)t.H * (t.W | 1) * sizeof(T);
    if (plane_bytes > 200 * 1024) return SS2D_ENOTSUP;
    const bool cta = t.planes < 148 * 8;
    int warps = cta ? 1 : (int)(48 * 1024 / plane_bytes);
    warps = warps < 1 ? 1 : warps > 8 ? 8 : warps;
    auto kern = cta ? orient_rows_kernel<T, true> : orient_rows_kernel<T, false>;
    const size_t smem = plane_bytes * warps;
    if (const int rc = allow_dynamic_smem(kern, smem)) return rc;
    long long ctas = (t.planes + warps - 1) / warps;
    if (ctas > 148 * 16) ctas = 148 * 16;
    launch(kern, (unsigned)ctas, cta ? 256 : warps * 32, smem, st, t, (int)p->image_row);
    count_launch();
    return check_launch();
}

template <typename T>
static int launch_transpose(const ss2d_expand_params* p, cudaStream_t st) {
    TransArgs t;
    t.xd = p->x_dbl; t.xt = p->workspace;
    t.xd_bs = p->x_dbl_batch_stride; t.xd_ks = p->x_dbl_route_stride; t.xd_rs = p->x_dbl_row_stride ? p->x_dbl_row_stride : p->H * p->W;
    t.C = (int)(p->R + 2 * p->N); t.B = (int)p->B; t.H = (int)p->H; t.W = (int)p->W; t.L = (int)(p->H * p->W);
    t.planes = 2 * t.C * t.B; t.xt_rs = expand_run(p);
    const size_t pv = 16 / sizeof(T);
    t.vec_ok = (t.xt_rs % pv) == 0 && (t.xd_bs % pv) == 0 && (t.xd_ks % pv) == 0 && (t.xd_rs % pv) == 0 && aligned_to(p->x_dbl, 16) && aligned_to(p->workspace, 16);
    const size_t plane_bytes = ((size_t)t.H * (t.W + 1) * sizeof(T) + 15) / 16 * 16;
    int warps = (int)(32 * 1024 / plane_bytes);
    if (warps < 1) warps = 1;
    if (warps > 8) warps = 8;
    const size_t smem = plane_bytes * warps;
    auto kern = plane_transpose_kernel<T>;
    if (const int rc = allow_dynamic_smem(kern, smem)) return rc;
    long long ctas = (t.planes + warps - 1) / warps;
    if (ctas > 148 * 16) ctas = 148 * 16;
    launch(kern, (unsigned)ctas, warps * 32, smem, st, t);
    count_launch();
    return check_launch();
}

int route_expand(const ss2d_expand_params* p, cudaStream_t st) {
    if (!p) return SS2D_EINVAL_NULL;
    if (!p->x_dbl || !p->dt_weight) return SS2D_EINVAL_NULL;
    for (int k = 0; k < 4; ++k)
        if (!p->delta[k] || !p->bc[k]) return SS2D_EINVAL_NULL;
    if (!dtype_ok(p->act_dtype)) return SS2D_EINVAL_DTYPE;
    if (p->B <= 0 || p->D <= 0 || p->R <= 0 || p->N <= 0 || p->H <= 0 || p->W <= 0) return SS2D_EINVAL_SHAPE;
    const long long L = p->H * p->W;
    if (L > 0x3fffffffLL || p->B * L > 0x7fffffffLL || p->R > 1024 || p->N > SS2D_MAX_DSTATE) return SS2D_EINVAL_SHAPE;
    const long long C = p->R + 2 * p->N;
    const long long xd_rs = p->x_dbl_row_stride ? p->x_dbl_row_stride : L;
    if (xd_rs < L || p->x_dbl_route_stride < L || (p->B > 1 && p->x_dbl_batch_stride < L)) return SS2D_EINVAL_STRIDE;
    const size_t s = dtype_size(p->act_dtype);
    if (!aligned_to(p->x_dbl, s) || !aligned_to(p->dt_weight, s)) return SS2D_EINVAL_ALIGN;
    for (int k = 0; k < 4; ++k) {
        if (!aligned_to(p->delta[k], s) || !aligned_to(p->bc[k], s)) return SS2D_EINVAL_ALIGN;
        if (p->B > 1 && (p->delta_batch_stride[k] < L || p->bc_batch_stride[k] < L)) return SS2D_EINVAL_STRIDE;
        if ((p->delta_channel_stride[k] && p->delta_channel_stride[k] < L) || (p->bc_row_stride[k] && p->bc_row_stride[k] < L)) return SS2D_EINVAL_STRIDE;
    }
    if (p->image_row) {
        const long long Lp = p->image_row;
        if (Lp % 8 != 0 || Lp < L || p->B * Lp > 0x7fffffffLL) return SS2D_EINVAL_SHAPE;
        for (int k = 0; k < 4; ++k)
            if (p->delta_batch_stride[k] != Lp || p->bc_batch_stride[k] != Lp || p->delta_channel_stride[k] < p->B * Lp || p->bc_row_stride[k] < p->B * Lp)
                return SS2D_EINVAL_STRIDE;
        if (!p->workspace || p->workspace_bytes < route_expand_workspace_bytes(p)) return SS2D_EWORKSPACE;
        if (!aligned_to(p->workspace, 16)) return SS2D_EINVAL_ALIGN;
        const int rc = p->act_dtype == SS2D_F32 ? launch_orient<float>(p, st) : p->act_dtype == SS2D_BF16 ? launch_orient<__nv_bfloat16>(p, st) : launch_orient<__half>(p, st);
        if (rc != SS2D_OK) return rc;
        ss2d_expand_params q = *p;        // the oriented rows as one long row per channel
        q.x_dbl = p->workspace; q.x_dbl_batch_stride = Lp; q.x_dbl_row_stride = p->B * Lp; q.x_dbl_route_stride = C * p->B * Lp;
        q.H = 1; q.W = Lp; q.image_row = 0; q.workspace = nullptr; q.workspace_bytes = 0; q.padded_rows = 0;
        return route_expand(&q, st);
    }
    // images adjacent in every tensor (channel-major maps): one run of B*L pixels per row, so that the
    // vector width does not depend on the size of a single map
    const bool transposed = p->workspace && transpose_fits(p) && p->H > 1 && p->W > 1;
    const bool pad = p->padded_rows && (transposed || p->H == 1 || p->W == 1);      // a gather could not tell the padding apart
    bool flat = (p->B > 1 || pad) && p->x_dbl_batch_stride == L;
    for (int k = 0; k < 4; ++k) flat = flat && p->delta_batch_stride[k] == L && p->bc_batch_stride[k] == L;
    const long long run = flat ? (pad ? expand_run(p) : p->B * L) : L;
    if (flat && pad) {
        if (xd_rs < run || p->x_dbl_route_stride < run) return SS2D_EINVAL_STRIDE;
        for (int k = 0; k < 4; ++k)
            if (p->delta_channel_stride[k] < run || p->bc_row_stride[k] < run) return SS2D_EINVAL_STRIDE;
    }
    // widest pixel vector that keeps every row start aligned in every tensor
    int vec = 8;
    auto fit = [&](long long x) { if (x < 0) x = -x; while (vec > 1 && (x % vec) != 0) vec >>= 1; };
    fit(run); fit(p->x_dbl_route_stride); fit(xd_rs);
    if (!flat) fit(p->x_dbl_batch_stride);
    fit((long long)(reinterpret_cast<uintptr_t>(p->x_dbl) / s));
    for (int k = 0; k < 4; ++k) {
        if (!flat) { fit(p->delta_batch_stride[k]); fit(p->bc_batch_stride[k]); }
        fit(p->delta_channel_stride[k] ? p->delta_channel_stride[k] : L); fit(p->bc_row_stride[k] ? p->bc_row_stride[k] : L);
        fit((long long)(reinterpret_cast<uintptr_t>(p->delta[k]) / s));
        fit((long long)(reinterpret_cast<uintptr_t>(p->bc[k]) / s));
    }
    // tensor cores for every rank: with the pixel-tile prefetch they are 10 % faster than the FMA kernel for R = 6, 12 too
    const bool mma_ok = vec == 8 && s == 2 && p->R <= 64 && (run % 8) == 0;
    // the staged rows (C rows x 64 items x vec floats) should stay near 28 KB so that several CTAs share an SM
    while (vec > 1 && C * 64 * vec * 4 > 28 * 1024) vec >>= 1;
    ExpandArgs a;
    a.xd = p->x_dbl; a.wdt = p->dt_weight;
    for (int k = 0; k < 4; ++k) {
        a.delta[k] = p->delta[k]; a.bc[k] = p->bc[k];
        a.d_bs[k] = p->delta_batch_stride[k]; a.bc_bs[k] = p->bc_batch_stride[k];
        a.d_cs[k] = p->delta_channel_stride[k] ? p->delta_channel_stride[k] : L;
        a.bc_rs[k] = p->bc_row_stride[k] ? p->bc_row_stride[k] : L;
    }
    a.xd_bs = p->x_dbl_batch_stride; a.xd_ks = p->x_dbl_route_stride; a.xd_rs = xd_rs;
    a.B = (int)p->B; a.D = (int)p->D; a.R = (int)p->R; a.N2 = (int)(2 * p->N); a.C = (int)C;
    a.H = (int)p->H; a.W = (int)p->W; a.L = (int)run; a.Limg = (int)L;
    a.Lmap = (int)(flat ? p->B * L : L);
    a.xt = nullptr; a.xt_rs = expand_run(p);
    // Where the pixel tiles leave SMs idle the column-major routes are gathered from the projected rows, a launch less (14 x 14
    // map of 384 channels: 5.2 us against 7.8 in two launches); on larger maps the strided 2-byte loads cost more.
    const bool gather = mma_ok && expand_idle(a, (flat ? 1 : p->B) * ((run + kMmaPix - 1) / kMmaPix));
    if (transposed && !gather) {
        if (p->workspace_bytes < route_expand_workspace_bytes(p)) return SS2D_EWORKSPACE;
        if (!aligned_to(p->workspace, 16)) return SS2D_EINVAL_ALIGN;
        int tr;
        if (p->act_dtype == SS2D_F32) tr = launch_transpose<float>(p, st);
        else if (p->act_dtype == SS2D_BF16) tr = launch_transpose<__nv_bfloat16>(p, st);
        else tr = launch_transpose<__half>(p, st);
        if (tr != SS2D_OK) return tr;
        a.xt = p->workspace;
    }
    if (flat) a.B = 1;
    a.items_per_plane = (int)(run / vec);
    a.items_total = (int)((flat ? 1 : p->B) * (run / vec));
    if (mma_ok) {
        if (p->act_dtype == SS2D_BF16) return launch_expand_mma<__nv_bfloat16>(a, st);
        return launch_expand_mma<__half>(a, st);
    }
    if (p->act_dtype == SS2D_F32) return launch_expand_v<float>(a, vec, st);
    if (p->act_dtype == SS2D_BF16) return launch_expand_v<__nv_bfloat16>(a, vec, st);
    return launch_expand_v<__half>(a, vec, st);
}

}  // namespace ss2d
