// out (M, N) = W (M, K) . x (K, N) (+ bias) for few pixels: the form of linear_cf.cu's projection for problems that leave most SMs
// without a 128-pixel tile (one image of a classifier: 196 pixels are two tiles, and each of their CTAs would first load all of W).
//
// A CTA of four warps computes a tile of 32 rows x 64 pixels.  Everything it needs (32 rows of W, 64 pixels of all K rows of x) is
// requested at once with cp.async, so that the whole load is one memory latency; the warps then split K between them
// (mma.sync m16n8k16, x through ldmatrix.trans) and meet in shared memory.  x is read once per 32 rows of W, from L2.
// With GELU it is the first half of an MLP block (the result stays fp32 until then), one launch instead of a library GEMM and a pass
// over its result.
// Bound: latency (two round trips to L2 and a launch).
#pragma once
#include "activations.cuh"
#include "common.cuh"

namespace ss2d {

constexpr int kLsM = 32, kLsN = 64, kLsWarps = 4, kLsXPitch = kLsN + 8;      // pitches keep ldmatrix conflict-free

struct LinearSmallArgs {
    const void *x, *w;
    const float* bias;
    void* out;
    int M, K, N, act;
    long long x_rs, out_rs;
};

inline size_t linear_small_smem(int64_t K) {
    const size_t stage = (size_t)K * kLsXPitch * 2 + (size_t)kLsM * (K + 8) * 2, red = (size_t)kLsWarps * kLsM * (kLsN + 4) * 4;
    return stage > red ? stage : red;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool ok) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(kLsWarps * 32) linear_small_kernel(const LinearSmallArgs a) {
    follow_previous();
    extern __shared__ __align__(16) unsigned char ls_raw[];
    const int K = a.K, M = a.M, WP = K + 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T* xs = reinterpret_cast<T*>(ls_raw);                  // [K][72]
    T* ws = xs + (size_t)K * kLsXPitch;                    // [32][K + 8]
    const int n0 = blockIdx.x * kLsN, m0 = blockIdx.y * kLsM;
    for (int i = threadIdx.x; i < K * (kLsN / 8); i += kLsWarps * 32) {
        const int k = i >> 3, c = (i & 7) * 8;
        const bool ok = n0 + c < a.N;                      // N is a multiple of 8
        cp_async16(xs + k * kLsXPitch + c, (const T*)a.x + k * a.x_rs + (ok ? n0 + c : 0), ok);
    }
    const int kv = K / 8;
    for (int i = threadIdx.x; i < kLsM * kv; i += kLsWarps * 32) {
        const int m = i / kv, c = (i - m * kv) * 8;
        const bool ok = m0 + m < M;
        cp_async16(ws + m * WP + c, (const T*)a.w + (long long)(ok ? m0 + m : 0) * K + c, ok);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float acc[2][8][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    for (int k0 = warp * 16; k0 < K; k0 += kLsWarps * 16) {
        uint32_t af[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {                      // rows 16 i .. 16 i + 15, k0 .. k0 + 15
            const unsigned p = (unsigned)__cvta_generic_to_shared(ws + (i * 16 + (lane & 15)) * WP + k0 + (lane >> 4) * 8);
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(af[i][0]), "=r"(af[i][1]), "=r"(af[i][2]), "=r"(af[i][3]) : "r"(p));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {                      // 16 pixels: two n8 operands
            uint32_t b[4];
            const unsigned p = (unsigned)__cvta_generic_to_shared(xs + (k0 + (lane & 15)) * kLsXPitch + j * 16 + (lane >> 4) * 8);
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                         : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(p));
            const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                MmaK16<T>::run(acc[i][2 * j], af[i], b0);
                MmaK16<T>::run(acc[i][2 * j + 1], af[i], b1);
            }
        }
    }
    __syncthreads();                                       // the operands are read: their room becomes the partial sums
    constexpr int RP = kLsN + 4;
    float* red = reinterpret_cast<float*>(ls_raw);         // [warp][32][68]
    {
        const int g = lane >> 2, t2 = (lane & 3) * 2;
        float* mine = red + warp * kLsM * RP;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                *reinterpret_cast<float2*>(mine + (i * 16 + g) * RP + j * 8 + t2) = make_float2(acc[i][j][0], acc[i][j][1]);
                *reinterpret_cast<float2*>(mine + (i * 16 + g + 8) * RP + j * 8 + t2) = make_float2(acc[i][j][2], acc[i][j][3]);
            }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kLsM * (kLsN / 8); i += kLsWarps * 32) {
        const int m = i >> 3, c = (i & 7) * 8;
        if (m0 + m >= M || n0 + c >= a.N) continue;
        float v[8];
        const float b = a.bias ? a.bias[m0 + m] : 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = b;
#pragma unroll
        for (int w = 0; w < kLsWarps; ++w) {
            const float4* q = reinterpret_cast<const float4*>(red + (w * kLsM + m) * RP + c);
            const float4 x = q[0], y = q[1];
            v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w; v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
        }
        if (a.act) {
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const float2 r = gelu_pair_poly(make_float2(v[e], v[e + 1]));
                v[e] = r.x; v[e + 1] = r.y;
            }
        }
        Vec<T, 8>::store((T*)a.out + (m0 + m) * a.out_rs + n0 + c, v);
    }
}

// Problems whose 128-pixel tiles are too few for the chip, whose operands fit a CTA's shared memory and whose result rows allow
// 16-byte stores.
inline bool linear_small_takes(const ss2d_linear_params* p) {
    const int64_t os = p->out_row_stride ? p->out_row_stride : p->N;
    const int64_t ctas = ((p->N + kLsN - 1) / kLsN) * ((p->M + kLsM - 1) / kLsM);
    return (p->N + 127) / 128 <= 74 && ctas <= 148 * 4 && linear_small_smem(p->K) <= 220 * 1024 && os % 8 == 0 && aligned_to(p->out, 16);
}

template <typename T> static int launch_linear_small(const ss2d_linear_params* p, cudaStream_t st) {
    LinearSmallArgs a = {p->x, p->w, (const float*)p->bias, p->out, (int)p->M, (int)p->K, (int)p->N, p->act, p->x_row_stride ? p->x_row_stride : p->N,
                         p->out_row_stride ? p->out_row_stride : p->N};
    const size_t smem = linear_small_smem(p->K);
    auto kern = linear_small_kernel<T>;
    if (const int rc = allow_dynamic_smem(kern, smem)) return rc;
    launch(kern, dim3((unsigned)((p->N + kLsN - 1) / kLsN), (unsigned)((p->M + kLsM - 1) / kLsM)), kLsWarps * 32, smem, st, a);
    count_launch();
    return check_launch();
}

}  // namespace ss2d
