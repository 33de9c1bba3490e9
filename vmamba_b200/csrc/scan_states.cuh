// Shared parts of the selective-scan kernels for 2 .. 16 states (scan_states_fwd.cuh, scan_states_bwd.cuh).
//
// Mapping.  The NS = 4, 8 or 16 states of a row (a smaller state count is padded with states whose A, B and C are zero)
// are split over SL = NS / 4 neighbouring lanes, four states per lane, so that a warp holds 32 / SL rows and the chip is
// full from a quarter of the rows that a lane-per-row form needs.  The arithmetic on a lane's four states runs as two
// packed f32x2 operations.  A row is walked in chunks of 32 elements: u and delta are loaded as 16-byte vectors (as
// single elements, coalesced, where the rows are not aligned), the step size is formed once per element while the chunk
// is staged in shared memory, and the chunk is then read back as four elements per load.  The B / C values of a chunk are
// staged once per CTA (all rows of a CTA belong to one image and one group).
//
// Segments.  Where the rows of a problem do not fill the chip, every row is cut into S segments of a multiple of 64
// elements that are walked side by side.  A first kernel leaves what a segment does to a state that enters it (its
// end state from zero and the sum of its step sizes; the decay over the segment is exp(A * sum)), and the main kernel
// folds the segments in front of its own.  The extra pass costs at most as many exponentials as the main one.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "scan_row.cuh"

namespace ss2d {

constexpr int kStChunk = 32;            // elements per chunk
constexpr int kStPitch = 36;            // floats between the rows of a staged chunk: 16-byte reads of 8 rows hit 32 banks
constexpr int kStRows = 32;             // rows per CTA, whatever the state count

// R: rows per lane.  Two rows share every read of B and C, which takes the shared-memory pipe out of the way (a 16-byte read
// occupies its write-back for four cycles even when the lanes read the same values), but leave half the warps.
template <int NS, int R_ = 1> struct StLayout {
    static constexpr int SL = NS / 4;           // lanes per row
    static constexpr int R = R_;
    static constexpr int RL = 32 / SL;          // lane row i holds rows i, i + RL
    static constexpr int RPW = R * RL;          // rows per warp
    static constexpr int kWarps = kStRows / RPW;
    static constexpr int BCP = NS + 4;          // floats between the elements of staged B / C
};

__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }

__device__ __forceinline__ void st_put8(float* dst, const float (&v)[8]) {
    float4* q = reinterpret_cast<float4*>(dst);
    q[0] = make_float4(v[0], v[1], v[2], v[3]);
    q[1] = make_float4(v[4], v[5], v[6], v[7]);
}

// Walks the RPW x 32 elements of a warp's chunk in the order in which the lanes load and store them: f8(row, el) for eight
// consecutive elements (VW > 1), f1(row, el) for single ones.
template <int RPW, int VW, typename F8, typename F1>
__device__ __forceinline__ void st_for_each(int lane, F8 f8, F1 f1) {
    if constexpr (VW > 1) {
#pragma unroll
        for (int i = 0; i < RPW / 8; ++i) f8(i * 8 + (lane >> 2), (lane & 3) * 8);
    } else {
#pragma unroll 4
        for (int row = 0; row < RPW; ++row) f1(row, lane);
    }
}

// The way back: RPW rows x 32 elements of fp32 from shared memory to global rows.
template <typename T, int RPW, int VW>
__device__ __forceinline__ void st_unstage(const float* src, T* rows, int64_t stride, int count, int t0, int L, int lane) {
    st_for_each<RPW, VW>(
        lane,
        [&](int row, int el) {
            const float4* q = reinterpret_cast<const float4*>(src + row * kStPitch + el);
            const float4 x = q[0], y = q[1];
            const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
            for (int h = 0; h < 8; h += VW)
                if (row < count && t0 + el + h < L) {
                    float o[VW];
#pragma unroll
                    for (int e = 0; e < VW; ++e) o[e] = v[h + e];
                    Vec<T, VW>::store(rows + row * stride + t0 + el + h, o);
                }
        },
        [&](int row, int el) {
            if (row < count && t0 + el < L) rows[row * stride + t0 + el] = from_f<T>(src[row * kStPitch + el]);
        });
}

template <int N> __device__ __forceinline__ void st_put(float* dst, const float (&v)[N]) {
    if constexpr (N == 8) st_put8(dst, v);
    else dst[0] = v[0];
}

// The same chunks held in registers between the load and the store to shared memory.  A lane's part is RPW / 8 runs of
// eight elements (VW > 1) or one element of every row (VW = 1).
template <typename T, int RPW, int VW> struct StRaw {
    static constexpr int kRuns = VW > 1 ? RPW / 8 : RPW, kVecs = VW > 1 ? 8 / VW : 1;
    typename Vec<T, VW>::Raw w[kRuns][kVecs];
    template <typename F> static __device__ __forceinline__ void for_each(int lane, F f) {
#pragma unroll
        for (int i = 0; i < kRuns; ++i) {
            if constexpr (VW > 1) f(i, i * 8 + (lane >> 2), (lane & 3) * 8, std::integral_constant<int, 8>{});
            else f(i, i, lane, std::integral_constant<int, 1>{});
        }
    }
    __device__ __forceinline__ void load(const T* rows, int64_t stride, int count, int t0, int L, int lane) {
        for_each(lane, [&](int i, int row, int el, auto) {
#pragma unroll
            for (int h = 0; h < kVecs; ++h) {
                w[i][h] = {};
                if (row < count && t0 + el + h * VW < L) w[i][h] = Vec<T, VW>::load_raw(rows + row * stride + t0 + el + h * VW);
            }
        });
    }
    template <int E> __device__ __forceinline__ void get(int i, float (&v)[E], const T*, int64_t, int, int, int) const {
#pragma unroll
        for (int h = 0; h < kVecs; ++h) {
            float x[VW];
            Vec<T, VW>::unpack(w[i][h], x);
#pragma unroll
            for (int e = 0; e < VW; ++e) v[h * VW + e] = x[e];
        }
    }
};
// VW 0: rows of any alignment in tensors that start and end on 16-byte boundaries, runs of eight cut out of aligned pieces.  (Single elements, VW 1, cost the few-state kernels their
// loads: 4 608 rows of 8 594 elements, 4 states, bf16 1021 -> 394 us.)
template <typename T, int RPW> struct StRaw<T, RPW, 0> {
    static constexpr int kRuns = RPW / 8;
    Row8<T, 0> w[kRuns];
    template <typename F> static __device__ __forceinline__ void for_each(int lane, F f) {
#pragma unroll
        for (int i = 0; i < kRuns; ++i) f(i, i * 8 + (lane >> 2), (lane & 3) * 8, std::integral_constant<int, 8>{});
    }
    __device__ __forceinline__ void load(const T* rows, int64_t stride, int count, int t0, int L, int lane) {
        for_each(lane, [&](int i, int row, int el, auto) {
            w[i] = {};
            if (row < count) w[i].load(rows + row * stride, t0 + el, 0, L);
        });
    }
    __device__ __forceinline__ void get(int i, float (&v)[8], const T* rows, int64_t stride, int t0, int L, int lane) const {
        w[i].get(rows + (i * 8 + (lane >> 2)) * stride, t0 + (lane & 3) * 8, 0, L, v);
    }
};
// B or C of one chunk, spread over the threads of the CTA.
template <typename T, int NS, int VW, int WARPS> struct StRawBC {
    static constexpr int kThreads = WARPS * 32, kItems = VW > 1 ? NS * 4 : NS * 32, kPer = (kItems + kThreads - 1) / kThreads;
    static constexpr int kVecs = VW > 1 ? 8 / VW : 1;
    typename Vec<T, VW>::Raw w[kPer][kVecs];
    static __device__ __forceinline__ void place(int i, int& n, int& el) {
        if constexpr (VW > 1) { n = i % NS; el = (i / NS) * 8; }
        else { n = i >> 5; el = i & 31; }
    }
    __device__ __forceinline__ void load(const T* src, int64_t state_stride, int N, int t0, int L) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            int n, el;
            place(threadIdx.x + j * kThreads, n, el);
#pragma unroll
            for (int h = 0; h < kVecs; ++h) {
                w[j][h] = {};
                if (n < N && el < kStChunk && t0 + el + h * VW < L) w[j][h] = Vec<T, VW>::load_raw(src + n * state_stride + t0 + el + h * VW);
            }
        }
    }
    __device__ __forceinline__ void put(float* dst, const T*, int64_t, int, int) const {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            int n, el;
            place(threadIdx.x + j * kThreads, n, el);
            if (kItems % kThreads == 0 || threadIdx.x + j * kThreads < kItems) {
#pragma unroll
                for (int h = 0; h < kVecs; ++h) {
                    float x[VW];
                    Vec<T, VW>::unpack(w[j][h], x);
#pragma unroll
                    for (int e = 0; e < VW; ++e) dst[(el + h * VW + e) * StLayout<NS>::BCP + n] = x[e];
                }
            }
        }
    }
};

template <typename T, int NS, int WARPS> struct StRawBC<T, NS, 0, WARPS> {
    static constexpr int kThreads = WARPS * 32, kItems = NS * 4, kPer = (kItems + kThreads - 1) / kThreads;
    Row8<T, 0> w[kPer];
    __device__ __forceinline__ void load(const T* src, int64_t state_stride, int N, int t0, int L) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int i = threadIdx.x + j * kThreads, n = i % NS, el = (i / NS) * 8;
            w[j] = {};
            if (n < N && el < kStChunk) w[j].load(src + n * state_stride, t0 + el, 0, L);
        }
    }
    __device__ __forceinline__ void put(float* dst, const T* src, int64_t state_stride, int t0, int L) const {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int i = threadIdx.x + j * kThreads, n = i % NS, el = (i / NS) * 8;
            if (kItems % kThreads == 0 || i < kItems) {
                float v[8];
                w[j].get(src + n * state_stride, t0 + el, 0, L, v);
#pragma unroll
                for (int e = 0; e < 8; ++e) dst[(el + e) * StLayout<NS>::BCP + n] = v[e];
            }
        }
    }
};

// Number of segments a row is cut into (1: none) and their length, given the warps that whole rows fill.  Cutting costs a
// second pass, so it starts below four warps per SM and then goes up to sixteen (16 states, bf16: 768 rows of 3 136
// elements 144 -> 36 us, 384 rows of 65 536 3.7 -> 0.29 ms; 6 144 rows, which fill five warps, 225 uncut, 255, 224 and 271 cut in two, three and
// four; fp32, 6 144 rows of 1 001 83 uncut, 95 and 91 cut in two and three).
// `resident`: sixteen is what the SM holds, and more would be a second round (rows of vectors: 3 072 rows of 3 136, 16 states, fp32, 161 us with
// seven segments, 132 with six); where it holds more, the number is rounded up (4 608 rows of 8 594, 4 states, bf16, 308 against 318).
struct StSegments { int count, len; };
inline StSegments st_segments(int64_t warps, int64_t L, bool resident) {
    const int64_t want = 148 * 16;
    if (warps * 4 > want || L < 192) return {1, (int)((L + 63) / 64 * 64)};
    int64_t s = (resident ? want : want + warps - 1) / warps;
    const int64_t most = (L + 63) / 64;
    if (s > most) s = most;
    const int64_t len = (((L + s - 1) / s) + 63) / 64 * 64;
    s = (L + len - 1) / len;
    return {(int)s, (int)len};
}

// What the segments in front of segment `seg` (behind it, with kBack) leave in the four states of a lane.
template <bool kBack>
__device__ __forceinline__ void st_fold_segments(float2 (&h)[2], const float2 (&A2)[2], const float* ends, const float* sums, int64_t row, int S,
                                                 int seg, int n0, int NSpad) {
    h[0] = h[1] = make_float2(0.f, 0.f);
    const int from = kBack ? S - 1 : 0, step = kBack ? -1 : 1;
    for (int j = from; j != seg; j += step) {
        const float d = sums[row * S + j];
        const float4 e = *reinterpret_cast<const float4*>(ends + (row * S + j) * NSpad + n0);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float2 x = __fmul2_rn(f2(d), A2[q]);
            h[q] = __ffma2_rn(make_float2(ex2_approx(x.x), ex2_approx(x.y)), h[q], q ? make_float2(e.z, e.w) : make_float2(e.x, e.y));
        }
    }
}

}  // namespace ss2d
