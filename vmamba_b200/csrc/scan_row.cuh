// Eight consecutive elements of a row, for the one-state selective-scan kernels.
#pragma once
#include "common.cuh"

namespace ss2d {

// Elements [pos, pos + 8) of a row of L elements, held as loaded; those outside the row read as zero.
// AL 8, 4 or 2: vectors of that many elements (row starts aligned to them, L and pos multiples of AL, pos >= 0).
// AL 0: any alignment and any pos.  The vector is cut out of the two or three aligned 16-byte pieces around it; only pieces
// that hold at least one element of the row are read.
template <typename T, int AL> struct Row8 {
    static constexpr int kN = 8 / AL;
    typename Vec<T, AL>::Raw w[kN];
    __device__ __forceinline__ void load(const T* __restrict__ row, int pos, int L) {
#pragma unroll
        for (int j = 0; j < kN; ++j) {
            w[j] = {};
            if (pos + j * AL < L) w[j] = Vec<T, AL>::load_raw(row + pos + j * AL);
        }
    }
    __device__ __forceinline__ void get(const T*, int, int, float (&v)[8]) const {
#pragma unroll
        for (int j = 0; j < kN; ++j) {
            float y[AL];
            Vec<T, AL>::unpack(w[j], y);
#pragma unroll
            for (int e = 0; e < AL; ++e) v[j * AL + e] = y[e];
        }
    }
};
template <typename T> struct Row8<T, 0> {
    static constexpr int kPiece = 16 / (int)sizeof(T), kPieces = 8 / kPiece, NW = kPieces * 4;
    uint32_t w[NW + 4];
    __device__ __forceinline__ void load(const T* __restrict__ row, int pos, int L) {
        const intptr_t at = reinterpret_cast<intptr_t>(row) + (intptr_t)pos * (int)sizeof(T);
        const uint4* q = reinterpret_cast<const uint4*>(at & ~(intptr_t)15);
        const int off = (int)(at & 15) / (int)sizeof(T), e0 = pos - off;       // e0: element at the start of the first piece
#pragma unroll
        for (int i = 0; i <= kPieces; ++i) {
            uint4 t = make_uint4(0, 0, 0, 0);
            const int e = e0 + i * kPiece;
            if (e < L && e + kPiece > 0 && (i < kPieces || off != 0)) t = __ldg(q + i);
            w[4 * i] = t.x; w[4 * i + 1] = t.y; w[4 * i + 2] = t.z; w[4 * i + 3] = t.w;
        }
    }
    __device__ __forceinline__ void get(const T* __restrict__ row, int pos, int L, float (&v)[8]) const {
        const unsigned off = (unsigned)(reinterpret_cast<uintptr_t>(row) + (intptr_t)pos * (int)sizeof(T)) & 15u;
        uint32_t x[NW + 4];
#pragma unroll
        for (int i = 0; i < NW + 4; ++i) x[i] = w[i];
        if (off & 8u) {
#pragma unroll
            for (int i = 0; i < NW + 2; ++i) x[i] = x[i + 2];
        }
        if (off & 4u) {
#pragma unroll
            for (int i = 0; i < NW + 1; ++i) x[i] = x[i + 1];
        }
        if constexpr (sizeof(T) == 2) {
            const unsigned sh = (off & 2u) * 8u;
#pragma unroll
            for (int i = 0; i < NW; ++i) {
                const float2 f = Half2Of<T>::unpack(__funnelshift_r(x[i], x[i + 1], sh));
                v[2 * i] = f.x; v[2 * i + 1] = f.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(x[i]);
        }
        if (pos < 0 || pos + 8 > L) {            // the pieces at the ends of a row hold elements of its neighbours
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (pos + e < 0 || pos + e >= L) v[e] = 0.f;
        }
    }
};

}  // namespace ss2d
