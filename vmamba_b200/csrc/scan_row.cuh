// Eight consecutive elements of a row at any alignment, for the one-state selective-scan kernels.
#pragma once
#include "common.cuh"

namespace ss2d {

// Elements [pos, pos + 8) of a row of L elements; the ones outside read as zero.  The address may be aligned to one element
// only: the vector is cut out of the two or three aligned 16-byte pieces around it (each of which holds at least one of
// its elements, so nothing outside the row's own 16-byte pieces is touched).  The misalignment is the same for all
// lanes of a warp when their vectors are whole vectors apart.
template <typename T>
__device__ __forceinline__ void load8_any(const T* __restrict__ row, int pos, int L, float (&v)[8]) {
    if (pos >= 0 && pos + 8 <= L) {
        constexpr int NW = 8 * (int)sizeof(T) / 4;            // 32-bit words of the vector
        const uintptr_t at = reinterpret_cast<uintptr_t>(row + pos);
        const uint4* q = reinterpret_cast<const uint4*>(at & ~(uintptr_t)15);
        const unsigned off = (unsigned)at & 15u;
        uint32_t w[NW + 4];
#pragma unroll
        for (int i = 0; i < NW / 4; ++i) {
            const uint4 t = __ldg(q + i);
            w[4 * i] = t.x; w[4 * i + 1] = t.y; w[4 * i + 2] = t.z; w[4 * i + 3] = t.w;
        }
        uint4 t = make_uint4(0, 0, 0, 0);
        if (off) t = __ldg(q + NW / 4);
        w[NW] = t.x; w[NW + 1] = t.y; w[NW + 2] = t.z; w[NW + 3] = t.w;
        if (off & 8u) {
#pragma unroll
            for (int i = 0; i < NW + 2; ++i) w[i] = w[i + 2];
        }
        if (off & 4u) {
#pragma unroll
            for (int i = 0; i < NW + 1; ++i) w[i] = w[i + 1];
        }
        if constexpr (sizeof(T) == 2) {
            const unsigned sh = (off & 2u) * 8u;
#pragma unroll
            for (int i = 0; i < NW; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], sh);
#pragma unroll
            for (int i = 0; i < NW; ++i) {
                const float2 f = Half2Of<T>::unpack(w[i]);
                v[2 * i] = f.x; v[2 * i + 1] = f.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(w[i]);
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = (pos + e >= 0 && pos + e < L) ? to_f<T>(__ldg(row + pos + e)) : 0.f;
    }
}

}  // namespace ss2d
