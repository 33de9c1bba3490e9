// Eight consecutive elements of a row, for the one-state selective-scan kernels.
#pragma once
#include "common.cuh"

namespace ss2d {

// The piece at p, or zeros.  16-bit rows: as one predicated load, which the compiler leaves where it is (1 024 rows of 16 385 elements 44.4 us; as a plain one
// under a condition 46.0).  fp32 rows, whose registers are full: as a plain one, which it may place (57 us, predicated 72).  Both come
// behind the wait for the kernel in front (follow_previous), which is volatile too.
#ifdef __CUDACC__
template <bool kPredicated> __device__ __forceinline__ uint4 piece_load(const uint4* p, bool in) {
    uint4 t = make_uint4(0, 0, 0, 0);
    if constexpr (!kPredicated) {
        if (in) t = *p;
    } else {
        asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %5, 0;\n mov.b32 %0, 0;\n mov.b32 %1, 0;\n mov.b32 %2, 0;\n mov.b32 %3, 0;\n"
                     " @p ld.global.v4.b32 {%0, %1, %2, %3}, [%4];\n}"
                     : "=&r"(t.x), "=&r"(t.y), "=&r"(t.z), "=&r"(t.w) : "l"(p), "r"((int)in));
    }
    return t;
}
#else                                                // for the host: what stands for common.cuh looks where it reads
template <bool kPredicated> uint4 piece_load(const uint4* p, bool in) { return in ? __ldg(p) : make_uint4(0, 0, 0, 0); }
#endif

// The bytes of a tensor of rows, and whether they start and end on 16-byte boundaries: then no aligned piece that holds an element
// of a row reaches beyond them.
struct Span { uintptr_t lo, hi; };
inline Span span_of(const void* first, size_t size, int64_t elements) {
    const uintptr_t p = reinterpret_cast<uintptr_t>(first);
    return {p, p + (uintptr_t)elements * size};
}
inline bool whole_pieces(Span s) { return s.lo % 16 == 0 && s.hi % 16 == 0; }

// Elements [pos, pos + 8) of a row of L elements, held as loaded; those outside the row read as zero.
// AL 8, 4, 2 or 1: vectors of that many elements (row starts aligned to them, L and pos multiples of AL, pos >= 0).
// AL 0: any alignment and any pos.  The vector is cut out of the two or three aligned 16-byte pieces around it; only pieces
// that hold at least one element of [from, L) are read.  They stay inside a tensor that starts and ends on 16-byte boundaries;
// of any other, the rows' elements in the outermost, partial piece are the caller's: the forward walk takes them one by one
// (Inner), the other kernels read such tensors by single elements.  A test for them in here, a branch around the loads or a
// second source of the values, keeps the loads from staying in flight: 1 024 rows of 16 385 elements 51 -> 69 and 57 us.
template <typename T, int AL> struct Row8 {
    static constexpr int kN = 8 / AL;
    typename Vec<T, AL>::Raw w[kN];
    __device__ __forceinline__ void load(const T* __restrict__ row, int pos, int, int L) {
#pragma unroll
        for (int j = 0; j < kN; ++j) {
            w[j] = {};
            if (pos + j * AL < L) w[j] = Vec<T, AL>::load_raw(row + pos + j * AL);
        }
    }
    __device__ __forceinline__ void get(const T*, int, int, int, float (&v)[8]) const {
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
    __device__ __forceinline__ void load(const T* __restrict__ row, int pos, int from, int L) {
        const intptr_t at = reinterpret_cast<intptr_t>(row) + (intptr_t)pos * (int)sizeof(T);
        const uint4* q = reinterpret_cast<const uint4*>(at & ~(intptr_t)15);
        const int off = (int)(at & 15) / (int)sizeof(T), e0 = pos - off;       // e0: element at the start of the first piece
#pragma unroll
        for (int i = 0; i <= kPieces; ++i) {
            const int e = e0 + i * kPiece;
            const uint4 t = piece_load<sizeof(T) == 2>(q + i, e < L && e + kPiece > from && (i < kPieces || off != 0));
            w[4 * i] = t.x; w[4 * i + 1] = t.y; w[4 * i + 2] = t.z; w[4 * i + 3] = t.w;
        }
    }
    __device__ __forceinline__ void get(const T* __restrict__ row, int pos, int from, int L, float (&v)[8]) const {
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
        if (pos < from || pos + 8 > L) {         // the pieces at the ends of a row hold elements of its neighbours
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (pos + e < from || pos + e >= L) v[e] = 0.f;
        }
    }
};


// [from, to): the elements of a row that lie in pieces inside the tensor; none: from = L, to < 0 (no piece is read).
// A walk over them costs what one over whole rows does (1 024 rows of 16 385, B and C of odd length: 51.2 -> 50.8 us).
struct Inner { int from, to; };
__device__ __forceinline__ Inner inner(int from, int to, int L) { return from < to ? Inner{from, to} : Inner{L, -64}; }
template <typename T> __device__ __forceinline__ Inner inner_of(const T* row, int L, Span s) {
    const uintptr_t p = reinterpret_cast<uintptr_t>(row), lo = (s.lo + 15) & ~(uintptr_t)15, hi = s.hi & ~(uintptr_t)15, end = p + (uintptr_t)L * sizeof(T);
    return inner(p < lo ? min(L, (int)((lo - p) / sizeof(T))) : 0, end > hi ? L - (int)((end - hi) / sizeof(T)) : L, L);
}
__device__ __forceinline__ Inner both(Inner a, Inner b, int L) { return inner(max(a.from, b.from), min(a.to, b.to), L); }
// The tensors of a scan call, forward or backward (the same members).
struct ScanSpans { Span u, delta, B, C; };
template <typename P> ScanSpans scan_spans(const P& p, size_t size) {
    const int64_t b = p.batch - 1, last = p.dim - 1, dlast = p.delta_ratio > 1 ? p.dim / p.delta_ratio - 1 : last, k = p.n_groups - 1, n = p.dstate - 1, L = p.seqlen;
    return {span_of(p.u, size, b * p.u_batch_stride + last * p.u_dim_stride + L), span_of(p.delta, size, b * p.delta_batch_stride + dlast * p.delta_dim_stride + L),
            span_of(p.B, size, b * p.B_batch_stride + k * p.B_group_stride + n * p.B_state_stride + L),
            span_of(p.C, size, b * p.C_batch_stride + k * p.C_group_stride + n * p.C_state_stride + L)};
}

}  // namespace ss2d
