// Asynchronous copies of 16-byte pieces into shared memory, and the sum of four routes: what the CrossScan / CrossMerge kernels share.
#pragma once
#include "common.cuh"

namespace ss2d {

__device__ __forceinline__ void piece_copy_async(void* to, const void* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void piece_wait() {       // of the whole CTA's copies
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

// V neighbours, 1, or 2 of 16 bits in a word.
template <typename T, int V> struct Pixels {
    T e;
    __device__ __forceinline__ void load(const T* p) { e = *p; }
    __device__ __forceinline__ void store(T* p) const { *p = e; }
    __device__ __forceinline__ T at(int) const { return e; }
    __device__ __forceinline__ void set(int, T x) { e = x; }
    __device__ __forceinline__ Pixels turned() const { return *this; }
};
template <typename T> struct Pixels<T, 2> {
    static_assert(sizeof(T) == 2, "");
    uint32_t w;
    __device__ __forceinline__ void load(const T* p) { w = *reinterpret_cast<const uint32_t*>(p); }
    __device__ __forceinline__ void store(T* p) const { *reinterpret_cast<uint32_t*>(p) = w; }
    __device__ __forceinline__ T at(int i) const { const uint16_t x = (uint16_t)(i ? w >> 16 : w); return *reinterpret_cast<const T*>(&x); }
    __device__ __forceinline__ void set(int i, T x) {
        const uint32_t b = *reinterpret_cast<const uint16_t*>(&x);
        w = i ? (w & 0xffffu) | b << 16 : b;         // the first one first
    }
    __device__ __forceinline__ Pixels turned() const { Pixels r; r.w = __byte_perm(w, 0, 0x1032); return r; }
};

// Sum of four routes in the association order of the reference's additions, rounded to the storage type after each.
template <typename T> __device__ __forceinline__ T flat_add(T x, T y) { return from_f<T>(to_f<T>(x) + to_f<T>(y)); }
template <typename T> __device__ __forceinline__ T flat_sum(int scans, T x0, T x1, T x2, T x3) {
    if (scans == 0 || scans == 2) return flat_add(flat_add(x0, x2), flat_add(x1, x3));
    if (scans == 3) return flat_add(flat_add(flat_add(x0, x1), x2), x3);
    return from_f<T>(((to_f<T>(x0) + to_f<T>(x1)) + to_f<T>(x2)) + to_f<T>(x3));
}

}  // namespace ss2d
