"""The vectors that the scan kernels cut out of aligned pieces (csrc/scan_row.cuh), compiled for the host: what they hold, and that
no load reaches beyond the tensor."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vmamba_b200", "csrc")

# in the place of common.cuh: loads that look whether they stay inside the tensor
COMMON = r"""
#pragma once
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
#define __restrict__
struct uint4 { uint32_t x, y, z, w; };
struct float2 { float x, y; };
template <typename T> float to_f(T v) { float f = (float)v; if (sizeof(T) == 4) memcpy(&f, &v, 4); return f; }
inline int min(int a, int b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
inline float __uint_as_float(uint32_t v) { float f; memcpy(&f, &v, 4); return f; }
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, unsigned s) { s &= 31; return s ? lo >> s | hi << (32 - s) : lo; }
extern const unsigned char *first, *behind;
extern long outside;
template <typename T> T __ldg(const T* p) {
    const unsigned char* q = (const unsigned char*)p;
    if (q < first || q + sizeof(T) > behind || (uintptr_t)q % sizeof(T)) { ++outside; return T{}; }
    T v; memcpy(&v, q, sizeof(T)); return v;
}
template <typename T, int V> struct Vec { struct Raw {}; static Raw load_raw(const T*) { return {}; } static void unpack(const Raw&, float (&)[V]) {} };
template <typename T> struct Half2Of { static float2 unpack(uint32_t w) { return {(float)(w & 0xffff), (float)(w >> 16)}; } };
"""
MAIN = r"""
#include "scan_row.cuh"
#include <cstdio>
const unsigned char *first, *behind;
long outside = 0;
alignas(16) static unsigned char memory[8192];
template <typename T> long wrong() {                  // T: 16-bit or 32-bit values that stand for themselves
    long bad = 0;
    for (int phase = 0; phase < 16 / (int)sizeof(T); ++phase)
        for (int L = 1; L <= 40; ++L)
            for (int stride = L; stride <= L + 3; ++stride) {
                const int rows = 5, n = (rows - 1) * stride + L;
                T* t = (T*)(memory + 1024) + phase;
                first = (unsigned char*)t; behind = (unsigned char*)(t + n);
                for (int i = 0; i < n; ++i) t[i] = (T)(1 + i);
                const ss2d::Span s = ss2d::span_of(t, sizeof(T), n);
                const bool pieces = ss2d::whole_pieces(s);
                for (int r = 0; r < rows; ++r)
                    for (int pos = -9; pos < L + 9; ++pos) {
                        const T* row = t + r * stride;
                        float x[8];
                        const ss2d::Inner in = ss2d::inner_of(row, L, s);
                        if (pieces) bad += in.from != 0 || in.to != L;
                        ss2d::Row8<T, 0> v;
                        v.load(row, pos, in.from, in.to);
                        v.get(row, pos, in.from, in.to, x);
                        for (int e = 0; e < 8; ++e) {
                            const uint32_t want = pos + e >= in.from && pos + e < in.to ? t[r * stride + pos + e] : 0;
                            float w = (float)want;
                            if (sizeof(T) == 4) memcpy(&w, &want, 4);
                            if (in.from < in.to) bad += in.from > 7 || L - in.to > 7;       // what is left for single elements
                            bad += memcmp(&w, &x[e], 4) != 0;
                        }
                    }
            }
    return bad;
}
int main() {
    const long bad = wrong<uint16_t>() + wrong<uint32_t>();
    printf("%ld %ld\n", bad, outside);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_vectors_of_any_alignment_stay_inside_the_tensor(tmp_path):
    shutil.copy(os.path.join(CSRC, "scan_row.cuh"), tmp_path)
    (tmp_path / "common.cuh").write_text(COMMON)
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-w", "-o", str(tmp_path / "main"), str(tmp_path / "main.cpp")])
    assert subprocess.check_output([str(tmp_path / "main")]).split() == [b"0", b"0"]       # wrong values, loads outside
