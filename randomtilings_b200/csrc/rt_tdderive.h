// rt_tdderive.h -- triangle-flip and butterfly-flip states of a triangle-dimer
// tiling of side n (TilingToTriangleFlips / TilingToButterflyFlips,
// TriangleDimerTiler.cpp:385-460), cell by cell, for the host's builders and the
// kernel that sets up a walk's arrays.
#pragma once

#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define RT_TDD_HD __host__ __device__ inline
#else
#define RT_TDD_HD inline
#endif

namespace rtb {

RT_TDD_HD int td_bit(int32_t x, int k) { return (x >> k) & 1; }

// State of cell (i, j) of the (n / 2) x n triangle array.
RT_TDD_HD int32_t td_triangle_state(const int32_t* t, int n, int i, int j) {
    if (i < 1 || i >= n / 2 - 1 || j < 1 || j >= n - 1) return 0;
    auto T = [&](int y, int x) { return t[(size_t)y * n + x]; };
    const int32_t a = T(2 * i + 1, j), c = T(2 * i + 1, j + 1);
    int d0, d1, d2;
    if (j % 2 == 0) {  // down triangle
        const int32_t u = T(2 * i, j + 1);
        d0 = td_bit(a, 2) + 2 * td_bit(a, 3) + 3 * td_bit(c, 3);
        d1 = td_bit(c, 2) + 2 * td_bit(a, 1) + 3 * td_bit(c, 1);
        d2 = 2 * td_bit(u, 0) + td_bit(a, 0) + 3 * td_bit(u, 1);
    } else {  // up triangle
        const int32_t w = T(2 * i + 2, j);
        d0 = td_bit(a, 0) + 2 * td_bit(a, 3) + 3 * td_bit(c, 3);
        d1 = td_bit(c, 0) + 2 * td_bit(a, 1) + 3 * td_bit(c, 1);
        d2 = 2 * td_bit(w, 3) + 3 * td_bit(w, 2) + td_bit(a, 2);
    }
    return d0 + 4 * d1 + 16 * d2;
}

// State of cell (i, j) of the n x n butterfly array.
RT_TDD_HD int32_t td_butterfly_state(const int32_t* t, int n, int i, int j) {
    if (i < 2 || i >= n - 2 || j < 2 || j >= n - 2 || (i % 2 == 0 && j % 2 == 0)) return 0;
    auto T = [&](int y, int x) { return t[(size_t)y * n + x]; };
    auto b = [](int32_t v, int k) { return td_bit(v, k); };
    const int32_t x = T(i, j);
    int f1, f4, f16, f64, c;
    if (i % 2 == 0) {
        const int32_t u = T(i - 1, j), ue = T(i - 1, j + 1), d = T(i + 1, j), dw = T(i + 1, j - 1);
        f1 = b(u, 3) + 2 * b(u, 0) + 3 * b(x, 0);
        f4 = b(ue, 0) + 2 * b(ue, 1) + 3 * b(x, 1);
        f16 = b(d, 1) + 2 * b(d, 2) + 3 * b(x, 2);
        f64 = b(dw, 2) + 2 * b(dw, 3) + 3 * b(x, 3);
        c = b(ue, 2);
    } else if (j % 2 == 0) {
        const int32_t ue = T(i - 1, j + 1), e = T(i, j + 1), dw = T(i + 1, j - 1), w = T(i, j - 1);
        f1 = b(ue, 0) + 2 * b(ue, 1) + 3 * b(x, 0);
        f4 = b(e, 1) + 2 * b(e, 2) + 3 * b(x, 1);
        f16 = b(dw, 2) + 2 * b(dw, 3) + 3 * b(x, 2);
        f64 = b(w, 3) + 2 * b(w, 0) + 3 * b(x, 3);
        c = b(e, 3);
    } else {
        const int32_t u = T(i - 1, j), e = T(i, j + 1), d = T(i + 1, j), w = T(i, j - 1);
        f1 = b(u, 0) + 2 * b(u, 1) + 3 * b(x, 0);
        f4 = b(e, 0) + 2 * b(e, 1) + 3 * b(x, 1);
        f16 = b(d, 2) + 2 * b(d, 3) + 3 * b(x, 2);
        f64 = b(w, 2) + 2 * b(w, 3) + 3 * b(x, 3);
        c = b(e, 3);
    }
    return f1 + 4 * f4 + 16 * f16 + 64 * f64 + 256 * c;
}

}  // namespace rtb
